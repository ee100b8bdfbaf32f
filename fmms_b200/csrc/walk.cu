// Dual tree walk, target by target, with the interaction lists as its output.
//
// The reference walks mutual cell pairs depth first (process_pair,
// walk.rs:94-190) and records them (walk.rs:342-488). Every decision depends on
// the pair alone, so the pairs can be taken in any order and from either end:
// here every cell c settles its own side of its pairs. It starts from the list
// its parent passed down and, for each source s of it,
//   - accepts s for M2L,
//   - takes s for P2P when both are leaves,
//   - replaces s by its children, or
//   - passes s down to its own children,
// exactly as the mutual pair (a, b), a the earlier of the two in depth-first
// order (as in the reference, where a pair's first cell comes from the earlier
// octant of their last common ancestor), would be treated. A self pair passes
// c's children down. Each mutual pair is met once from each end, so c's M2L and
// P2P lists come out whole, contiguous and in an order that depends on the tree
// alone: no list has to be sorted or scattered. (The walk used to append mutual
// pairs with atomics, a frontier at a time, and a counting sort and segment sorts
// made the lists. Walk and lists alone on the device: N = 2^22, 64 clusters,
// 14.4 + 47 -> 21.3 + 2.5 ms; uniform 2^20 0.41 + 0.99 -> 0.44 + 0.07; 10^3
// bodies 0.145 + 0.22 -> 0.13 + 0.01.)
//
// The sources of a cell are taken in blocks of WK_BLOCK inherited entries; of a
// block first in, first out: its entries, then the children of those that split
// in their order, and so on until none is left. This order does not depend on
// how many sources a step takes, so a cell may be walked by one warp or by many,
// and the lists (and every sum over them) come out the same.
//
// One launch per level of the tree. A level of many cells takes a warp per cell;
// where there are few, or for the cells whose walk is long (a shallow leaf beside
// a dense core meets 10^4 sources and more), 8 or 32 warps share a cell. The lists
// grow in chunks of 32 entries from a pool; a last kernel copies them into
// contiguous arrays.
//
// This file is compiled with --fmad=false: the MAC reproduces the reference's
// FP64 operation order.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace fmmx {

static __device__ OrderTables g_tab;

void upload_tables_walk(const OrderTables& t, cudaStream_t s) {
    cudaMemcpyToSymbolAsync(g_tab, &t, sizeof(t), 0, cudaMemcpyHostToDevice, s);
}

// ------------------------------------------------------------ MAC
// What the error-controlled MAC reads of a cell, in one row of p + 2 pairs:
// (mass, fmin), then (P_k, rho^{p-k}) for k = 0 .. p, the powers built up as the
// reference does (rho^j = rho^{j-1} rho).
__global__ void k_mac_rows(int nc, CellsView cv, int p, const double* __restrict__ pows,
                           const double* __restrict__ fminv, double2* __restrict__ rows) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        double2* row = rows + (size_t)c * (p + 2);
        row[0] = make_double2(cv.mass[c], fminv[c]);
        const double rho = cv.rho[c];
        double rp = 1.0;
        for (int j = 0; j <= p; ++j) {
            row[1 + p - j] = make_double2(pows[(size_t)c * (p + 1) + p - j], rp);
            rp *= rho;
        }
    }
}

// error_estimate + accept, mac.rs:23-95, in both directions of a pair
// (walk.rs:138-139). The operations and their order are the reference's
// (including the inner r*r of error_estimate); what the two directions share
// (r, its power, the radii's factor) is the same bits either way round.
__device__ __noinline__ bool accept_dehnen_exact(const MacParams& mp, const double2* __restrict__ row_c,
                                                 const double2* __restrict__ row_s, double r2, double rc, double rs) {
    const double sum_rho = rc + rs;
    const double r = sqrt(r2);
    if (r == 0.0) return false;
    const int p = mp.p;
    const double rr2 = r * r;
    double rp = 1.0;
    for (int i = 0; i < p / 2; ++i) rp *= rr2;
    if (p % 2 == 1) rp *= r;
    const double2 mc = row_c[0], ms = row_s[0];
    double sc = 0.0, ss = 0.0;  // c's multipoles onto s's radius, s's onto c's
    for (int k = 0; k <= p; ++k) {
        const double bk = g_tab.binom[p][k];
        const double2 vc = row_c[1 + k], vs = row_s[1 + k];
        sc += bk * vc.x * vs.y;
        ss += bk * vs.x * vc.y;
    }
    const double w = sum_rho == 0.0 ? 0.0 : 8.0 * fmax(rc, rs) / sum_rho;
    const double est_c = sum_rho == 0.0 ? 0.0 : w * (sc / (mc.x * rp));
    const double est_s = sum_rho == 0.0 ? 0.0 : w * (ss / (ms.x * rp));
    const bool ok_c = est_c == 0.0 || est_c * mc.x / r2 < mp.eps * ms.y;
    const bool ok_s = est_s == 0.0 || est_s * ms.x / r2 < mp.eps * mc.y;
    return ok_c && ok_s;
}

// The same decision with the divisions multiplied out,
//   8 max(rho) sum_k binom P_k rho^{p-k} < eps fmin (rho_c + rho_s) r^p r^2,
// where it is certain: every term is non-negative, so both sides are within
// (p + 10) roundings (below 1e-14) of their exact values, and so are the sides
// of the reference's comparison; a gap of 1e-9 decides. Closer pairs, and values
// outside the normal range, take the reference's own operations.
__device__ __forceinline__ bool accept_dehnen_pair(const MacParams& mp, const double2* __restrict__ row_c,
                                                   const double2* __restrict__ row_s, const double4 gc,
                                                   const double4 gs) {
    const double dx = gs.x - gc.x, dy = gs.y - gc.y, dz = gs.z - gc.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double rc = gc.w, rs = gs.w;
    const double sum_rho = rc + rs;
    if (r2 <= sum_rho * sum_rho) return false;
    const int p = mp.p;
    double t = (p & 1) ? r2 * rsqrt(r2) : 1.0;  // r^p
    {
        double q = r2;
        for (int e = p >> 1; e > 0; e >>= 1) {
            if (e & 1) t *= q;
            q *= q;
        }
    }
    const double2 mc = row_c[0], ms = row_s[0];
    double sc = 0.0, ss = 0.0;
#pragma unroll 4
    for (int k = 0; k <= p; ++k) {
        const double bk = g_tab.binom[p][k];
        const double2 vc = row_c[1 + k], vs = row_s[1 + k];
        sc = fma(bk * vc.x, vs.y, sc);
        ss = fma(bk * vs.x, vc.y, ss);
    }
    const double big = 8.0 * fmax(rc, rs);
    const double lc = big * sc, ls = big * ss;
    const double right = mp.eps * sum_rho * t * r2;
    const double hc = right * ms.y, hs = right * mc.y;
    const bool normal = lc > 1e-280 && ls > 1e-280 && hc > 1e-280 && hs > 1e-280 && t > 1e-280 && lc < 1e280 &&
                        ls < 1e280 && hc < 1e280 && hs < 1e280 && t < 1e280;
    if (normal) {
        const double lo = 1.0 - 1e-9, hi = 1.0 + 1e-9;
        if (lc > hc * hi || ls > hs * hi) return false;
        if (lc < hc * lo && ls < hs * lo) return true;
    }
    return accept_dehnen_exact(mp, row_c, row_s, r2, rc, rs);
}

// Separation condition (extension, with softening): the bodies of the two
// cells are at least mp.gap apart, r - rho_A - rho_B >= gap.
__device__ __forceinline__ bool gap_ok(const MacParams& mp, const double4 ga, const double4 gb) {
    if (!(mp.gap > 0.0)) return true;
    const double dx = gb.x - ga.x, dy = gb.y - ga.y, dz = gb.z - ga.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    return sqrt(r2) - (ga.w + gb.w) >= mp.gap;
}

// The geometric MAC (extension): accept when (rho_A + rho_B) < theta r, both
// ways round as the reference's walk applies its MAC (walk.rs:138-139), and
// gap_ok. The two directions and gap_ok evaluate the same r2 (the squares of
// b - a and a - b are equal bit for bit) and the same rho sum (addition
// commutes), so one square root decides all three.
__device__ __forceinline__ bool accept_theta_pair(const MacParams& mp, const double4 ga, const double4 gb) {
    const double dx = gb.x - ga.x, dy = gb.y - ga.y, dz = gb.z - ga.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double sum_rho = ga.w + gb.w;
    const double r = sqrt(r2);
    if (!(sum_rho < mp.theta * r)) return false;
    return !(mp.gap > 0.0) || r - sum_rho >= mp.gap;
}

// ------------------------------------------------------------ walk
// children of a cell: 8 ids (-1 absent), 32-byte aligned, read as two int4
__device__ __forceinline__ void load_children(const CellsView& cv, int c, int (&ch)[8]) {
    const int4* p = reinterpret_cast<const int4*>(cv.child + 8 * (size_t)c);
    const int4 u = p[0], v = p[1];
    ch[0] = u.x; ch[1] = u.y; ch[2] = u.z; ch[3] = u.w;
    ch[4] = v.x; ch[5] = v.y; ch[6] = v.z; ch[7] = v.w;
}

// geo[c] = (centre, rho), with the sign of rho set for a leaf: a pair's test
// reads one 32-byte record per source.
__device__ __forceinline__ bool geo_leaf(const double4 g) { return signbit(g.w); }
__device__ __forceinline__ double4 geo_abs(double4 g) {
    g.w = fabs(g.w);
    return g;
}

// One list under construction; every thread of the cell's group holds the same values.
struct ListTail {
    uint32_t n = 0;
    uint32_t head = ~0u, last = ~0u;
    // chunks that `add` more entries need beyond the last one
    __device__ __forceinline__ uint32_t room() const { return (32u - (n & 31u)) & 31u; }
    __device__ __forceinline__ uint32_t chunks(uint32_t add) const {
        const uint32_t r = room();
        return add > r ? (add - r + 31) >> 5 : 0u;
    }
};

// Entry `rank` of `add` new ones (value v, if mine); the new chunks are base, base + 1, ...
// A chunk beyond the pool is not written: the overflow flag is set and the walk
// is redone. `first`: the thread that links the chunks and notes whose they are
// (owner: the cell, the list -- 0 M2L, 1 P2P, 2 passed down, which has links instead
// -- whether a heavy cell's second walk wrote it, and its place in the list).
__device__ __forceinline__ void list_add(const WalkPool& P, ListTail& t, uint32_t add, uint32_t base, bool mine,
                                         uint32_t rank, uint32_t v, bool first, uint32_t cell, uint32_t kind,
                                         uint32_t redone) {
    const uint32_t r = t.room(), q = t.chunks(add);
    if (mine) {
        const uint32_t id = rank < r ? t.last : base + ((rank - r) >> 5);
        const uint32_t at = rank < r ? (t.n & 31u) + rank : (rank - r) & 31u;
        if (id < P.cap) P.entry[(size_t)32 * id + at] = v;
    }
    if (q) {
        if (first) {
            if (kind == 2u && t.last < P.cap) P.next[t.last] = base;
            for (uint32_t k = 0; k < q && base + k < P.cap; ++k) {
                if (kind == 2u) P.next[base + k] = base + k + 1;
                P.owner[base + k] = kind == 2u ? make_uint2(~0u, 0u)
                                               : make_uint2(cell, kind << 30 | redone << 29 | (((t.n + 31) >> 5) + k));
            }
        }
        if (t.head == ~0u) t.head = base;
        t.last = base + q - 1;
    }
    t.n += add;
}

// counts of a group step in one word: M2L, P2P, passed down (up to 1024 each), children (up to 8192)
__device__ __forceinline__ unsigned long long pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return (unsigned long long)a | (unsigned long long)b << 12 | (unsigned long long)c << 24 |
           (unsigned long long)d << 36;
}

// Inherited entries per block, a multiple of 32. Short blocks leave the steps
// that empty a queue half filled, long ones need longer queues (64 entries:
// clustered N = 2^22 22.5 -> 27.5 ms).
#define WK_BLOCK 256u

// W warps per cell; the queue of RING sources in shared memory, or (RING = 0) in
// the block's part of `gring` (gcap entries: the sources waiting at any time are
// disjoint subtrees, so as many as there are leaves always suffice).
// list_mode: the cells are heavy.list[0 .. *heavy.count), else the level's. A cell
// whose queue is full, or (W = 1) that has taken `limit` sources, is left to
// the heavy list. Bound at shallow levels by the steps' barriers and L2 round
// trips (the sources' records, then the children of those that split: issue 20
// to 40 % of the time); where a level has many cells by issue with the theta
// criterion (53 to 55 %, 17 to 22 warps per SM) and by round trips with Dehnen's
// (26 to 29 %, 8 to 11 warps of 128 registers).
template <bool DEHNEN, int W, int RING>
__global__ void __launch_bounds__(32 * W) k_walk_level(const int32_t* __restrict__ level_cells, int lcnt, CellsView cv,
                                                       const int32_t* __restrict__ parent, MacParams mp,
                                                       const double2* __restrict__ rows, WalkPool P, WalkLists Ls,
                                                       WalkHeavy heavy, int* __restrict__ work, uint32_t limit,
                                                       uint32_t batch, uint32_t* __restrict__ gring, uint32_t gcap) {
    extern __shared__ __align__(16) uint32_t sring[];
    __shared__ unsigned long long wsum[2][W];
    __shared__ double2 srow[DEHNEN ? FMMX_MAXP + 2 : 1];  // the cell's row of the MAC
    __shared__ uint32_t bcast[4];  // chunk base, cell, self pair's children, next inherited chunk
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint32_t* ring = RING ? sring : gring + (size_t)blockIdx.x * gcap;
    const uint32_t cap = RING ? (uint32_t)RING : gcap;
    {   // after an overflow the lists are incomplete: the host retries with a larger pool (one read for the group,
        // since another block of this launch may be setting the flag)
        int stop = 0;
        if (tid == 0) stop = *reinterpret_cast<volatile int*>(P.overflow);
        if (W == 1 ? __any_sync(FULL, stop) : __syncthreads_or(stop)) return;
    }
    auto barrier = [&]() {
        if (W == 1) __syncwarp();
        else __syncthreads();
    };
    const int ncell = RING ? lcnt : min((int)*heavy.count, lcnt);
    const int32_t* cells = RING ? level_cells : heavy.list;
    uint32_t res_next = 0, res_end = 0;  // reserved chunks
    unsigned long long pops = 0, inter = 0, nm2l = 0, np2p = 0;  // thread sums (n*: thread 0)
    // the unused rest of the reservation (fewer than `batch` chunks): nobody's
    auto give_back = [&]() {
        const uint32_t id = res_next + (uint32_t)tid;
        if (id < res_end && id < P.cap) P.owner[id] = make_uint2(~0u, 0u);
    };
    int par_w = 0;  // parity of the step's wsum slots
    for (int round = 0;; ++round) {
        int j = blockIdx.x;  // the block's first cell; from then on the next one that no block has
        if (round > 0) {
            if (W == 1) {
                if (lane == 0) j = (int)gridDim.x + atomicAdd(work, 1);
                j = __shfl_sync(FULL, j, 0);
            } else {
                __syncthreads();
                if (tid == 0) bcast[1] = gridDim.x + (uint32_t)atomicAdd(work, 1);
                __syncthreads();
                j = (int)bcast[1];
            }
        }
        if (j >= ncell) break;
        const int c = cells[j];
        const int par = parent[c];
        const double4 gcs = cv.geo[c];
        const bool cleaf = geo_leaf(gcs);
        const double4 gc = geo_abs(gcs);
        const uint32_t tn = cv.count[c];
        ListTail lm, lp, ld;
        uint32_t taken = 0, cpops = tid == 0 ? 1u : 0u;  // the self pair
        unsigned long long cinter = 0;
        bool given_up = false;
        // q chunks in a row: from the group's reservation (every thread tracks it), refilled `batch` at a time
        // (what is left of the old one then belongs to nobody)
        auto reserve = [&](uint32_t q) -> uint32_t {
            if (q > res_end - res_next) {
                give_back();
                const uint32_t take = q > batch ? q : batch;
                uint32_t b = 0;
                if (tid == 0) b = atomicAdd(P.used, take);
                if (W == 1) {
                    b = __shfl_sync(FULL, b, 0);
                } else {
                    __syncthreads();
                    if (tid == 0) bcast[0] = b;
                    __syncthreads();
                    b = bcast[0];
                }
                res_next = b;
                res_end = b + take;
            }
            const uint32_t id = res_next;
            res_next += q;
            if (id + q > P.cap && tid == 0) atomicOr(P.overflow, 1);
            return id;
        };
        if (DEHNEN) {
            barrier();
            for (int k = tid; k < mp.p + 2; k += 32 * W) srow[k] = rows[(size_t)c * (mp.p + 2) + k];
            barrier();
        }
        {   // the self pair: a leaf interacts with itself, another cell passes its children down
            const int ch = cleaf ? (tid == 0 ? c : -1) : (tid < 8 ? cv.child[8 * (size_t)c + tid] : -1);
            unsigned have = __ballot_sync(FULL, ch >= 0);
            if (W > 1) {
                if (tid == 0) bcast[2] = have;
                __syncthreads();
                have = bcast[2];
            }
            const uint32_t add = (uint32_t)__popc(have), base = reserve(1);
            const uint32_t rank = (uint32_t)__popc(have & ((1u << lane) - 1u));
            if (cleaf) {
                list_add(P, lp, add, base, ch >= 0, rank, (uint32_t)ch, tid == 0, (uint32_t)c, cleaf ? 1u : 2u, RING ? 0u : 1u);
                if (tid == 0) cinter = (unsigned long long)tn * (tn - 1);
            } else {
                list_add(P, ld, add, base, ch >= 0, rank, (uint32_t)ch, tid == 0, (uint32_t)c, cleaf ? 1u : 2u, RING ? 0u : 1u);
            }
        }
        uint32_t inh = par < 0 ? 0u : Ls.down_n[par], at = par < 0 ? ~0u : Ls.down_head[par];
        uint32_t blk = 0;             // entries left of the current block
        uint32_t head = 0, size = 0;  // the queue
        // the next step's sources, their records on the way
        uint32_t s = (uint32_t)c, k = 0;
        bool have = false;
        double4 gss = gcs;
        auto fetch = [&]() {
            barrier();  // the queue's last writes
            have = false;
            k = 0;
            if (blk == 0 && size == 0) blk = min(inh, WK_BLOCK);
            if (blk > 0) {  // inherited chunks, one per warp
                k = min(blk, 32u * W);
                const uint32_t nchunk = (k + 31) >> 5;
                uint32_t mine = at;
                have = (uint32_t)tid < k;
                if (W > 1) {  // every warp follows the links to its chunk; the last one's successor is the next step's
                    for (uint32_t h = 0; h < (uint32_t)wid && h + 1 < nchunk; ++h) mine = P.next[mine];
                    if (inh > k) {
                        if ((uint32_t)tid == 32 * (nchunk - 1)) bcast[3] = P.next[mine];
                        __syncthreads();
                        at = bcast[3];
                    }
                } else if (inh > k) {
                    at = P.next[at];
                }
                if (have) s = P.entry[(size_t)32 * mine + lane];
                inh -= k;
                blk -= k;
            } else if (size > 0) {
                k = min(size, 32u * W);
                have = (uint32_t)tid < k;
                if (have) {
                    uint32_t q = head + tid;
                    if (q >= cap) q -= cap;
                    s = ring[q];
                }
                head += k;
                if (head >= cap) head -= cap;
                size -= k;
            }
            if (have && s != (uint32_t)c) gss = cv.geo[s];
        };
        fetch();
        while (k > 0) {
            taken += k;
            const uint32_t s0 = s;
            bool m2l = false, p2p = false, down = false;
            int npush = 0;
            int ch[8];
            if (have && s0 != (uint32_t)c) {  // (the self pair is done)
                if (s0 > (uint32_t)c) ++cpops;  // each mutual pair once
                const bool sleaf = geo_leaf(gss);
                const double4 gs = geo_abs(gss);
                bool acc;
                if (DEHNEN)
                    acc = accept_dehnen_pair(mp, srow, rows + (size_t)s0 * (mp.p + 2), gc, gs) && gap_ok(mp, gc, gs);
                else
                    acc = accept_theta_pair(mp, gc, gs);
                if (acc) {
                    m2l = true;
                } else if (cleaf && sleaf) {
                    p2p = true;
                    cinter += (unsigned long long)tn * cv.count[s0];
                } else {
                    // the larger cell splits, a leaf never, a tie the earlier one
                    const bool c_splits = sleaf || (!cleaf && ((uint32_t)c < s0 ? gc.w >= gs.w : gc.w > gs.w));
                    if (c_splits) {
                        down = true;
                    } else {
                        load_children(cv, (int)s0, ch);
#pragma unroll
                        for (int o = 0; o < 8; ++o) npush += ch[o] >= 0;
                    }
                }
            }
            // ranks within the group
            const unsigned mm = __ballot_sync(FULL, m2l), mq = __ballot_sync(FULL, p2p), md = __ballot_sync(FULL, down);
            int incl = npush;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            const uint32_t wpush = (uint32_t)__shfl_sync(FULL, incl, 31);
            unsigned long long before = 0, all = pack4(__popc(mm), __popc(mq), __popc(md), wpush);
            if (W > 1) {
                if (lane == 0) wsum[par_w][wid] = all;
                __syncthreads();
                const unsigned long long own = lane < W ? wsum[par_w][lane] : 0ull;
                unsigned long long sc = own;
#pragma unroll
                for (int o = 1; o < W; o <<= 1) {
                    const unsigned long long t = __shfl_up_sync(FULL, sc, o);
                    if (lane >= o) sc += t;
                }
                before = __shfl_sync(FULL, sc, wid) - __shfl_sync(FULL, own, wid);
                all = __shfl_sync(FULL, sc, W - 1);
                par_w ^= 1;
            }
            const uint32_t am = (uint32_t)(all & 0xfff), ap = (uint32_t)((all >> 12) & 0xfff),
                           ad = (uint32_t)((all >> 24) & 0xfff), apush = (uint32_t)(all >> 36);
            if (apush) {
                if (RING && (size + apush > cap || (W == 1 && taken > limit))) {
                    given_up = true;
                    break;
                }
                if (npush > 0) {
                    uint32_t pos = head + size + (uint32_t)(before >> 36) + (uint32_t)(incl - npush);
#pragma unroll
                    for (int o = 0; o < 8; ++o) {
                        if (ch[o] < 0) continue;
                        uint32_t q = pos++;
                        if (q >= cap) q -= cap;
                        ring[q] = (uint32_t)ch[o];
                    }
                }
                size += apush;
            }
            fetch();  // (ahead of the list entries, whose chunks may wait for an atomic)
            const unsigned below = (1u << lane) - 1u;
            const uint32_t qm = lm.chunks(am), qp = lp.chunks(ap), qd = ld.chunks(ad);
            const uint32_t base = qm + qp + qd ? reserve(qm + qp + qd) : 0u;
            if (am)
                list_add(P, lm, am, base, m2l, (uint32_t)(before & 0xfff) + __popc(mm & below), s0, tid == 0,
                         (uint32_t)c, 0u, RING ? 0u : 1u);
            if (ap)
                list_add(P, lp, ap, base + qm, p2p, (uint32_t)((before >> 12) & 0xfff) + __popc(mq & below), s0, tid == 0,
                         (uint32_t)c, 1u, RING ? 0u : 1u);
            if (ad)
                list_add(P, ld, ad, base + qm + qp, down, (uint32_t)((before >> 24) & 0xfff) + __popc(md & below), s0,
                         tid == 0, (uint32_t)c, 2u, RING ? 0u : 1u);
        }
        barrier();
        if (given_up) {
            if (tid == 0) heavy.list[atomicAdd(heavy.count, 1)] = c;
            continue;
        }
        pops += cpops;
        inter += cinter;
        if (tid == 0) {
            nm2l += lm.n;
            np2p += lp.n;
            Ls.down_n[c] = ld.n;
            Ls.down_head[c] = ld.head;
            Ls.redone[c] = RING ? 0 : 1;
            Ls.sizes[c] = near_sizes(lm.n, lp.n, tn, P2P_GRAIN);
        }
    }
    give_back();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        pops += __shfl_xor_sync(FULL, pops, o);
        inter += __shfl_xor_sync(FULL, inter, o);
    }
    if (lane == 0) {
        if (pops) atomicAdd(Ls.totals, pops);
        if (inter) atomicAdd(Ls.totals + 1, inter);
        if (nm2l) atomicAdd(Ls.totals + 2, nm2l);
        if (np2p) atomicAdd(Ls.totals + 3, np2p);
    }
}

// The lists into contiguous arrays, off[c] the exclusive sums of sizes[c]
// (ncells + 1 entries, sizes[ncells] = 0): the first blocks' threads take a cell
// each (offsets, leaves of the work units), then every warp 32 chunks at a time;
// a chunk's owner gives its place, so a list of 10^4 entries is copied by many
// warps (a chunk nobody used has owner ~0). Followed as a chain by one warp per
// cell the longest list took 0.55 ms at N = 3e5 (64 clusters).
__global__ void k_lists_gather(int nc, uint32_t nchunks, WalkPool P, WalkLists Ls, const uint4* __restrict__ off,
                               uint32_t* __restrict__ m2l_off, uint32_t* __restrict__ p2p_off,
                               uint32_t* __restrict__ uoff, uint32_t* __restrict__ soff, uint32_t* __restrict__ m2l,
                               uint32_t* __restrict__ p2p, int32_t* __restrict__ ucell) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= nc; c += gridDim.x * blockDim.x) {
        const uint4 o = off[c];
        m2l_off[c] = o.x;
        p2p_off[c] = o.y;
        uoff[c] = o.z;
        soff[c] = o.w;
        if (c < nc)
            for (uint32_t u = 0; u < Ls.sizes[c].z; ++u) ucell[o.z + u] = c;
    }
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); 32 * b < nchunks; b += warps) {
        // lane: one chunk's place and entries
        const uint32_t id = 32 * b + lane;
        uint32_t dst = 0, n = 0, kind = 0;
        if (id < nchunks && id < P.cap) {  // (the unused tail of a reservation may lie beyond the pool)
            const uint2 w = P.owner[id];
            if (w.x != ~0u) {
                const uint32_t idx = w.y & 0x1fffffffu;
                const uint4 o = off[w.x], sz = Ls.sizes[w.x];
                kind = w.y >> 30;
                const uint32_t len = kind ? sz.y : sz.x;
                // (a heavy cell's first walk, given up, leaves chunks behind)
                if (((w.y >> 29) & 1u) == Ls.redone[w.x] && 32 * idx < len) {
                    dst = (kind ? o.y : o.x) + 32 * idx;
                    n = min(32u, len - 32 * idx);
                }
            }
        }
#pragma unroll 4
        for (int k = 0; k < 32; ++k) {
            const uint32_t nk = __shfl_sync(0xffffffffu, n, k), dk = __shfl_sync(0xffffffffu, dst, k),
                           kk = __shfl_sync(0xffffffffu, kind, k);
            if ((uint32_t)lane < nk) (kk ? p2p : m2l)[dk + lane] = P.entry[(size_t)32 * (32 * b + k) + lane];
        }
    }
}

// Warps per cell, by the cells of the level (per SM), and queue lengths of the
// three forms: 32 warps (128 KB) up to one cell per SM, 8 warps (32 KB) up to
// 16, else a warp (8 KB; 4 KB leaves twice as many heavy cells, clustered
// N = 2^22 33 ms against 22.5; 16 KB a third of the warps, 37 ms). The lines are
// flat: 2 and 32 cells per SM cost the Plummer 2e5 walk 0.40 ms against 0.34 and
// gain the cuspy 1e5 one 0.05 of 1.0. A warp that has taken WK_LIMIT sources
// leaves its cell to the heavy form.
#define WK_T32 1
#define WK_T8 16
#define WK_RING1 2048
#define WK_RING8 8192
#define WK_RING32 32768
#define WK_LIMIT 16384

template <bool DEHNEN, int W, int RING>
static void launch_form(unsigned most, cudaStream_t s, const int32_t* level_cells, int lcnt, CellsView cv,
                        const int32_t* parent, MacParams mp, const double2* rows, WalkPool P,
                        WalkLists Ls, WalkHeavy heavy, int* work, uint32_t limit, uint32_t* gring, uint32_t gcap) {
    auto kern = k_walk_level<DEHNEN, W, RING>;
    constexpr size_t smem = (size_t)RING * sizeof(uint32_t);
    unsigned grid = most;
    uint32_t batch = W == 1 ? 6u : 16u;  // chunks reserved per atomic: a small level wants little waste
    if (RING) {
        if (smem > 48 * 1024)  // (per device, so at every launch)
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        static std::atomic<int> per_sm{0};
        if (per_sm.load() == 0) {
            int b = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, 32 * W, smem) != cudaSuccess || b < 1) b = 1;
            per_sm.store(b);
        }
        const unsigned resident = (unsigned)per_sm.load() * (unsigned)g_nsm;
        grid = std::min((unsigned)lcnt, resident);
        if (W == 1 && (unsigned)lcnt > resident) batch = 16;  // (many warps on one counter: few atomics)
    }
    kern<<<grid, 32 * W, smem, s>>>(level_cells, lcnt, cv, parent, mp, rows, P, Ls, heavy, work, limit, batch,
                                    gring, gcap);
}

template <bool DEHNEN>
static int launch_level(cudaStream_t s, const int32_t* level_cells, int lcnt, int nleaves, CellsView cv,
                        const int32_t* parent, MacParams mp, const double2* rows, WalkPool P,
                        WalkLists Ls, WalkHeavy heavy, int* work, int* heavy_work) {
    // sources waiting at once are disjoint subtrees: a queue of nleaves entries is never full
    bool may_give_up;
    if (lcnt <= WK_T32 * g_nsm) {
        launch_form<DEHNEN, 32, WK_RING32>(0, s, level_cells, lcnt, cv, parent, mp, rows, P, Ls, heavy, work, 0,
                                           nullptr, 0);
        may_give_up = nleaves > WK_RING32;
    } else if (lcnt <= WK_T8 * g_nsm) {
        launch_form<DEHNEN, 8, WK_RING8>(0, s, level_cells, lcnt, cv, parent, mp, rows, P, Ls, heavy, work, 0,
                                         nullptr, 0);
        may_give_up = nleaves > WK_RING8;
    } else {
        launch_form<DEHNEN, 1, WK_RING1>(0, s, level_cells, lcnt, cv, parent, mp, rows, P, Ls, heavy, work, WK_LIMIT,
                                         nullptr, 0);
        may_give_up = true;
    }
    if (!may_give_up) return 1;
    launch_form<DEHNEN, 32, 0>(heavy.blocks, s, nullptr, lcnt, cv, parent, mp, rows, P, Ls, heavy, heavy_work, 0,
                               heavy.ring, heavy.ring_cap);
    return 2;
}

int launch_walk_level(bool dehnen, cudaStream_t s, const int32_t* level_cells, int lcnt, int nleaves, CellsView cv,
                      const int32_t* parent, MacParams mp, const double2* rows, WalkPool P,
                      WalkLists Ls, WalkHeavy heavy, int* work, int* heavy_work) {
    return dehnen ? launch_level<true>(s, level_cells, lcnt, nleaves, cv, parent, mp, rows, P, Ls, heavy, work,
                                       heavy_work)
                  : launch_level<false>(s, level_cells, lcnt, nleaves, cv, parent, mp, rows, P, Ls, heavy, work,
                                        heavy_work);
}

unsigned walk_heavy_blocks(int nleaves) {
    // a block per SM, fewer where their queues would take more than 1 GB
    const uint64_t by_mem = (1ull << 28) / (uint64_t)std::max(nleaves, 1);
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)g_nsm, by_mem));
}
bool walk_needs_heavy(const int* lvl_count, int nlevels, int nleaves) {
    if (nleaves > WK_RING8) return true;
    for (int L = 0; L < nlevels; ++L)
        if (lvl_count[L] > WK_T8 * g_nsm) return true;
    return false;
}

void launch_lists_gather(cudaStream_t s, int nc, uint32_t nchunks, WalkPool P, WalkLists Ls, const uint4* off, uint32_t* m2l_off,
                         uint32_t* p2p_off, uint32_t* uoff, uint32_t* soff, uint32_t* m2l, uint32_t* p2p,
                         int32_t* ucell) {
    k_lists_gather<<<grid_for(std::max<size_t>(nchunks, nc + 1), 256), 256, 0, s>>>(
        nc, nchunks, P, Ls, off, m2l_off, p2p_off, uoff, soff, m2l, p2p, ucell);
}

}  // namespace fmmx
