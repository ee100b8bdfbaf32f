// Bit-exact stages of the engine: bounding box, Morton keys, octree topology,
// cell geometry, P2M/M2M, multipole power and the f pre-pass (the walk with its
// MAC is in walk.cu).
//
// Everything here feeds the multipole acceptance decisions, so it reproduces
// the reference's FP64 operation order exactly and this file is compiled with
// --fmad=false (the reference never contracts a*b+c into an FMA). sqrt and
// division are IEEE round-to-nearest in CUDA double precision, as in the
// reference. Citations are file:line in crates/fmm/src.
#include <float.h>

#include "common.cuh"
#include "kernels.h"

namespace fmmx {

// The order tables in global memory: the kernels read them with lane-
// dependent indices (a lane per order m or per degree), which the constant
// cache would serialise over the distinct addresses; global loads are served
// from L1 in parallel.
static __device__ OrderTables g_tab;

void upload_tables_exact(const OrderTables& t, cudaStream_t s) {
    cudaMemcpyToSymbolAsync(g_tab, &t, sizeof(t), 0, cudaMemcpyHostToDevice, s);
}

// ------------------------------------------------------------ bounding box
// tree.rs:98-111. min/max are exact, so any reduction order gives the same box.
__global__ void k_bbox_partial(const double* __restrict__ pos, size_t n, double* __restrict__ part,
                               int* __restrict__ bad) {
    double lo[3] = {INFINITY, INFINITY, INFINITY};
    double hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    int nonfinite = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double v = pos[3 * i + d];
            nonfinite |= !isfinite(v);
            lo[d] = fmin(lo[d], v);
            hi[d] = fmax(hi[d], v);
        }
    }
    __shared__ double s[6][256];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        s[d][threadIdx.x] = lo[d];
        s[3 + d][threadIdx.x] = hi[d];
    }
    if (nonfinite) atomicOr(bad, 1);
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                s[d][threadIdx.x] = fmin(s[d][threadIdx.x], s[d][threadIdx.x + w]);
                s[3 + d][threadIdx.x] = fmax(s[3 + d][threadIdx.x], s[3 + d][threadIdx.x + w]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int d = 0; d < 6; ++d) part[blockIdx.x * 6 + d] = s[d][0];
}

// box = {lo[3], hi[3], side, inv_side}; side as tree.rs:107-111.
// One warp: lanes reduce strided partials, then a shuffle reduction (min and
// max are exact, so the order does not matter).
__global__ void k_bbox_final(const double* __restrict__ part, int nparts, double* __restrict__ box) {
    if (blockIdx.x != 0 || threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    double lo[3] = {INFINITY, INFINITY, INFINITY};
    double hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int b = lane; b < nparts; b += 32)
        for (int d = 0; d < 3; ++d) {
            lo[d] = fmin(lo[d], part[b * 6 + d]);
            hi[d] = fmax(hi[d], part[b * 6 + 3 + d]);
        }
    for (int o = 16; o > 0; o >>= 1)
        for (int d = 0; d < 3; ++d) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    if (lane != 0) return;
    double side = fmax(fmax(fmax(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]), DBL_MIN);
    for (int d = 0; d < 3; ++d) {
        box[d] = lo[d];
        box[3 + d] = hi[d];
    }
    box[6] = side;
    box[7] = 1.0 / side;
}

// The system of a forest that holds input i: the last one with off[sys] <= i.
__device__ __forceinline__ int system_of(const uint64_t* __restrict__ off, int nsys, size_t i) {
    int lo = 0, hi = nsys;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Order-preserving encoding of a double as an unsigned integer.
__device__ __forceinline__ unsigned long long enc_order(double v) {
    const long long b = __double_as_longlong(v);
    return b < 0 ? ~(unsigned long long)b : (unsigned long long)b | 0x8000000000000000ull;
}
__device__ __forceinline__ double dec_order(unsigned long long u) {
    return __longlong_as_double((long long)((u & 0x8000000000000000ull) ? u & 0x7fffffffffffffffull : ~u));
}

// Boxes of a forest of independent systems (segments [off[s], off[s+1]) of the
// input): every block reduces BBOX_CHUNK consecutive bodies, system by system,
// into enc[6 s ..] = minima of the encoded lo and -hi (all bits set at the
// start); minima are exact, so the order does not matter. (One block per
// system took 221 us for 48 systems of together 10^6 bodies: the largest
// system's block ran alone.)
__global__ void k_bbox_seg(const double* __restrict__ pos, size_t n, const uint64_t* __restrict__ off, int nsys,
                           unsigned long long* __restrict__ enc, int* __restrict__ bad) {
    const size_t b0 = (size_t)blockIdx.x * BBOX_CHUNK, e0 = min(n, b0 + BBOX_CHUNK);
    __shared__ unsigned long long sh[6][8];
    for (int sys = system_of(off, nsys, b0); sys < nsys && off[sys] < e0; ++sys) {
        const size_t b = max((size_t)off[sys], b0), e = min((size_t)off[sys + 1], e0);
        double v[6] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY};
        int nonfinite = 0;
        for (size_t i = b + threadIdx.x; i < e; i += blockDim.x) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double q = pos[3 * i + d];
                nonfinite |= !isfinite(q);
                v[d] = fmin(v[d], q);
                v[3 + d] = fmin(v[3 + d], -q);
            }
        }
        if (nonfinite) atomicOr(bad, 1);
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int d = 0; d < 6; ++d) v[d] = fmin(v[d], __shfl_xor_sync(0xffffffffu, v[d], o));
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int d = 0; d < 6; ++d) sh[d][threadIdx.x >> 5] = enc_order(v[d]);
        __syncthreads();
        if (threadIdx.x < 6) {
            unsigned long long m = sh[threadIdx.x][0];
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = min(m, sh[threadIdx.x][w]);
            atomicMin(enc + 6 * sys + threadIdx.x, m);
        }
        __syncthreads();
    }
}
__global__ void k_bbox_seg_final(const unsigned long long* __restrict__ enc, int nsys, double* __restrict__ box) {
    for (int sys = blockIdx.x * blockDim.x + threadIdx.x; sys < nsys; sys += gridDim.x * blockDim.x) {
        double* bx = box + 8 * sys;
        for (int d = 0; d < 3; ++d) {
            bx[d] = dec_order(enc[6 * sys + d]);
            bx[3 + d] = -dec_order(enc[6 * sys + 3 + d]);
        }
        const double side = fmax(fmax(fmax(bx[3] - bx[0], bx[4] - bx[1]), bx[5] - bx[2]), DBL_MIN);
        bx[6] = side;
        bx[7] = 1.0 / side;
    }
}

// ------------------------------------------------------------ Morton keys
// dilate, tree.rs:28-35
__device__ __forceinline__ uint64_t dilate21(uint64_t x) {
    x &= (1ULL << FMMX_BITS) - 1;
    x = (x | (x << 32)) & 0x001f00000000ffffULL;
    x = (x | (x << 16)) & 0x001f0000ff0000ffULL;
    x = (x | (x << 8)) & 0x100f00f00f00f00fULL;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ULL;
    return (x | (x << 2)) & 0x1249249249249249ULL;
}

// morton_key, tree.rs:37-46: every axis is quantised against lo[0].
__device__ __forceinline__ uint64_t quant(double c, double lo0, double inv_side) {
    double v = (c - lo0) * inv_side;
    if (v != v) return 0;
    v = v < 0.0 ? 0.0 : (v > 1.0 ? 1.0 : v);
    return (uint64_t)(v * (double)((1ULL << FMMX_BITS) - 1));
}

__global__ void k_keys(const double* __restrict__ pos, size_t n, const double* __restrict__ box,
                       uint64_t* __restrict__ keys, uint32_t* __restrict__ idx) {
    const double lo0 = box[0], inv = box[7];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        uint64_t k = dilate21(quant(pos[3 * i + 2], lo0, inv));
        k |= dilate21(quant(pos[3 * i + 1], lo0, inv)) << 1;
        k |= dilate21(quant(pos[3 * i + 0], lo0, inv)) << 2;
        keys[i] = k;
        idx[i] = (uint32_t)i;
    }
}

// Keys of a forest: each body is quantised in its own system's box.
__global__ void k_keys_seg(const double* __restrict__ pos, size_t n, const uint64_t* __restrict__ off, int nsys,
                           const double* __restrict__ box, uint64_t* __restrict__ keys, uint32_t* __restrict__ idx) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int sys = system_of(off, nsys, i);
        const double lo0 = box[8 * sys], inv = box[8 * sys + 7];
        uint64_t k = dilate21(quant(pos[3 * i + 2], lo0, inv));
        k |= dilate21(quant(pos[3 * i + 1], lo0, inv)) << 1;
        k |= dilate21(quant(pos[3 * i + 0], lo0, inv)) << 2;
        keys[i] = k;
        idx[i] = (uint32_t)i;
    }
}

// Bodies::from_parts / gather_into, bodies.rs:27-60: slot k <- particle order[k].
__global__ void k_gather(const double* __restrict__ pos, const double* __restrict__ mass,
                         const uint32_t* __restrict__ order, size_t n, double* __restrict__ x, double* __restrict__ y,
                         double* __restrict__ z, double* __restrict__ m) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        uint32_t id = order[k];
        x[k] = pos[3 * (size_t)id];
        y[k] = pos[3 * (size_t)id + 1];
        z[k] = pos[3 * (size_t)id + 2];
        m[k] = mass[id];
    }
}

// System of each entry of `order` (sorted by key over the whole forest) and its
// position, for the second, stable sort by system; then keys and order in that
// sort's order.
__global__ void k_entry_system(const uint32_t* __restrict__ order, size_t n, const uint64_t* __restrict__ off, int nsys,
                               uint32_t* __restrict__ sys, uint32_t* __restrict__ at) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        sys[i] = (uint32_t)system_of(off, nsys, order[i]);
        at[i] = (uint32_t)i;
    }
}
__global__ void k_permute_entries(const uint32_t* __restrict__ at, size_t n, const uint64_t* __restrict__ keys_in,
                                  const uint32_t* __restrict__ order_in, uint64_t* __restrict__ keys,
                                  uint32_t* __restrict__ order) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t q = at[i];
        keys[i] = keys_in[q];
        order[i] = order_in[q];
    }
}

// ------------------------------------------------------------ topology
// The reference builds cells by depth-first recursion (build_rec,
// tree.rs:404-445). Here every cell is found from the sorted keys alone, all
// levels at once. A cell is a block of slots whose keys share their first L
// octal digits; it exists if its parent (the block one digit shorter) holds
// more than n_leaf bodies, and is split again while it does so itself, down to
// level 21. With
//   d_i = the digits slot i shares with slot i - 1 (-1 at a system's start) and
//   w_i = the digits slot i shares with slot i + n_leaf (-1: another system),
// the blocks that start at slot i are those of levels above d_i; one of them
// holds more than n_leaf bodies up to level w_i, and the block of level d_i
// around slot i, the parent of the first, is looked up where w_i does not
// decide. So slot i starts the cells of levels d_i + 1 .. min(21, m_i + 1),
// m_i the deepest level whose block around i is over-full, and the last of them
// is a leaf. Depth-first pre-order is the order of (first slot, level): a
// prefix sum of the counts numbers the cells, and body i's leaf is the last cell
// that starts at or before it. (The build used to run a launch per level, a
// binary search per octant and thread, and a radix sort into depth-first order:
// N = 2e5, 10 levels, 0.46 ms for the levels and 0.1 ms for the order.)
__device__ __forceinline__ int common_digits(uint64_t a, uint64_t b) {
    const uint64_t x = a ^ b;
    return x ? (__clzll((long long)x) - 1) / 3 : FMMX_MAXLEVEL;
}

// the slots [beg, end) of the system that holds slot i
__device__ __forceinline__ void system_range(const uint64_t* __restrict__ off, int nsys, uint32_t n, uint32_t i,
                                             uint32_t& beg, uint32_t& end) {
    beg = 0;
    end = n;
    if (nsys > 1) {
        const int s = system_of(off, nsys, i);
        beg = (uint32_t)off[s];
        end = (uint32_t)off[s + 1];
    }
}

// first slot of [lo, i] that shares at least L digits with slot i
__device__ __forceinline__ uint32_t block_begin(const uint64_t* __restrict__ keys, uint32_t lo, uint32_t i, int L) {
    const uint64_t k = keys[i];
    while (lo < i) {
        const uint32_t mid = lo + ((i - lo) >> 1);
        if (common_digits(keys[mid], k) >= L) i = mid;
        else lo = mid + 1;
    }
    return i;
}
// first slot of (i, hi] that shares fewer than L digits with slot i (hi if none)
__device__ __forceinline__ uint32_t block_end(const uint64_t* __restrict__ keys, uint64_t k, uint32_t lo, uint32_t hi,
                                              int L) {
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (common_digits(keys[mid], k) >= L) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Cells that start at each slot (count[n] = 0 for the prefix sum), the cells
// of each level and the number of leaves (lvl[0 .. 21] and lvl[22], zero at
// the start).
__global__ void __launch_bounds__(TREE_BLOCK) k_cell_count(const uint64_t* __restrict__ keys, uint32_t n,
                                                           const uint64_t* __restrict__ off, int nsys,
                                                           uint32_t n_leaf, uint32_t* __restrict__ count,
                                                           int* __restrict__ lvl) {
    __shared__ int hist[FMMX_NLEVELS + 1];
    if (threadIdx.x <= FMMX_NLEVELS) hist[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * (uint32_t)(TREE_BLOCK * TREE_PER_THREAD) + threadIdx.x;
    for (int q = 0; q < TREE_PER_THREAD; ++q) {
        const uint32_t i = base + q * TREE_BLOCK;
        if (i > n) break;
        uint32_t c = 0;
        if (i < n) {
            uint32_t beg, end;
            system_range(off, nsys, n, i, beg, end);
            const uint64_t k = keys[i];
            const int d = i == beg ? -1 : common_digits(keys[i - 1], k);
            const int w = n_leaf < end - i ? common_digits(keys[i + n_leaf], k) : -1;
            int m = w;  // deepest over-full block around i
            if (w <= d) {
                m = -2;
                if (d < 0) {
                    m = -1;  // a root exists whatever it holds
                } else {
                    const uint32_t lo = i - beg > n_leaf ? i - n_leaf : beg;
                    const uint32_t s = block_begin(keys, lo, i, d);
                    // more than n_leaf bodies: the block begins before `lo`, or reaches slot s + n_leaf
                    const bool over = n_leaf < end - s && common_digits(keys[s + n_leaf], k) >= d;
                    if (over) m = d;
                }
            }
            if (m >= d) {
                const int last = min(FMMX_MAXLEVEL, m + 1);
                c = (uint32_t)(last - d);
                for (int L = d + 1; L <= last; ++L) atomicAdd(&hist[L], 1);
                if (c) atomicAdd(&hist[FMMX_NLEVELS], 1);
            }
        }
        count[i] = c;
    }
    __syncthreads();
    if (threadIdx.x <= FMMX_NLEVELS && hist[threadIdx.x]) atomicAdd(&lvl[threadIdx.x], hist[threadIdx.x]);
}

// The cells in depth-first order (id0: the prefix sum of k_cell_count's
// counts), the level lists (roots in system order, else arbitrary; cursor[22]
// zero at the start), the bodies' leaves and the cells' box sizes.
__global__ void __launch_bounds__(TREE_BLOCK) k_cell_emit(const uint64_t* __restrict__ keys, uint32_t n,
                                                          const uint64_t* __restrict__ off, int nsys, uint32_t n_leaf,
                                                          const uint32_t* __restrict__ id0, LevelStarts ls,
                                                          int* __restrict__ cursor, const double* __restrict__ box,
                                                          CellsMut cells, int32_t* __restrict__ level_cells,
                                                          int32_t* __restrict__ body_leaf, double* __restrict__ h) {
    __shared__ int hist[FMMX_NLEVELS], lbase[FMMX_NLEVELS];
    if (threadIdx.x < FMMX_NLEVELS) hist[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * (uint32_t)(TREE_BLOCK * TREE_PER_THREAD) + threadIdx.x;
    for (int q = 0; q < TREE_PER_THREAD; ++q) {  // this block's cells of each level
        const uint32_t i = base + q * TREE_BLOCK;
        if (i >= n) break;
        const uint32_t c0 = id0[i], c1 = id0[i + 1];
        body_leaf[i] = (int32_t)c1 - 1;
        if (c0 == c1) continue;
        uint32_t beg, end;
        system_range(off, nsys, n, i, beg, end);
        const int d = i == beg ? -1 : common_digits(keys[i - 1], keys[i]);
        for (uint32_t c = c0; c < c1; ++c) atomicAdd(&hist[d + 1 + (int)(c - c0)], 1);
    }
    __syncthreads();
    if (threadIdx.x < FMMX_NLEVELS) {
        const int v = hist[threadIdx.x];
        lbase[threadIdx.x] = ls.start[threadIdx.x] + (v ? atomicAdd(&cursor[threadIdx.x], v) : 0);
        hist[threadIdx.x] = 0;
    }
    __syncthreads();
    for (int q = 0; q < TREE_PER_THREAD; ++q) {
        const uint32_t i = base + q * TREE_BLOCK;
        if (i >= n) break;
        const uint32_t c0 = id0[i], c1 = id0[i + 1];
        if (c0 == c1) continue;
        int sys = 0;
        uint32_t beg = 0, end = n;
        if (nsys > 1) {
            sys = system_of(off, nsys, i);
            beg = (uint32_t)off[sys];
            end = (uint32_t)off[sys + 1];
        }
        const uint64_t k = keys[i];
        const int d = i == beg ? -1 : common_digits(keys[i - 1], k);
        int par = -1;
        if (d >= 0) {  // the block of level d around slot i
            const uint32_t s = block_begin(keys, beg, i, d);
            const int ds = s == beg ? -1 : common_digits(keys[s - 1], keys[s]);
            par = (int)id0[s] + d - ds - 1;
        }
        const double side = box[8 * sys + 6];
        uint32_t e = end;
        for (uint32_t c = c0; c < c1; ++c) {
            const int L = d + 1 + (int)(c - c0);
            const bool leaf = c + 1 == c1;
            // bounds of the block's end: a leaf above level 21 holds at most n_leaf bodies, an internal cell more
            uint32_t lo = i + 1, hi = e;
            if (leaf && L < FMMX_MAXLEVEL) hi = min(hi, i + max(n_leaf, 1u));
            else if (!leaf) lo = i + n_leaf + 1;
            e = block_end(keys, k, lo, hi, L);
            cells.first[c] = i;
            cells.count[c] = e - i;
            cells.level[c] = (uint8_t)L;
            cells.leaf[c] = leaf ? 1 : 0;
            cells.parent[c] = par;
            if (par >= 0) cells.child[8 * (size_t)par + ((k >> (3 * (FMMX_MAXLEVEL - L))) & 7)] = (int32_t)c;
            h[c] = ldexp(side, -L);
            if (L == 0) level_cells[sys] = (int32_t)c;
            else level_cells[lbase[L] + atomicAdd(&hist[L], 1)] = (int32_t)c;
            par = (int)c;
        }
    }
}

// ------------------------------------------------------------ geometry
__device__ __forceinline__ double dist3(double ax, double ay, double az, double bx, double by, double bz) {
    double dx = ax - bx, dy = ay - by, dz = az - bz;
    return sqrt(dx * dx + dy * dy + dz * dz);
}
__device__ __forceinline__ double dist2_3(double ax, double ay, double az, double bx, double by, double bz) {
    double dx = ax - bx, dy = ay - by, dz = az - bz;
    return dx * dx + dy * dy + dz * dz;
}

// Item accessors for the Ritter sphere: leaf bodies (radius 0) or child cells.
struct LeafItems {
    const double *x, *y, *z;
    uint32_t first, count;
    __device__ int size() const { return (int)count; }
    __device__ void get(int i, double& cx, double& cy, double& cz, double& r) const {
        cx = x[first + i];
        cy = y[first + i];
        cz = z[first + i];
        r = 0.0;
    }
};
struct ChildItems {
    int ids[8];
    int nitems;
    const double *cx, *cy, *cz, *rho;
    __device__ int size() const { return nitems; }
    __device__ void get(int i, double& x, double& y, double& z, double& r) const {
        int c = ids[i];
        x = cx[c];
        y = cy[c];
        z = cz[c];
        r = rho[c];
    }
};

// Ritter grow/enclose sphere, tree.rs:290-389 (operation order kept).
template <class Items>
__device__ void ritter(const Items& it, double cen[3]) {
    int n = it.size();
    int a = 0, b = 0;
    double best = -1.0;
    double ax, ay, az, ar, qx, qy, qz, qr;
    it.get(a, ax, ay, az, ar);
    for (int i = 0; i < n; ++i) {
        it.get(i, qx, qy, qz, qr);
        double d2 = dist2_3(qx, qy, qz, ax, ay, az);
        if (d2 > best) { best = d2; b = i; }
    }
    a = b;
    best = -1.0;
    it.get(a, ax, ay, az, ar);
    for (int i = 0; i < n; ++i) {
        it.get(i, qx, qy, qz, qr);
        double d2 = dist2_3(qx, qy, qz, ax, ay, az);
        if (d2 > best) { best = d2; b = i; }
    }
    double pa[3], pb[3], ra, rb_;
    it.get(a, pa[0], pa[1], pa[2], ra);
    it.get(b, pb[0], pb[1], pb[2], rb_);
    double dir[3];
    {
        double dx = pb[0] - pa[0], dy = pb[1] - pa[1], dz = pb[2] - pa[2];
        double d = fmax(sqrt(dx * dx + dy * dy + dz * dz), DBL_MIN);
        dir[0] = dx / d; dir[1] = dy / d; dir[2] = dz / d;
    }
    double fa[3] = {pa[0] + ra * dir[0], pa[1] + ra * dir[1], pa[2] + ra * dir[2]};
    double fb[3] = {pb[0] - rb_ * dir[0], pb[1] - rb_ * dir[1], pb[2] - rb_ * dir[2]};
    double c[3] = {(fa[0] + fb[0]) * 0.5, (fa[1] + fb[1]) * 0.5, (fa[2] + fb[2]) * 0.5};
    double r = dist3(fa[0], fa[1], fa[2], fb[0], fb[1], fb[2]) * 0.5;
    for (int pass = 0; pass < 2; ++pass) {
        for (int i = 0; i < n; ++i) {
            it.get(i, qx, qy, qz, qr);
            double d = dist3(qx, qy, qz, c[0], c[1], c[2]);
            if (d + qr > r) {
                double dd = fmax(d, DBL_MIN);
                double dv[3] = {(qx - c[0]) / dd, (qy - c[1]) / dd, (qz - c[2]) / dd};
                double pp[3] = {qx + qr * dv[0], qy + qr * dv[1], qz + qr * dv[2]};
                double d_far = d + qr;
                double t = (d_far - r) / (2.0 * d_far);
                for (int k = 0; k < 3; ++k) c[k] += t * (pp[k] - c[k]);
                r = (d_far + r) * 0.5;
            }
        }
    }
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = 0; i < n; ++i) {
        it.get(i, qx, qy, qz, qr);
        double q[3] = {qx, qy, qz};
        for (int d = 0; d < 3; ++d) {
            lo[d] = fmin(lo[d], q[d] - qr);
            hi[d] = fmax(hi[d], q[d] + qr);
        }
    }
    double cb[3] = {(lo[0] + hi[0]) * 0.5, (lo[1] + hi[1]) * 0.5, (lo[2] + hi[2]) * 0.5};
    double rbb = 0.0;
    for (int i = 0; i < n; ++i) {
        it.get(i, qx, qy, qz, qr);
        rbb = fmax(rbb, dist3(qx, qy, qz, cb[0], cb[1], cb[2]) + qr);
    }
    if (rbb < r) {
        cen[0] = cb[0]; cen[1] = cb[1]; cen[2] = cb[2];
    } else {
        cen[0] = c[0]; cen[1] = c[1]; cen[2] = c[2];
    }
}

// Octree::geometry with Ritter centres, tree.rs:152-227, one level at a time from
// the deepest, a thread per cell (each sphere is a serial scan of its items;
// centres of mass: k_geometry_com).
__global__ void k_geometry_ritter(const int32_t* __restrict__ level_cells, int lstart, int lcnt, CellsMut cells,
                                  const double* __restrict__ x, const double* __restrict__ y,
                                  const double* __restrict__ z, const double* __restrict__ m) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < lcnt; j += gridDim.x * blockDim.x) {
        const int c = level_cells[lstart + j];
        double mass = 0.0, cen[3], rho = 0.0;
        if (cells.leaf[c]) {
            const uint32_t f = cells.first[c], e = f + cells.count[c];
            for (uint32_t k = f; k < e; ++k) mass += m[k];
            LeafItems it{x, y, z, f, e - f};
            ritter(it, cen);
            for (uint32_t k = f; k < e; ++k) rho = fmax(rho, dist3(x[k], y[k], z[k], cen[0], cen[1], cen[2]));
        } else {
            const int32_t* ch = cells.child + 8 * (size_t)c;
            ChildItems it;
            it.nitems = 0;
            for (int o = 0; o < 8; ++o)
                if (ch[o] >= 0) {
                    mass += cells.mass[ch[o]];
                    it.ids[it.nitems++] = ch[o];
                }
            it.cx = cells.cx;
            it.cy = cells.cy;
            it.cz = cells.cz;
            it.rho = cells.rho;
            ritter(it, cen);
            for (int o = 0; o < 8; ++o) {
                int q = ch[o];
                if (q < 0) continue;
                rho = fmax(rho, cells.rho[q] + dist3(cells.cx[q], cells.cy[q], cells.cz[q], cen[0], cen[1], cen[2]));
            }
        }
        cells.mass[c] = mass;
        cells.cx[c] = cen[0];
        cells.cy[c] = cen[1];
        cells.cz[c] = cen[2];
        cells.rho[c] = rho;
    }
}

// Octree::geometry with centres of mass, tree.rs:152-227, in one launch: a
// warp per leaf, then up the tree -- the warp that finishes a cell's last child
// goes on with the cell, so nobody waits. The sums run in the reference's order
// (bodies in slot order, children in octant order): the lanes form the terms of
// 32 bodies side by side and lanes 0..3 add one component each; rho is the
// square root of the largest squared distance (the root is monotone and
// correctly rounded, so it is the largest distance). Bound by the latency of
// the FP64 add chains and of one L2 round trip per level. A thread per cell and
// a launch per level took 0.27 ms at N = 2e5 (10 levels) and 0.11 ms at 2^20.
// arrive: one zero per cell.
__global__ void __launch_bounds__(32 * GEO_WARPS) k_geometry_com(int nc, CellsMut cells, const double* __restrict__ x,
                                                                 const double* __restrict__ y,
                                                                 const double* __restrict__ z,
                                                                 const double* __restrict__ m,
                                                                 unsigned* __restrict__ arrive,
                                                                 double4* __restrict__ geo) {
    __shared__ double buf_all[GEO_WARPS][4][33];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double(*buf)[33] = buf_all[threadIdx.x >> 5];
    const int nwarps = gridDim.x * GEO_WARPS;
    for (int c0 = blockIdx.x * GEO_WARPS + (threadIdx.x >> 5); c0 < nc; c0 += nwarps) {
        if (!cells.leaf[c0]) continue;
        int c = c0;
        {
            const uint32_t f = cells.first[c], cnt = cells.count[c];
            double s = 0.0;  // lanes 0..3: mass, m x, m y, m z
            double bx = 0, by = 0, bz = 0;
            for (uint32_t b0 = 0; b0 < cnt; b0 += 32) {
                const int nb = (int)min(32u, cnt - b0);
                if (lane < nb) {
                    const uint32_t k = f + b0 + lane;
                    bx = x[k];
                    by = y[k];
                    bz = z[k];
                    const double mk = m[k];
                    buf[0][lane] = mk;
                    buf[1][lane] = mk * bx;
                    buf[2][lane] = mk * by;
                    buf[3][lane] = mk * bz;
                }
                __syncwarp();
                if (lane < 4)
                    for (int k = 0; k < nb; ++k) s += buf[lane][k];
                __syncwarp();
            }
            const double mass = __shfl_sync(FULL, s, 0);
            const double q = s / mass;
            const double cx = __shfl_sync(FULL, q, 1), cy = __shfl_sync(FULL, q, 2), cz = __shfl_sync(FULL, q, 3);
            double d2 = 0.0;
            for (uint32_t b0 = 0; b0 < cnt; b0 += 32) {
                if (b0 + lane < cnt) {
                    if (cnt > 32) {
                        const uint32_t k = f + b0 + lane;
                        bx = x[k];
                        by = y[k];
                        bz = z[k];
                    }
                    d2 = fmax(d2, dist2_3(bx, by, bz, cx, cy, cz));
                }
            }
            for (int o = 16; o > 0; o >>= 1) d2 = fmax(d2, __shfl_xor_sync(FULL, d2, o));
            if (lane == 0) {
                const double rho = sqrt(d2);
                cells.mass[c] = mass;
                cells.cx[c] = cx;
                cells.cy[c] = cy;
                cells.cz[c] = cz;
                cells.rho[c] = rho;
                geo[c] = make_double4(cx, cy, cz, -rho);  // the sign marks a leaf
            }
        }
        for (int par = cells.parent[c]; par >= 0; par = cells.parent[c]) {
            const int ch = lane < 8 ? cells.child[8 * (size_t)par + lane] : -1;
            const unsigned have = __ballot_sync(FULL, ch >= 0);
            unsigned prev = 0;
            if (lane == 0) {
                __threadfence();  // this cell's values before the arrival
                prev = atomicAdd(&arrive[par], 1u);
            }
            prev = __shfl_sync(FULL, prev, 0);
            if (prev + 1 != (unsigned)__popc(have)) break;  // a sibling's warp goes on
            __threadfence();
            // the children's values come from other SMs: read past the L1
            double cm = 0, cx = 0, cy = 0, cz = 0, cr = 0;
            if (ch >= 0) {
                cm = __ldcg(cells.mass + ch);
                cx = __ldcg(cells.cx + ch);
                cy = __ldcg(cells.cy + ch);
                cz = __ldcg(cells.cz + ch);
                cr = __ldcg(cells.rho + ch);
            }
            const double px = cm * cx, py = cm * cy, pz = cm * cz;
            double mass = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
#pragma unroll
            for (int o = 0; o < 8; ++o) {
                const double vm = __shfl_sync(FULL, cm, o), vx = __shfl_sync(FULL, px, o),
                             vy = __shfl_sync(FULL, py, o), vz = __shfl_sync(FULL, pz, o);
                if ((have >> o) & 1) {
                    mass += vm;
                    sx += vx;
                    sy += vy;
                    sz += vz;
                }
            }
            sx /= mass;
            sy /= mass;
            sz /= mass;
            double rho = ch >= 0 ? cr + dist3(cx, cy, cz, sx, sy, sz) : 0.0;
            for (int o = 4; o > 0; o >>= 1) rho = fmax(rho, __shfl_xor_sync(FULL, rho, o));
            c = par;
            if (lane == 0) {
                rho = fmax(rho, 0.0);
                cells.mass[c] = mass;
                cells.cx[c] = sx;
                cells.cy[c] = sy;
                cells.cz[c] = sz;
                cells.rho[c] = rho;
                geo[c] = make_double4(sx, sy, sz, rho);
            }
        }
    }
}

// ------------------------------------------------------------ upward pass
__device__ __forceinline__ void split_nm(int e, int& n, int& m) {
    int q = (int)sqrt((double)e);
    while (q * q > e) --q;
    while ((q + 1) * (q + 1) <= e) ++q;
    n = q;
    m = e - q * (q + 1);
}

// Υ column m for r = (dx,dy,dz), into u (full table when mirror is set):
// upsilon_table_into, harmonic.rs:141-173, operation order kept.
__device__ __forceinline__ void upsilon_column(double dx, double dy, double dz, double r2, int p, int m, zd* u) {
    zd d = mk(1.0, 0.0);
    for (int j = 1; j <= m; ++j) d = zmul(zscale(mk(dx, dy), g_tab.inv2m[j]), d);
    u[cidx(m, m)] = d;
    zd u1 = d, u2 = mk(0.0, 0.0);
    for (int n = m + 1; n <= p; ++n) {
        double a = (double)(2 * n - 1) * dz;
        zd t = zscale(u1, a);
        if (n >= m + 2) t = zsub(t, zscale(u2, r2));
        zd un = zscale(t, g_tab.invc[n][m]);
        u[cidx(n, m)] = un;
        u2 = u1;
        u1 = un;
    }
    if (m > 0) {
        double sgn = (m % 2 == 0) ? 1.0 : -1.0;
        for (int n = m; n <= p; ++n) u[cidx(n, -m)] = zscale(zconj(u[cidx(n, m)]), sgn);
    }
}

// Shared memory of k_upward_exact per warp: the cell's accumulator (dim
// complex), then the m >= 0 Υ tables of a round of B bodies, entry-major in
// separate real and imaginary arrays of stride B + 1 (conflict-free both when a
// lane writes its body's table and when lanes read one body's entries).
__host__ __device__ size_t upward_exact_smem_per_warp(int p) {
    const int B = p2m_round(p), H = (p + 1) * (p + 2) / 2;
    return (size_t)dimp(p) * sizeof(zd) + 2 * (size_t)H * (B + 1) * sizeof(double);
}

// The leaves among the given cells, a warp each (all levels in one launch; the
// internal cells follow level by level in k_m2m_exact_block): P2M (p2m_cell,
// moments.rs:30-53), then the multipole power (:150-168).
//
// P2M: the lanes build the Υ tables of B bodies at once (a lane per body, the
// recursion of upsilon_table_into, harmonic.rs:141-173); then each lane owns
// the m >= 0 coefficients e = lane, lane + 32, ... and adds m_k Υ_k[e] over
// the round's bodies in slot order, so every coefficient is the reference's
// sum in the reference's order.
__global__ void k_upward_exact(const int32_t* __restrict__ level_cells, int lstart, int lcnt, CellsView cells,
                               const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, const double* __restrict__ m, int p,
                               zd* __restrict__ moments, double* __restrict__ pows) {
    extern __shared__ unsigned char smem_raw[];
    const int dim = dimp(p);
    const int H = (p + 1) * (p + 2) / 2;
    const int B = p2m_round(p), S = B + 1;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    unsigned char* wbase = smem_raw + (size_t)wib * upward_exact_smem_per_warp(p);
    zd* acc = reinterpret_cast<zd*>(wbase);
    double* tre = reinterpret_cast<double*>(acc + dim);  // Υ tables, real parts
    double* tim = tre + (size_t)H * S;                   //      imaginary parts
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int j = warp; j < lcnt; j += nwarps) {
        const int c = level_cells[lstart + j];
        if (!cells.leaf[c]) continue;
        const double zx = cells.cx[c], zy = cells.cy[c], zz = cells.cz[c];
        for (int e = lane; e < dim; e += 32) acc[e] = mk(0.0, 0.0);
        __syncwarp();
        {
            const uint32_t fst = cells.first[c], end = fst + cells.count[c];
            double ar[8], ai[8];  // this lane's coefficients e = lane + 32 t (m >= 0 half, H <= 231)
#pragma unroll
            for (int t = 0; t < 8; ++t) ar[t] = ai[t] = 0.0;
            for (uint32_t k0 = fst; k0 < end; k0 += B) {
                const int nb = (int)min((uint32_t)B, end - k0);
                if (lane < nb) {
                    const uint32_t k = k0 + lane;
                    const double dx = x[k] - zx, dy = y[k] - zy, dz = z[k] - zz;
                    const double r2 = dx * dx + dy * dy + dz * dz;
                    zd d = mk(1.0, 0.0);
                    for (int mm = 0; mm <= p; ++mm) {
                        if (mm > 0) d = zmul(zscale(mk(dx, dy), g_tab.inv2m[mm]), d);
                        int h = mm * (mm + 1) / 2 + mm;  // half index of (mm, mm)
                        tre[h * S + lane] = d.re;
                        tim[h * S + lane] = d.im;
                        zd u1 = d, u2 = mk(0.0, 0.0);
                        for (int n = mm + 1; n <= p; ++n) {
                            const double a = (double)(2 * n - 1) * dz;
                            zd t = zscale(u1, a);
                            if (n >= mm + 2) t = zsub(t, zscale(u2, r2));
                            const zd un = zscale(t, g_tab.invc[n][mm]);
                            h += n;  // half index of (n, mm)
                            tre[h * S + lane] = un.re;
                            tim[h * S + lane] = un.im;
                            u2 = u1;
                            u1 = un;
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const int e = lane + 32 * t;
                    if (e < H) {
                        for (int b = 0; b < nb; ++b) {
                            const double mk_ = m[k0 + b];
                            ar[t] += tre[e * S + b] * mk_;
                            ai[t] += tim[e * S + b] * mk_;
                        }
                    }
                }
                __syncwarp();
            }
            // the m >= 0 sums into the full layout; negative orders mirror
            // exactly (every increment of M_n^{-m} is (-1)^m conj of the
            // M_n^m increment)
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int e = lane + 32 * t;
                if (e < H) {
                    int n = 0;
                    while ((n + 1) * (n + 2) / 2 <= e) ++n;
                    const int mm = e - n * (n + 1) / 2;
                    acc[cidx(n, mm)] = mk(ar[t], ai[t]);
                }
            }
            __syncwarp();
            for (int e = lane; e < dim; e += 32) {
                int n, mm;
                split_nm(e, n, mm);
                if (mm < 0) {
                    double sgn = ((-mm) % 2 == 0) ? 1.0 : -1.0;
                    acc[e] = zscale(zconj(acc[cidx(n, -mm)]), sgn);
                }
            }
            __syncwarp();
        }
        zd* out = moments + (size_t)c * dim;
        for (int e = lane; e < dim; e += 32) out[e] = acc[e];
        for (int n = lane; n <= p; n += 32) {
            double s = 0.0;
            for (int mm = -n; mm <= n; ++mm) {
                int am = mm < 0 ? -mm : mm;
                zd v = acc[cidx(n, mm)];
                double w = g_tab.fact[n - am] * g_tab.fact[n + am];
                s += w * (v.re * v.re + v.im * v.im);
            }
            pows[(size_t)c * (p + 1) + n] = sqrt(s);
        }
        __syncwarp();
    }
}

// M2M of the internal cells of a level, one block per cell:
// the Υ tables of the (up to 8) child offsets and each child's convolution
// sums s_o[e] (8 dim independent chains) are computed side by side; then
// every coefficient adds its children's sums in octant order, as m2m_cell
// (moments.rs:56-90) does one child after the other. Power as in
// k_upward_exact. Shared memory: 16 dim complex.
__global__ void __launch_bounds__(M2M_EXACT_WIDE) k_m2m_exact_block(const int32_t* __restrict__ level_cells, int lstart,
                                                         int lcnt, CellsView cells, int p, zd* __restrict__ moments,
                                                         double* __restrict__ pows) {
    extern __shared__ unsigned char smem_raw[];
    const int dim = dimp(p);
    zd* ut = reinterpret_cast<zd*>(smem_raw);  // 8 Υ tables
    zd* st = ut + 8 * dim;                      // 8 child sums
    __shared__ int ch[8];
    const int tid = threadIdx.x;
    for (int j = blockIdx.x; j < lcnt; j += gridDim.x) {
        const int c = level_cells[lstart + j];
        if (cells.leaf[c]) continue;  // uniform: the whole block skips
        if (tid < 8) ch[tid] = cells.child[8 * c + tid];
        __syncthreads();
        const double zx = cells.cx[c], zy = cells.cy[c], zz = cells.cz[c];
        for (int t = tid; t < 8 * (p + 1); t += blockDim.x) {
            const int o = t / (p + 1), mm = t % (p + 1);
            const int cc = ch[o];
            if (cc < 0) continue;
            const double dx = cells.cx[cc] - zx, dy = cells.cy[cc] - zy, dz = cells.cz[cc] - zz;
            const double r2 = dx * dx + dy * dy + dz * dz;
            upsilon_column(dx, dy, dz, r2, p, mm, ut + o * dim);
        }
        __syncthreads();
        for (int t = tid; t < 8 * dim; t += blockDim.x) {
            const int o = t / dim, e = t % dim;
            const int cc = ch[o];
            if (cc < 0) continue;
            int n, mm;
            split_nm(e, n, mm);
            const zd* u = ut + o * dim;
            const zd* mc = moments + (size_t)cc * dim;
            zd s = mk(0.0, 0.0);
            for (int k = 0; k <= n; ++k) {
                const int nk = n - k;
                const int lo = max(-k, mm - nk), hi = min(k, mm + nk);
                for (int l = lo; l <= hi; ++l) s = zadd(s, zmul(u[cidx(k, l)], mc[cidx(nk, mm - l)]));
            }
            st[o * dim + e] = s;
        }
        __syncthreads();
        zd* out = moments + (size_t)c * dim;
        zd* acc = ut;  // the tables are no longer needed: the sums land in slot 0
        for (int e = tid; e < dim; e += blockDim.x) {
            zd a = mk(0.0, 0.0);
            for (int o = 0; o < 8; ++o)
                if (ch[o] >= 0) a = zadd(a, st[o * dim + e]);
            out[e] = a;
            acc[e] = a;
        }
        __syncthreads();
        for (int n = tid; n <= p; n += blockDim.x) {
            double s = 0.0;
            for (int mm = -n; mm <= n; ++mm) {
                int am = mm < 0 ? -mm : mm;
                zd v = acc[cidx(n, mm)];
                double w = g_tab.fact[n - am] * g_tab.fact[n + am];
                s += w * (v.re * v.re + v.im * v.im);
            }
            pows[(size_t)c * (p + 1) + n] = sqrt(s);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ f pre-pass
// f_walk, mac.rs:99-147: monopole treecode estimate of f_b = sum m/r^2 with a
// LIFO stack (children pushed in octant order, so popped in reverse).
// In a forest the walk starts at the root of the body's own system (roots
// are level 0, in system order; slots of system s are [off[s], off[s+1])).
//
// A warp walks for 32 neighbouring bodies at once: a stack entry carries the
// lanes that still have to look at its cell, and a cell is expanded for the
// lanes that do not accept it. The cells a lane meets keep their order among
// themselves, so every body's sum is the reference's, term by term. A cell's
// record goes onto the stack with it (eight lanes read eight children at once),
// and a leaf's bodies are read side by side into shared memory: one L2 round trip
// per expansion or leaf instead of several per body and cell. Bound by the latency
// of the dependent FP64 terms, a division each, and then by those round trips
// (10^5 bodies: 15 warps per SM, issue 47 %, FP64 pipe 28 %; stalls 4.1 wait, 1.4
// long scoreboard per issue). (A thread per body with its own stack took
// 0.90 ms for 16,384 bodies and 1.58 ms for a cuspy profile of 10^5.)
#define FPRE_STACK (8 * FMMX_NLEVELS + 32)
struct FpreWarp {
    double4 geo[FPRE_STACK];  // centre, rho (sign set: leaf)
    double mass[FPRE_STACK];  // of a leaf: its first slot and count
    int cell[FPRE_STACK];
    unsigned lanes[FPRE_STACK];
    double4 body[32];
};

__global__ void __launch_bounds__(32 * FPRE_WARPS) k_fprepass(CellsView cells, const double* __restrict__ x,
                                                              const double* __restrict__ y,
                                                              const double* __restrict__ z,
                                                              const double* __restrict__ m, size_t n,
                                                              const uint64_t* __restrict__ off, int nsys,
                                                              const int32_t* __restrict__ roots,
                                                              double* __restrict__ f, int* __restrict__ err) {
    extern __shared__ __align__(32) unsigned char smem_raw[];
    FpreWarp& S = reinterpret_cast<FpreWarp*>(smem_raw)[threadIdx.x >> 5];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const size_t stride = (size_t)gridDim.x * FPRE_WARPS * 32;
    // stack entry e of cell c for the given lanes
    auto put = [&](int e, int c, unsigned lanes) {
        const double4 g = cells.geo[c];
        S.geo[e] = g;
        S.mass[e] = signbit(g.w) ? __hiloint2double((int)cells.count[c], (int)cells.first[c]) : cells.mass[c];
        S.cell[e] = c;
        S.lanes[e] = lanes;
    };
    for (size_t base = ((size_t)blockIdx.x * FPRE_WARPS + (threadIdx.x >> 5)) * 32; base < n; base += stride) {
        const size_t i = base + lane;
        const bool mine = i < n;
        const double px = mine ? x[i] : 0.0, py = mine ? y[i] : 0.0, pz = mine ? z[i] : 0.0;
        int sp = 0;
        {  // the roots of the lanes' systems
            const int root = mine ? (nsys > 1 ? roots[system_of(off, nsys, i)] : roots[0]) : -1;
            unsigned left = __ballot_sync(FULL, mine);
            while (left) {
                const int r = __shfl_sync(FULL, root, __ffs(left) - 1);
                const unsigned who = __ballot_sync(FULL, root == r);
                if (lane == 0) put(sp, r, who);
                ++sp;
                left &= ~who;
            }
        }
        double fi = 0.0;
        while (sp > 0) {
            __syncwarp();
            --sp;
            const double4 g = S.geo[sp];
            const unsigned who = S.lanes[sp];
            const bool in = (who >> lane) & 1u;
            const double mass = S.mass[sp];
            const int c = S.cell[sp];
            __syncwarp();
            if (signbit(g.w)) {
                const uint32_t fst = (uint32_t)__double2loint(mass), end = fst + (uint32_t)__double2hiint(mass);
                for (uint32_t k0 = fst; k0 < end; k0 += 32) {
                    const int nb = (int)min(32u, end - k0);
                    if (lane < nb) {
                        const uint32_t k = k0 + lane;
                        S.body[lane] = make_double4(x[k], y[k], z[k], m[k]);
                    }
                    __syncwarp();
                    if (in) {
                        for (int b = 0; b < nb; ++b) {
                            const double4 q = S.body[b];
                            const double dx = px - q.x, dy = py - q.y, dz = pz - q.z;
                            const double r2 = dx * dx + dy * dy + dz * dz;
                            if (k0 + b != i && r2 > 0.0) fi += q.w / r2;
                        }
                    }
                    __syncwarp();
                }
            } else {
                const double dx = px - g.x, dy = py - g.y, dz = pz - g.z;
                const double d2 = dx * dx + dy * dy + dz * dz;
                const bool far = d2 > g.w * g.w;
                if (in && far) fi += mass / d2;
                const unsigned open = __ballot_sync(FULL, in && !far);
                if (open) {
                    if (sp + 8 > FPRE_STACK) {  // cannot happen: at most 7 entries a level stay behind
                        if (lane == 0) atomicOr(err, 1);
                        break;
                    }
                    const int ch = lane < 8 ? cells.child[8 * (size_t)c + lane] : -1;
                    const unsigned have = __ballot_sync(FULL, ch >= 0);
                    if (ch >= 0) put(sp + __popc(have & ((1u << lane) - 1u)), ch, open);
                    sp += __popc(have);
                }
            }
        }
        if (mine) f[i] = fi;
        __syncwarp();
    }
}

void launch_fprepass(cudaStream_t s, CellsView cells, const double* x, const double* y, const double* z,
                     const double* m, size_t n, const uint64_t* off, int nsys, const int32_t* roots, double* f,
                     int* err) {
    const size_t smem = FPRE_WARPS * sizeof(FpreWarp);
    cudaFuncSetAttribute(k_fprepass, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_fprepass<<<grid_for((n + 31) / 32, FPRE_WARPS), 32 * FPRE_WARPS, smem, s>>>(cells, x, y, z, m, n, off, nsys,
                                                                                 roots, f, err);
}

// fmin of every cell (mac.rs:151-173), the smallest f of its bodies: a warp per
// leaf, then up the tree as in k_geometry_com. arrive: one zero per cell.
__global__ void __launch_bounds__(128) k_fmin(int nc, CellsView cv, const int32_t* __restrict__ parent,
                                              const double* __restrict__ f, double* __restrict__ fmin_out,
                                              unsigned* __restrict__ arrive) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * 4;
    for (int c0 = blockIdx.x * 4 + (threadIdx.x >> 5); c0 < nc; c0 += warps) {
        if (!cv.leaf[c0]) continue;
        int c = c0;
        const uint32_t fst = cv.first[c], cnt = cv.count[c];
        double mn = INFINITY;
        for (uint32_t i = lane; i < cnt; i += 32) mn = fmin(mn, f[fst + i]);
        for (;;) {
            for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_xor_sync(FULL, mn, o));
            if (lane == 0) fmin_out[c] = mn;
            const int par = parent[c];
            if (par < 0) break;
            const int ch = lane < 8 ? cv.child[8 * (size_t)par + lane] : -1;
            const unsigned have = __ballot_sync(FULL, ch >= 0);
            unsigned prev = 0;
            if (lane == 0) {
                __threadfence();
                prev = atomicAdd(&arrive[par], 1u);
            }
            prev = __shfl_sync(FULL, prev, 0);
            if (prev + 1 != (unsigned)__popc(have)) break;  // a sibling's warp goes on
            __threadfence();
            mn = ch >= 0 ? __ldcg(fmin_out + ch) : INFINITY;
            c = par;
        }
    }
}

// (centre, rho) of every cell in one 32-byte record for the walk and the near
// field, the sign of rho set for a leaf
__global__ void k_pack_geo(int nc, CellsMut cells, double4* __restrict__ geo) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x)
        geo[c] = make_double4(cells.cx[c], cells.cy[c], cells.cz[c], cells.leaf[c] ? -cells.rho[c] : cells.rho[c]);
}

}  // namespace fmmx
