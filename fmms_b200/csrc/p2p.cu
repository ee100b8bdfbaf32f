// Near field: the work units of both forms, and the plain (FP64) P2P over the
// directed leaf list.
//
// Interaction (p2p.rs:24-39, with optional Plummer softening s^2):
//   d = x_j - x_i, r2 = |d|^2 + s^2, inv = 1/sqrt(r2),
//   a_i += m_j inv^3 d, pot_i += m_j inv,
// a target skipping its own body (the i != j of the reference's self kernel,
// p2p.rs:13-46).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace fmmx {

// The bodies of the leaves with several shares: the shares' partial sums, in
// share order (one warp per leaf).
__global__ void k_p2p_combine(int ncells, DirList L, CellsView cv, P2pUnits U, double* __restrict__ ax,
                              double* __restrict__ ay, double* __restrict__ az, double* __restrict__ pot) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
        if (U.soff[c + 1] == U.soff[c]) continue;
        const uint32_t tn = cv.count[c], tf = cv.first[c];
        const uint32_t nu = p2p_shares_of(U, c, tn);
        const double4* pp = U.part + U.soff[c];
        for (uint32_t i = lane; i < tn; i += 32) {
            double4 s = pp[i];
            for (uint32_t k = 1; k < nu; ++k) {
                const double4 v = pp[(size_t)k * tn + i];
                s.x += v.x;
                s.y += v.y;
                s.z += v.z;
                s.w += v.w;
            }
            ax[tf + i] = s.x;
            ay[tf + i] = s.y;
            az[tf + i] = s.z;
            pot[tf + i] = s.w;
        }
    }
}

__global__ void k_near_sizes(int ncells, const uint32_t* __restrict__ count, uint32_t grain, WalkLists Ls) {
    unsigned long long units = 0, parts = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += gridDim.x * blockDim.x) {
        const uint4 o = Ls.sizes[c];
        const uint4 v = near_sizes(o.x, o.y, count[c], grain);
        Ls.sizes[c] = v;
        units += v.z;
        parts += v.w;
    }
    for (int o = 16; o > 0; o >>= 1) {
        units += __shfl_xor_sync(0xffffffffu, units, o);
        parts += __shfl_xor_sync(0xffffffffu, parts, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (units) atomicAdd(Ls.totals + 4, units);
        if (parts) atomicAdd(Ls.totals + 5, parts);
    }
}

void launch_near_sizes(cudaStream_t s, int ncells, const uint32_t* count, uint32_t grain, WalkLists Ls) {
    k_near_sizes<<<grid_for(ncells, 256), 256, 0, s>>>(ncells, count, grain, Ls);
}

void launch_p2p_combine(cudaStream_t s, int ncells, DirList L, CellsView cv, P2pUnits U, double* ax, double* ay,
                        double* az, double* pot) {
    k_p2p_combine<<<grid_for((size_t)ncells * 32, 256), 256, 0, s>>>(ncells, L, cv, U, ax, ay, az, pot);
}

// ------------------------------------------------------------- plain form
// A warp per work unit, persistent, no block barriers: two targets per lane,
// groups of G = ceil(nt / 2) lanes over the targets, R = 32 / G groups over the
// source bodies of each tile, reduced in group order at the end. A table gives
// each source body's leaf, and the next tile's loads are in flight while a tile
// is computed. Bound by the FP64 pipe, 66 % busy at 15 bodies per leaf (about 20
// FP64 instructions per interaction, the reciprocal square root half of them), and
// the latency of its chains (N = 2^18: 1.37 ms; a block per leaf took 2.20).
#define P2PD_CHUNK 128
#define P2PD_MAP 2048
#define P2PD_TILE 64
#define P2PD_WARPS 4

struct P2pF64Smem {
    union {
        double4 t[P2PD_TILE];
        double red[8][32];
    };
    uint32_t shift[P2PD_CHUNK];  // first slot of the leaf - its first position in the chunk
    uint8_t own[P2PD_MAP];
};

template <bool SELF>
__device__ __forceinline__ void p2p_f64_term(double x, double y, double z, double m, bool self, double xi, double yi,
                                             double zi, double soft2, double& ax, double& ay, double& az, double& pt) {
    const double dx = x - xi, dy = y - yi, dz = z - zi;
    double r2 = dx * dx + dy * dy + dz * dz + soft2;
    double mj = m;
    if (SELF && self) {
        r2 = 1.0;
        mj = 0.0;
    }
    const double inv = rsqrt(r2);
    const double mi = mj * inv;
    const double f = mi * (inv * inv);
    ax += f * dx;
    ay += f * dy;
    az += f * dz;
    pt += mi;
}

__global__ void __launch_bounds__(32 * P2PD_WARPS, 5) k_p2p_f64(DirList L, CellsView cv, P2pUnits U,
                                                              const double* __restrict__ x,
                                                              const double* __restrict__ y,
                                                              const double* __restrict__ z,
                                                              const double* __restrict__ m, double soft2,
                                                              double* __restrict__ ax, double* __restrict__ ay,
                                                              double* __restrict__ az, double* __restrict__ pot) {
    constexpr int BPT = P2PD_TILE / 32;  // bodies staged per lane
    constexpr int H = P2PD_CHUNK / 32;
    __shared__ P2pF64Smem smem_w[P2PD_WARPS];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    P2pF64Smem& S = smem_w[threadIdx.x >> 5];
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(U.next, 1u);
        u = __shfl_sync(FULL, u, 0);
        if (u >= U.nunits) break;
        const int c = U.ucell[u];
        const uint32_t lb = L.seg_begin[c], len = L.seg_end[c] - lb;
        const uint32_t tf = cv.first[c], tn = cv.count[c];
        const uint32_t ns_all = p2p_shares_of(U, c, tn);
        const uint32_t k = u - U.uoff[c], share = k % ns_all, t0 = (k / ns_all) * P2P_NT;
        const uint32_t beg = lb + (uint32_t)((uint64_t)len * share / ns_all);
        const uint32_t end = lb + (uint32_t)((uint64_t)len * (share + 1) / ns_all);
        const int nt = (int)min((uint32_t)P2P_NT, tn - t0);
        const int G = (nt + 1) >> 1;
        const int R = 32 / G;
        const int g = lane % G, rep = lane / G;
        const bool active = rep < R;
        const int i0 = g, i1 = min(g + G, nt - 1);  // (an odd last target is computed twice, written once)
        const uint32_t s0 = tf + t0 + i0, s1 = tf + t0 + i1;
        const double x0 = x[s0], y0 = y[s0], z0 = z[s0], x1 = x[s1], y1 = y[s1], z1 = z[s1];
        double a0x = 0, a0y = 0, a0z = 0, p0 = 0, a1x = 0, a1y = 0, a1z = 0, p1 = 0;
        for (uint32_t sc = beg; sc < end;) {
            const int ns = (int)min((uint32_t)P2PD_CHUNK, end - sc);
            __syncwarp();
            int src[H];
            uint32_t nb[H], fs[H];
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const int q = lane + 32 * h;
                src[h] = q < ns ? (int)L.src[sc + q] : -1;
            }
#pragma unroll
            for (int h = 0; h < H; ++h) {
                nb[h] = src[h] >= 0 ? cv.count[src[h]] : 0;
                fs[h] = src[h] >= 0 ? cv.first[src[h]] : 0;
            }
            uint32_t base = 0;
            int nl = 0, self_at = -1;  // leaves whose bodies fit in the table; the target leaf's first position
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const int q = lane + 32 * h;
                uint32_t incl = nb[h];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                incl += base;
                const uint32_t excl = incl - nb[h];
                const bool fits = src[h] >= 0 && (incl <= P2PD_MAP || q == 0);
                nl += __popc(__ballot_sync(FULL, fits));
                if (fits) {
                    S.shift[q] = fs[h] - excl;
                    if (src[h] == c) self_at = (int)excl;
                    if (incl <= P2PD_MAP)
                        for (uint32_t e = excl; e < incl; ++e) S.own[e] = (uint8_t)q;
                    nb[h] = incl;  // keeps the last leaf's end
                }
                base = __shfl_sync(FULL, incl, 31);
            }
            uint32_t total = 0;
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const uint32_t v = __shfl_sync(FULL, nb[h], (nl - 1) & 31);
                if ((nl - 1) >> 5 == h) total = v;
            }
            const bool mapped = total <= P2PD_MAP;
            const int sp = __reduce_max_sync(FULL, self_at);
            __syncwarp();
            sc += nl;
            double4 v[BPT];
            auto issue = [&](uint32_t b0) {  // load the bodies of the tile at b0
#pragma unroll
                for (int e = 0; e < BPT; ++e) {
                    const uint32_t p = b0 + lane + 32 * e;
                    if (p < total) {
                        const uint32_t slot = p + S.shift[mapped ? S.own[p] : 0];
                        v[e] = make_double4(x[slot], y[slot], z[slot], m[slot]);
                    }
                }
            };
            issue(0);
            for (uint32_t b0 = 0; b0 < total; b0 += P2PD_TILE) {
                const int nbt = (int)min((uint32_t)P2PD_TILE, total - b0);
                __syncwarp();
#pragma unroll
                for (int e = 0; e < BPT; ++e)
                    if (lane + 32 * e < nbt) S.t[lane + 32 * e] = v[e];
                __syncwarp();
                issue(b0 + P2PD_TILE);
                if (active) {
                    if (sp < 0 || sp >= (int)b0 + nbt || sp + (int)tn <= (int)b0) {
                        for (int j = rep; j < nbt; j += R) {
                            const double4 q = S.t[j];
                            p2p_f64_term<false>(q.x, q.y, q.z, q.w, false, x0, y0, z0, soft2, a0x, a0y, a0z, p0);
                            p2p_f64_term<false>(q.x, q.y, q.z, q.w, false, x1, y1, z1, soft2, a1x, a1y, a1z, p1);
                        }
                    } else {
                        const int o0 = sp - (int)b0 + (int)t0 + i0, o1 = sp - (int)b0 + (int)t0 + i1;
                        for (int j = rep; j < nbt; j += R) {
                            const double4 q = S.t[j];
                            p2p_f64_term<true>(q.x, q.y, q.z, q.w, j == o0, x0, y0, z0, soft2, a0x, a0y, a0z, p0);
                            p2p_f64_term<true>(q.x, q.y, q.z, q.w, j == o1, x1, y1, z1, soft2, a1x, a1y, a1z, p1);
                        }
                    }
                }
            }
        }
        __syncwarp();
        S.red[0][lane] = a0x; S.red[1][lane] = a0y; S.red[2][lane] = a0z; S.red[3][lane] = p0;
        S.red[4][lane] = a1x; S.red[5][lane] = a1y; S.red[6][lane] = a1z; S.red[7][lane] = p1;
        __syncwarp();
        for (int o = lane; o < 4 * nt; o += 32) {
            const int t = o >> 2, comp = o & 3;
            const int gi = t < G ? t : t - G;  // target t = gi + half * G
            const int row = (t < G ? 0 : 4) + comp;
            double s = 0.0;
            for (int r = 0; r < R; ++r) s += S.red[row][r * G + gi];
            if (ns_all == 1) {
                double* out = comp == 0 ? ax : comp == 1 ? ay : comp == 2 ? az : pot;
                out[tf + t0 + t] = s;
            } else {
                reinterpret_cast<double*>(U.part + U.soff[c] + (size_t)share * tn + t0 + t)[comp] = s;
            }
        }
        __syncwarp();
    }
}

void launch_p2p_f64(int nsm, cudaStream_t s, DirList L, int ncells, CellsView cv, P2pUnits U, const double* x,
                    const double* y, const double* z, const double* m, double soft2, double* ax, double* ay,
                    double* az, double* pot) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_p2p_f64, 32 * P2PD_WARPS, 0) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const unsigned need = (unsigned)(((uint64_t)U.nunits + P2PD_WARPS - 1) / P2PD_WARPS);
    k_p2p_f64<<<std::max(1u, std::min(need, (unsigned)(nsm * per_sm))), 32 * P2PD_WARPS, 0, s>>>(
        L, cv, U, x, y, z, m, soft2, ax, ay, az, pot);
    launch_p2p_combine(s, ncells, L, cv, U, ax, ay, az, pot);
}

}  // namespace fmmx
