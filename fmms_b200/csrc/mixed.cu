// Mixed-precision form: FP32 expansions and P2P, FP64 only where the reference
// needs it (centre-relative coordinates, the MAC, M2M/L2L on the top three
// tree levels).
//
// Expansions are stored for m >= 0 only (a real field has
// v_{-m} = (-1)^m conj(v_m)) and normalised by a per-cell length l (the cell's
// radius rho, or a small fraction of its box size when rho = 0):
//     M^_n^m = M_n^m / l^n,      F^_n^m = F_n^m l^{n+1}.
// Every translation then works on O(1) quantities, so FP32 neither overflows
// nor underflows at p = 12 for cells down to the level-21 cut:
//   P2M: M^_n^m  = sum_b m_b Υ_n^m((x_b - s)/l)
//   M2M: M^_p[n][m] = sum_k sum_l Υ_k^l((s_c - s_p)/l_p) M^_c[n-k][m-l] (l_c/l_p)^{n-k}
//   L2L: F^_c[n][m] = (l_c/l_p)^{n+1} sum_{k,l} conj(Υ_k^l((s_p - s_c)/l_p)) F^_p[n+k][m+l]
//   L2P: Ψ_0^0 = (1/l) sum conj(Υ_k^l(r^)) F^_k^l,  Ψ_1^m = (1/l^2) sum conj(Υ_k^l(r^)) F^_{k+1}^{m+l}
// (the unnormalised forms are moments.rs:30-90 and translate.rs:175-309).
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace fmmx {

// The order tables in global memory: the kernels read them with lane-
// dependent indices (a lane per order m or per degree), which the constant
// cache would serialise over the distinct addresses; global loads are served
// from L1 in parallel.
static __device__ OrderTables g_tab;

// FP32 copies of the recursion's constants (a double read would need a
// conversion per use).
struct FloatTables {
    float inv2m[FMMX_MAXP + 1];
    float invc[FMMX_MAXP + 1][FMMX_MAXP + 1];
};
static __device__ FloatTables g_tabf;
template <typename A>
__device__ __forceinline__ A tab_inv2m(int m) {
    if constexpr (sizeof(A) == 4) return g_tabf.inv2m[m];
    else return g_tab.inv2m[m];
}
template <typename A>
__device__ __forceinline__ A tab_invc(int n, int m) {
    if constexpr (sizeof(A) == 4) return g_tabf.invc[n][m];
    else return g_tab.invc[n][m];
}

void upload_tables_mixed(const OrderTables& t, cudaStream_t s) {
    cudaMemcpyToSymbolAsync(g_tab, &t, sizeof(t), 0, cudaMemcpyHostToDevice, s);
    FloatTables f;
    for (int m = 0; m <= FMMX_MAXP; ++m) f.inv2m[m] = (float)t.inv2m[m];
    for (int n = 0; n <= FMMX_MAXP; ++n)
        for (int m = 0; m <= FMMX_MAXP; ++m) f.invc[n][m] = (float)t.invc[n][m];
    cudaMemcpyToSymbolAsync(g_tabf, &f, sizeof(f), 0, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);  // the staging copy dies here
}

// Touches the tables' lines at once. The recursions read a table row per step;
// cold, each would wait for the L2 in turn (3 us of a kernel on a small tree).
template <typename A>
__device__ __forceinline__ void warm_tables(int p) {
    for (int i = threadIdx.x; i < 3 * (p + 1); i += blockDim.x) {
        const int n = i / 3, m = min(8 * (i % 3), FMMX_MAXP);
        if constexpr (sizeof(A) == 4) asm volatile("" ::"f"(g_tabf.invc[n][m]), "f"(g_tabf.inv2m[m]));
        else asm volatile("" ::"d"(g_tab.invc[n][m]), "d"(g_tab.inv2m[m]));
    }
}

__host__ __device__ constexpr int hx(int n, int m) { return n * (n + 1) / 2 + m; }

__device__ __forceinline__ void split_h(int e, int& n, int& m) {
    int q = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
    while (q * (q + 1) / 2 > e) --q;
    while ((q + 1) * (q + 2) / 2 <= e) ++q;
    n = q;
    m = e - q * (q + 1) / 2;
}

// Normalising length of every cell: rho, or the cell's box size h when rho = 0
// (a single body, or coincident bodies: then every moment above the monopole
// is exactly zero and any positive length works), kept >= 1e-30 so that it is
// a normal FP32 number (a system of coincident bodies has box size DBL_MIN).
__global__ void k_cell_scale(int nc, const double* __restrict__ rho, const double* __restrict__ h,
                             double* __restrict__ ell, float* __restrict__ ellf) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        double l = rho[c];
        if (!(l > 0.0)) l = h[c];
        l = fmax(l, 1e-30);
        ell[c] = l;
        ellf[c] = (float)l;
    }
}

// Cell radii about the build's centres for the current positions, on a
// reused tree: the bodies have drifted since the build, and a cell whose built
// radius is tiny (a tight pair) would otherwise normalise its moments by a
// length far below the bodies' distances from its centre, overflowing FP32
// (M_n / l^n). Never below the built radius. A warp per leaf over its bodies, then
// up the tree: the warp that finishes a cell's last child goes on with the cell
// (the construction of tree.rs:152-227 with the centres held fixed). arrive: one
// zero per cell.
__global__ void __launch_bounds__(128) k_rho_now(int nc, CellsView cv, const int32_t* __restrict__ parent,
                                                 const double* __restrict__ x, const double* __restrict__ y,
                                                 const double* __restrict__ z, double* __restrict__ rho,
                                                 unsigned* __restrict__ arrive) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * 4;
    for (int c0 = blockIdx.x * 4 + (threadIdx.x >> 5); c0 < nc; c0 += warps) {
        if (!cv.leaf[c0]) continue;
        int c = c0;
        double r = 0.0;
        {
            const double cx = cv.cx[c], cy = cv.cy[c], cz = cv.cz[c];
            const uint32_t f = cv.first[c], cnt = cv.count[c];
            for (uint32_t i = lane; i < cnt; i += 32) {
                const double dx = x[f + i] - cx, dy = y[f + i] - cy, dz = z[f + i] - cz;
                r = fmax(r, sqrt(dx * dx + dy * dy + dz * dz));
            }
        }
        for (;;) {
            for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(FULL, r, o));
            r = fmax(cv.rho[c], r);
            if (lane == 0) rho[c] = r;
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
            r = 0.0;
            if (ch >= 0) {
                const double dx = cv.cx[ch] - cv.cx[par], dy = cv.cy[ch] - cv.cy[par], dz = cv.cz[ch] - cv.cz[par];
                r = __ldcg(rho + ch) + sqrt(dx * dx + dy * dy + dz * dz);
            }
            c = par;
        }
    }
}

// FP64 full-layout moments (the exact upward pass) -> normalised FP32 half layout.
__global__ void k_moments_to_mixed(int nc, int p, const zd* __restrict__ full, const double* __restrict__ ell,
                                   zf* __restrict__ half) {
    const int H = (p + 1) * (p + 2) / 2, D = (p + 1) * (p + 1), HS = half_stride(p);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)nc * H;
         i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i / H), e = (int)(i % H);
        int n, m;
        split_h(e, n, m);
        const double s = pow(ell[c], -n);
        const zd v = full[(size_t)c * D + n * (n + 1) + m];
        half[(size_t)c * HS + e] = mk<float>((float)(v.re * s), (float)(v.im * s));
    }
}

// P2M of the leaves among cells [0, nc) (list == nullptr) or list[0 .. nc), a
// warp per leaf and a lane per body: the lane runs through its body's Υ and
// adds m Υ into its own column of shared memory; the columns are summed at the
// end, lane e taking entry e from its own column on (distinct banks). A =
// double for the leaves of the top three levels (`top`), float below. Bound by
// latency at the 9 warps per SM that the columns leave room for (p = 10: issue
// 39 %, shared-memory pipe 15 %). (A 128-thread block per leaf, a thread per column
// and body group, took 0.31 ms for 32,768 leaves of 32 bodies at p = 10.)
template <typename A>
__global__ void __launch_bounds__(128) k_p2m_mixed(const int32_t* __restrict__ list, int nc, bool top,
                                                              CellsView cv, const double* __restrict__ ell,
                                                              const double* __restrict__ x,
                                                              const double* __restrict__ y,
                                                              const double* __restrict__ z,
                                                              const double* __restrict__ m, int p,
                                                              zf* __restrict__ mom) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int H = (p + 1) * (p + 2) / 2;
    const int lane = threadIdx.x & 31;
    cplx<A>* sbuf = reinterpret_cast<cplx<A>*>(smem_raw) + (size_t)(threadIdx.x >> 5) * 32 * H;
    cplx<A>* col = sbuf + lane;
    const int wpb = blockDim.x >> 5, warps = gridDim.x * wpb;
    warm_tables<A>(p);
    for (int j = blockIdx.x * wpb + (threadIdx.x >> 5); j < nc; j += warps) {
        const int c = list ? list[j] : j;
        if (!cv.leaf[c] || (cv.level[c] <= 2) != top) continue;
        const double sx = cv.cx[c], sy = cv.cy[c], sz = cv.cz[c];
        const double il = 1.0 / ell[c];
        const uint32_t f = cv.first[c], cnt = cv.count[c];
        for (uint32_t b0 = 0; b0 < cnt; b0 += 32) {
            const bool mine = b0 + lane < cnt;
            const uint32_t q = f + b0 + (mine ? lane : 0);
            const A rx = (A)((x[q] - sx) * il), ry = (A)((y[q] - sy) * il), rz = (A)((z[q] - sz) * il);
            const A mb = mine ? (A)m[q] : A(0);
            const A r2 = rx * rx + ry * ry + rz * rz;
            cplx<A> d = mk<A>(mb, A(0));  // (the mass rides along: the recursions are linear)
            auto add = [&](int e, cplx<A> v) {
                if (b0 == 0) {
                    col[32 * e] = v;
                } else {
                    const cplx<A> o = col[32 * e];
                    col[32 * e] = mk<A>(o.re + v.re, o.im + v.im);
                }
            };
            for (int mm = 0; mm <= p; ++mm) {
                if (mm > 0) d = zmul(zscale(mk<A>(rx, ry), tab_inv2m<A>(mm)), d);
                int e = hx(mm, mm);
                add(e, d);
                cplx<A> u1 = d, u2 = mk<A>(A(0), A(0));
                for (int n = mm + 1; n <= p; ++n) {
                    const A a = (A)(2 * n - 1) * rz;
                    const cplx<A> un = zscale(zsub(zscale(u1, a), zscale(u2, r2)), tab_invc<A>(n, mm));
                    u2 = u1;
                    u1 = un;
                    e += n;  // (n, mm)
                    add(e, un);
                }
            }
        }
        __syncwarp();
        zf* out = mom + (size_t)c * half_stride(p);
        const int nl = (int)min(cnt, 32u);
        for (int e = lane; e < H; e += 32) {
            A sr = 0, si = 0;
            const cplx<A>* row = sbuf + 32 * e;
            if (nl == 32) {
#pragma unroll 8
                for (int l = 0; l < 32; ++l) {
                    const cplx<A> v = row[(l + lane) & 31];
                    sr += v.re;
                    si += v.im;
                }
            } else {  // the first nl columns, from lane mod nl on
                int l = lane % nl;
                for (int k = 0; k < nl; ++k) {
                    const cplx<A> v = row[l];
                    sr += v.re;
                    si += v.im;
                    if (++l == nl) l = 0;
                }
            }
            out[e] = mk<float>((float)sr, (float)si);
        }
        __syncwarp();
    }
}

// Υ column m (harmonic.rs:141-173) of r in precision A, stored in the full layout
// (entry (n, m) at n(n+1) + m for |m| <= n), with v_{n,-m} = (-1)^m conj(v_{n,m}).
template <typename A>
__device__ __forceinline__ void ups_column_full(A x, A y, A z, A r2, int p, int m, cplx<A>* u) {
    auto put = [&](int n, cplx<A> v) {
        u[n * (n + 1) + m] = v;
        if (m) u[n * (n + 1) - m] = (m & 1) ? mk<A>(-v.re, v.im) : mk<A>(v.re, -v.im);
    };
    cplx<A> d = mk<A>(A(1), A(0));
    for (int j = 1; j <= m; ++j) d = zmul(zscale(mk<A>(x, y), tab_inv2m<A>(j)), d);
    put(m, d);
    cplx<A> u1 = d, u2 = mk<A>(A(0), A(0));
    for (int n = m + 1; n <= p; ++n) {
        const A a = (A)(2 * n - 1) * z;
        const cplx<A> un = zscale(zsub(zscale(u1, a), zscale(u2, r2)), tab_invc<A>(n, m));
        put(n, un);
        u2 = u1;
        u1 = un;
    }
}

// M2M of every internal cell in one launch: a block per cell, up the tree from
// the cells without internal children (the leaves' moments are there); the block
// that finishes a cell's last internal child goes on with the cell, so no block
// waits. First the Υ of the eight child offsets (a thread per child and column)
// and the children's moments, both in the full layout (both signs of m), so that
// a product is two loads and four FMAs; then a thread per (child, entry) sums that
// child's contribution and the children are added in octant order. A = double on
// the top three levels, float below. Bound by latency: the products of a cell
// (13,700 at p = 10) take a few hundred instructions a thread between barriers
// (issue 44 %, 8.4 barrier stalls per issue). arrive: one zero per cell. (With P2M in the same kernel and a launch per level: N = 1e3, 7
// levels, 0.15 ms; N = 2^20 uniform 0.70 ms.)
#define M2M_BLOCK 512
#define M2M_SCAN 32  // cells a block looks over at a time for its starting points
template <typename A>
__device__ __forceinline__ void m2m_cell(int c, const int* __restrict__ ch, CellsView cv,
                                         const double* __restrict__ ell, int p, zf* __restrict__ mom,
                                         unsigned char* smem_raw) {
    const int P1 = p + 1, H = P1 * (P1 + 1) / 2, F2 = P1 * P1;
    cplx<A>* u = reinterpret_cast<cplx<A>*>(smem_raw);  // 8 x F2: Υ of the child offsets
    cplx<A>* part = u + 8 * F2;                         // 8 x H: the children's contributions
    zf* cm = reinterpret_cast<zf*>(part + 8 * H);       // 8 x F2: the children's moments
    const int tid = threadIdx.x;
    const double sx = cv.cx[c], sy = cv.cy[c], sz = cv.cz[c];
    const double il = 1.0 / ell[c];
    for (int w = tid; w < 8 * P1; w += M2M_BLOCK) {
        const int o = w / P1, mc = w % P1;
        if (ch[o] < 0) continue;
        const A dx = (A)((cv.cx[ch[o]] - sx) * il), dy = (A)((cv.cy[ch[o]] - sy) * il),
                dz = (A)((cv.cz[ch[o]] - sz) * il);
        ups_column_full<A>(dx, dy, dz, dx * dx + dy * dy + dz * dz, p, mc, u + o * F2);
    }
    for (int w = tid; w < 8 * H; w += M2M_BLOCK) {  // (written by other SMs in this launch: read past the L1)
        const int o = w / H, e = w % H;
        if (ch[o] < 0) continue;
        const float2 v = __ldcg(reinterpret_cast<const float2*>(mom + (size_t)ch[o] * half_stride(p)) + e);
        int n, mm;
        split_h(e, n, mm);
        zf* t = cm + o * F2 + n * (n + 1);
        t[mm] = mk<float>(v.x, v.y);
        if (mm) t[-mm] = (mm & 1) ? mk<float>(-v.x, v.y) : mk<float>(v.x, -v.y);
    }
    __syncthreads();
    for (int w = tid; w < 8 * H; w += M2M_BLOCK) {  // the entries of most products first
        const int o = w & 7, e = H - 1 - (w >> 3);
        A sr = 0, si = 0;
        if (ch[o] >= 0) {
            int n, mm;
            split_h(e, n, mm);
            const A ratio = (A)(ell[ch[o]] * il);
            A rpow = 1;  // ratio^{n-k}, built from k = n down
            for (int k = n; k >= 0; --k) {
                const int nk = n - k;
                const int lo = max(-k, mm - nk), hi = min(k, mm + nk);
                const cplx<A>* uk = u + o * F2 + k * (k + 1);
                const zf* mk_ = cm + o * F2 + nk * (nk + 1) + mm;
                A tr = 0, ti = 0;
                for (int l = lo; l <= hi; ++l) {
                    const cplx<A> uu = uk[l];
                    const zf mv = mk_[-l];
                    tr += uu.re * (A)mv.re - uu.im * (A)mv.im;
                    ti += uu.re * (A)mv.im + uu.im * (A)mv.re;
                }
                sr += tr * rpow;
                si += ti * rpow;
                rpow *= ratio;
            }
        }
        part[o * H + e] = mk<A>(sr, si);
    }
    __syncthreads();
    zf* out = mom + (size_t)c * half_stride(p);
    for (int e = tid; e < H; e += M2M_BLOCK) {
        A sr = 0, si = 0;
        for (int o = 0; o < 8; ++o) {
            sr += part[o * H + e].re;
            si += part[o * H + e].im;
        }
        out[e] = mk<float>((float)sr, (float)si);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(M2M_BLOCK) k_m2m_mixed(int nc, CellsView cv, const int32_t* __restrict__ parent,
                                                        const double* __restrict__ ell, int p, zf* __restrict__ mom,
                                                        unsigned* __restrict__ arrive) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int ch[8], start[M2M_SCAN], nstart, next;
    const int tid = threadIdx.x;
    warm_tables<float>(p);
    warm_tables<double>(p);
    for (int b = blockIdx.x * M2M_SCAN; b < nc; b += gridDim.x * M2M_SCAN) {
        if (tid < M2M_SCAN) {  // internal cells without internal children, in order
            const int c = b + tid;
            bool first = c < nc && !cv.leaf[c];
            if (first)
                for (int o = 0; o < 8; ++o) {
                    const int q = cv.child[8 * (size_t)c + o];
                    if (q >= 0 && !cv.leaf[q]) first = false;
                }
            const unsigned mask = __ballot_sync(0xffffffffu, first);
            if (first) start[__popc(mask & ((1u << tid) - 1u))] = c;
            if (tid == 0) nstart = __popc(mask);
        }
        __syncthreads();
        const int ns = nstart;
        for (int k = 0; k < ns; ++k) {
            for (int c = start[k]; c >= 0;) {
                if (tid < 8) ch[tid] = cv.child[8 * (size_t)c + tid];
                __syncthreads();
                if (cv.level[c] <= 2) m2m_cell<double>(c, ch, cv, ell, p, mom, smem_raw);
                else m2m_cell<float>(c, ch, cv, ell, p, mom, smem_raw);
                // the parent, if this was its last internal child
                if (tid < 32) {
                    const int par = parent[c];
                    int go = -1;
                    if (par >= 0) {
                        const int q = tid < 8 ? cv.child[8 * (size_t)par + tid] : -1;
                        const unsigned inner = __ballot_sync(0xffffffffu, q >= 0 && !cv.leaf[q]);
                        if (tid == 0) {
                            __threadfence();  // the block's moments (ordered before by the barrier) before the arrival
                            if (atomicAdd(&arrive[par], 1u) + 1 == (unsigned)__popc(inner)) {
                                __threadfence();
                                go = par;
                            }
                        }
                    }
                    if (tid == 0) next = go;
                }
                __syncthreads();
                c = next;
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

// top: cells of the top three levels, ntop of them; nc cells in all
void launch_upward_mixed(cudaStream_t s, const int32_t* top, int ntop, int nc, CellsView cv, const int32_t* parent,
                         const double* ell, const double* x, const double* y, const double* z, const double* m, int p,
                         zf* mom, unsigned* arrive) {
    const int H = (p + 1) * (p + 2) / 2, F2 = (p + 1) * (p + 1);
    auto warps = [&](size_t col) {  // per block: as many as its columns leave room for, 1 .. 4
        int w = 4;
        while (w > 1 && w * col > FMMX_SMEM_MOST) w >>= 1;
        return w;
    };
    const size_t cf = (size_t)32 * H * sizeof(zf), cd = (size_t)32 * H * sizeof(zd);
    const int wf = warps(cf), wd = warps(cd);
    allow_smem(k_p2m_mixed<float>, wf * cf);
    allow_smem(k_p2m_mixed<double>, wd * cd);
    k_p2m_mixed<double><<<grid_for(ntop, wd), 32 * wd, wd * cd, s>>>(top, ntop, true, cv, ell, x, y, z, m, p, mom);
    if (nc > ntop)
        k_p2m_mixed<float><<<grid_for(nc, wf), 32 * wf, wf * cf, s>>>(nullptr, nc, false, cv, ell, x, y, z, m, p, mom);
    const size_t sm = 8 * (size_t)(F2 + H) * sizeof(zd) + 8 * (size_t)F2 * sizeof(zf);
    allow_smem(k_m2m_mixed, sm);
    if (nc > 1)
        k_m2m_mixed<<<grid_for(nc, M2M_SCAN), M2M_BLOCK, sm, s>>>(nc, cv, parent, ell, p, mom, arrive);
}

// L2L for the cells of one level (L >= 1), one warp per cell; A as above.
//
// Output (n, m) of the child's locals is ratio^{n+1} sum_{k <= p-n, |l| <= k}
// conj(Υ_{k,l}(r)) L_{n+k, m+l} of the parent: (p-n+1)^2 products, 121 for
// the monopole and 1 for degree p at p = 10. A thread per output leaves most
// lanes idle behind the low degrees, so the products of all outputs are laid
// out as one list ("items": output by output, k then l) of
// T = q (q+1)^2 (q+2) / 12 entries (q = p + 1; 1,716 at p = 10) and every lane
// takes an equal contiguous run of it. An output that lies inside one lane's
// run is finished there; one that crosses runs leaves a partial sum in each
// (slot 0: the output the run starts in, slot 1: the one it ends in), added
// afterwards, in lane order, by the lane holding its first product -- a fixed
// order, so the result bits do not depend on scheduling. The list (item: Υ
// index, parent index, output, and a last-product flag) is made once per
// context, l2l_schedule; every block copies it (building it in the kernel took
// most of the 14 us of a launch over a few cells). Υ and the parent's locals sit
// in shared memory in the full layout (both signs of m), so a product is two
// loads and four FMAs.
#define L2LB_WARPS 4

__host__ __device__ constexpr int l2l_items(int p) {
    return (p + 1) * (p + 2) * (p + 2) * (p + 3) / 12;
}

// first item | n << 16 of every output (and the item count), then the items
void l2l_schedule(int p, std::vector<uint32_t>& out) {
    const int H = (p + 1) * (p + 2) / 2, T = l2l_items(p);
    out.assign(H + 1 + T, 0);
    int s = 0;
    for (int n = 0; n <= p; ++n)
        for (int m = 0; m <= n; ++m) {
            const int e = hx(n, m);
            out[e] = (uint32_t)s | ((uint32_t)n << 16);
            for (int k = 0; k <= p - n; ++k)
                for (int l = -k; l <= k; ++l, ++s)
                    out[H + 1 + s] = (uint32_t)(k * (k + 1) + l) | ((uint32_t)((n + k) * (n + k + 1) + m + l) << 9) |
                                     ((uint32_t)e << 18) | (k == p - n && l == k ? 0x80000000u : 0u);
        }
    out[H] = (uint32_t)T;
}

template <typename A>
static size_t l2l_smem(int p) {
    const int P1 = p + 1, H = P1 * (P1 + 1) / 2, F2 = P1 * P1;
    return (size_t)L2LB_WARPS * (F2 + 64 + H) * sizeof(cplx<A>) + (size_t)L2LB_WARPS * F2 * sizeof(zf) +
           (size_t)(H + 1 + l2l_items(p)) * sizeof(uint32_t);
}

template <typename A>
__global__ void __launch_bounds__(L2LB_WARPS * 32) k_l2l_mixed(const int32_t* __restrict__ level_cells, int lstart,
                                                              int lcnt, CellsView cv,
                                                              const int32_t* __restrict__ parent,
                                                              const double* __restrict__ ell, int p,
                                                              const uint32_t* __restrict__ sched,
                                                              zf* __restrict__ loc) {
    extern __shared__ __align__(16) unsigned char lsm[];
    const int P1 = p + 1, H = P1 * (P1 + 1) / 2, F2 = P1 * P1, T = l2l_items(p);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    cplx<A>* U = reinterpret_cast<cplx<A>*>(lsm) + wid * F2;                      // Υ(r), full layout
    cplx<A>* Pp = reinterpret_cast<cplx<A>*>(lsm) + L2LB_WARPS * F2 + wid * 64;  // [lane][2] partials
    cplx<A>* R = reinterpret_cast<cplx<A>*>(lsm) + L2LB_WARPS * (F2 + 64) + wid * H;  // sums per output
    zf* F = reinterpret_cast<zf*>(reinterpret_cast<cplx<A>*>(lsm) + L2LB_WARPS * (F2 + 64 + H)) + wid * F2;
    uint32_t* einfo = reinterpret_cast<uint32_t*>(reinterpret_cast<zf*>(reinterpret_cast<cplx<A>*>(lsm) +
                                                                        L2LB_WARPS * (F2 + 64 + H)) +
                                                  L2LB_WARPS * F2);  // first item | n << 16
    uint32_t* items = einfo + H + 1;

    warm_tables<A>(p);
#pragma unroll 8
    for (int e = threadIdx.x; e < H + 1 + T; e += blockDim.x) einfo[e] = sched[e];
    __syncthreads();

    const int W = ((T + 31) / 32) | 1;  // an odd stride keeps the lanes' item reads on distinct banks
    const int r0 = min(T, lane * W), r1 = min(T, r0 + W);
    for (int j = blockIdx.x * L2LB_WARPS + wid; j < lcnt; j += gridDim.x * L2LB_WARPS) {
        const int c = level_cells[lstart + j];
        const int par = parent[c];
        if (par < 0) continue;
        const double il = 1.0 / ell[par];
        const A rx = (A)((cv.cx[par] - cv.cx[c]) * il), ry = (A)((cv.cy[par] - cv.cy[c]) * il),
                rz = (A)((cv.cz[par] - cv.cz[c]) * il);
        if (lane <= p) ups_column_full<A>(rx, ry, rz, rx * rx + ry * ry + rz * rz, p, lane, U);
        const zf* lp = loc + (size_t)par * half_stride(p);
        for (int e = lane; e < H; e += 32) {
            const int n = (int)(einfo[e] >> 16), m = e - n * (n + 1) / 2;
            const zf v = lp[e];
            F[n * (n + 1) + m] = v;
            if (m) F[n * (n + 1) - m] = (m & 1) ? mk<float>(-v.re, v.im) : mk<float>(v.re, -v.im);
        }
        __syncwarp();
        A sr = 0, si = 0;
        uint32_t it = 0, ahead = r0 < r1 ? items[r0] : 0u;
#pragma unroll 4
        for (int i = r0; i < r1; ++i) {
            it = ahead;
            if (i + 1 < r1) ahead = items[i + 1];
            const cplx<A> a = U[it & 511u];
            const zf b = F[(it >> 9) & 511u];
            sr += a.re * (A)b.re + a.im * (A)b.im;  // conj(a) * b
            si += a.re * (A)b.im - a.im * (A)b.re;
            if (it & 0x80000000u) {
                const int e = (int)((it >> 18) & 255u);
                if ((int)(einfo[e] & 0xffffu) >= r0) R[e] = mk<A>(sr, si);  // the whole output is in this run
                else Pp[2 * lane] = mk<A>(sr, si);                          // it started in an earlier run
                sr = 0;
                si = 0;
            }
        }
        if (r1 > r0 && !(it & 0x80000000u)) {  // the run ends inside an output
            const int e = (int)((it >> 18) & 255u);
            Pp[2 * lane + ((int)(einfo[e] & 0xffffu) <= r0 ? 0 : 1)] = mk<A>(sr, si);
        }
        __syncwarp();
        if (r1 > r0) {
            const int e = (int)((items[r1 - 1] >> 18) & 255u);
            const int s0 = (int)(einfo[e] & 0xffffu), s1 = (int)(einfo[e + 1] & 0xffffu);
            if (s0 >= r0 && s1 > r1) {  // an output that starts in this run and crosses into the next ones
                cplx<A> acc = Pp[2 * lane + (s0 == r0 ? 0 : 1)];
                for (int q = lane + 1; q * W < s1; ++q) {
                    acc.re += Pp[2 * q].re;
                    acc.im += Pp[2 * q].im;
                }
                R[e] = acc;
            }
        }
        __syncwarp();
        const A ratio = (A)(ell[c] * il);
        zf* lc = loc + (size_t)c * half_stride(p);
        for (int e = lane; e < H; e += 32) {
            const int n = (int)(einfo[e] >> 16);
            A sc = ratio;
            for (int q = 0; q < n; ++q) sc *= ratio;
            const zf cur = lc[e];
            const cplx<A> v = R[e];
            lc[e] = mk<float>((float)((A)cur.re + v.re * sc), (float)((A)cur.im + v.im * sc));
        }
        __syncwarp();
    }
}

void launch_l2l_mixed(bool fp64, unsigned grid, cudaStream_t s, const int32_t* level_cells, int lstart, int lcnt,
                      CellsView cv, const int32_t* parent, const double* ell, int p, const uint32_t* sched,
                      zf* loc) {
    const unsigned blocks = std::max(1u, std::min(grid, (unsigned)((lcnt + L2LB_WARPS - 1) / L2LB_WARPS)));
    if (fp64) {
        const size_t sm = l2l_smem<double>(p);
        allow_smem(k_l2l_mixed<double>, sm);
        k_l2l_mixed<double><<<blocks, L2LB_WARPS * 32, sm, s>>>(level_cells, lstart, lcnt, cv, parent, ell, p, sched,
                                                               loc);
    } else {
        const size_t sm = l2l_smem<float>(p);
        allow_smem(k_l2l_mixed<float>, sm);
        k_l2l_mixed<float><<<blocks, L2LB_WARPS * 32, sm, s>>>(level_cells, lstart, lcnt, cv, parent, ell, p, sched,
                                                               loc);
    }
}

// L2P at every body plus the near field, scattered to particle-id order: a
// thread per body, Υ of its offset generated column by column (two-term
// recursion in k) and contracted on the fly. The orders +l and -l of a real field
// contribute equally to Ψ_0^0 and Ψ_1^0, and to Ψ_1^1 through L_{k+1,l+1} and
// L_{k+1,l-1}, so only l >= 0 is run through; L_{k,l} is the last step's
// L_{k+1,l}. Bound by issue, 69 % of the time, and the loads of the locals
// (N = 2^20, p = 10: 0.13 ms; 0.25 with both signs written out).
__global__ void k_l2p_mixed(size_t n, const int32_t* __restrict__ body_leaf, const uint32_t* __restrict__ order,
                            CellsView cv, const double* __restrict__ ell, int p, const zf* __restrict__ loc,
                            const double* __restrict__ x, const double* __restrict__ y,
                            const double* __restrict__ z, const double* __restrict__ nax,
                            const double* __restrict__ nay, const double* __restrict__ naz,
                            const double* __restrict__ npot, double* __restrict__ acc, double* __restrict__ pot) {
    warm_tables<float>(p);
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const int c = body_leaf[k];
        const double l = ell[c], il = 1.0 / l;
        const float rx = (float)((cv.cx[c] - x[k]) * il), ry = (float)((cv.cy[c] - y[k]) * il),
                    rz = (float)((cv.cz[c] - z[k]) * il);
        const float r2 = rx * rx + ry * ry + rz * rz;
        const zf* L = loc + (size_t)c * half_stride(p);
        float p00 = 0, p11r = 0, p11i = 0, p10 = 0;
        zf d = mk<float>(1.f, 0.f);
        for (int lm = 0; lm <= p; ++lm) {
            if (lm > 0) d = zmul(zscale(mk<float>(rx, ry), g_tabf.inv2m[lm]), d);
            zf u = d, u2 = mk<float>(0.f, 0.f);
            zf f0 = L[hx(lm, lm)];
            float s00 = 0, s10 = 0;
            for (int kk = lm; kk <= p; ++kk) {
                s00 += u.re * f0.re + u.im * f0.im;
                if (kk == p) break;
                const zf* row = L + hx(kk + 1, lm);
                const zf f10 = row[0], f11 = row[1];
                s10 += u.re * f10.re + u.im * f10.im;
                p11r += u.re * f11.re + u.im * f11.im;
                p11i += u.re * f11.im - u.im * f11.re;
                if (lm > 0) {
                    const zf h = row[-1];
                    p11r -= u.re * h.re + u.im * h.im;
                    p11i += u.re * h.im - u.im * h.re;
                }
                const float a = (float)(2 * kk + 1) * rz;
                const zf un = zscale(zsub(zscale(u, a), zscale(u2, r2)), g_tabf.invc[kk + 1][lm]);
                u2 = u;
                u = un;
                f0 = f10;
            }
            const float w = lm > 0 ? 2.f : 1.f;
            p00 += w * s00;
            p10 += w * s10;
        }
        const uint32_t id = order[k];
        acc[3 * (size_t)id + 0] = nax[k] - ((double)p11r * il) * il;
        acc[3 * (size_t)id + 1] = nay[k] - ((double)p11i * il) * il;
        acc[3 * (size_t)id + 2] = naz[k] - ((double)p10 * il) * il;
        pot[id] = npot[k] + (double)p00 * il;
    }
}

// ------------------------------------------------------------------ P2P
// FP32 near field with FP64 sums. Bodies are kept relative to their own leaf's
// centre in FP32 (the FP64 subtraction, once per evaluation); a source body is
// moved to the target leaf's frame by its leaf's offset from the target leaf's
// centre (an FP64 difference rounded once per source leaf), so d = x_j - x_i
// carries roundings of quantities no larger than the pair's leaf separation.
// A lane sums a few dozen source pairs in FP32 (two partial sums per
// component) and adds them into FP64. 1/r by the hardware rsqrt.

// The hardware reciprocal square root (about 2^-22 relative error), flushing
// subnormal inputs: r2 is a squared distance plus the squared softening, far
// above the subnormal range whenever it is positive. No Newton step: its
// error is of the order of the FP32 rounding of the partial sums, which
// dominates the near-field error. Measured at N = 2^20 (uniform cube, p = 10,
// theta 0.5, 4096 targets against the FP64 direct sum): p99 relative force
// error 1.3787e-6 with a Newton step, 1.3773e-6 without; theta 0.3, p = 12:
// 6.42e-7 and 6.49e-7.
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Source bodies in pairs, leaf by leaf (an odd leaf's last pair is padded with
// a massless body far away): pair q of leaf c at pairs[2 (pair_base(c) + q)] =
// (x, x', y, y') and the next float4 (z, z', m, m'), relative to the leaf's
// centre. The bases are disjoint without a prefix sum: the next leaf's first
// slot plus cell id exceeds this one's by at least count + 1.
__host__ __device__ __forceinline__ uint32_t pair_base(uint32_t first, uint32_t c) {
    return (uint32_t)(((uint64_t)first + c + 1) >> 1);
}
size_t p2p_pairs_floats4(size_t n, int ncells) { return 2 * ((n + (size_t)ncells + 1) / 2 + 1); }

__global__ void k_local_pairs(size_t n, const int32_t* __restrict__ body_leaf, CellsView cv,
                              const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ z, const double* __restrict__ m, float* __restrict__ pairs) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const int c = body_leaf[k];
        const uint32_t f = cv.first[c], i = (uint32_t)k - f;
        float* o = pairs + 8 * ((size_t)pair_base(f, (uint32_t)c) + (i >> 1)) + (i & 1);
        o[0] = (float)(x[k] - cv.cx[c]);
        o[2] = (float)(y[k] - cv.cy[c]);
        o[4] = (float)(z[k] - cv.cz[c]);
        o[6] = (float)m[k];
        if ((i & 1) == 0 && i + 1 == cv.count[c]) {
            o[1] = 1e18f;
            o[3] = o[5] = o[7] = 0.f;
        }
    }
}

// One pair of source bodies (j, j+1) against one target, on packed FP32x2
// arithmetic (sm_100's two-wide FP32 instructions: one issue slot for two
// lanes of work): -x is the target's coordinate negated in both halves.
// The pair's two partial sums stay apart in the two halves of each
// accumulator until the tile ends.
__device__ __forceinline__ void p2p_pair(const float4 a, const float4 b, float2 nx, float2 ny, float2 nz,
                                         float2 soft2, float2& ax, float2& ay, float2& az, float2& pt) {
    const float2 dx = __fadd2_rn(make_float2(a.x, a.y), nx);
    const float2 dy = __fadd2_rn(make_float2(a.z, a.w), ny);
    const float2 dz = __fadd2_rn(make_float2(b.x, b.y), nz);
    float2 r2 = __ffma2_rn(dz, dz, soft2);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dx, dx, r2);
    const float2 inv = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    const float2 mi = __fmul2_rn(make_float2(b.z, b.w), inv);
    const float2 f = __fmul2_rn(mi, __fmul2_rn(inv, inv));
    ax = __ffma2_rn(f, dx, ax);
    ay = __ffma2_rn(f, dy, ay);
    az = __ffma2_rn(f, dz, az);
    pt = __fadd2_rn(pt, mi);
}

// The pair with the target's own body at half h (0 or 1) of it: that half
// becomes a massless body 1 + |x| away (no term). One unit alone is lost in the
// rounding where |x| is 2^24 and more (positions in metres): r = 0, 0 times infinity.
__device__ __forceinline__ void mask_self(float4& a, float4& b, int h, float x, float y, float z) {
    const float away = x + (1.f + fabsf(x));
    if (h == 0) {
        a.x = away; a.z = y; b.x = z; b.z = 0.f;
    } else {
        a.y = away; a.w = y; b.y = z; b.w = 0.f;
    }
}

// A warp per work unit, persistent, no block barriers. Two targets per lane:
// groups of G = ceil(nt / 2) lanes hold the targets and R = 32 / G groups split
// the source pairs of each tile. The sources are taken in chunks of up to
// P2PW_CHUNK leaves and P2PW_MAP pairs; a table gives each pair's leaf, so that
// staging a pair is a lookup, two 16-byte loads, six additions and two 16-byte
// stores, and the next tile's loads are in flight while a tile is computed. The
// target's own body is masked only in the tiles that overlap the target leaf.
// Bound by the FMA pipe and latency: per interaction 7.5 packed FP32x2 and MUFU
// instructions plus staging shared by the unit's targets; FMA pipe 62 % busy at 15
// bodies per leaf. Four blocks per SM of 128 registers and no unrolling of the
// pair loop (uniform 2^20, leaf 64: 2.03 ms; five blocks of 96 registers 2.08,
// six of 80 2.08; unrolled by two 2.12, 2.14, 2.12).
#define P2PW_CHUNK 128
#define P2PW_MAP 1024
#define P2PW_WARPS 4
#define P2PM_FLUSH 16

template <int TP>  // source pairs per tile
struct P2pWarpSmem {
    union {
        struct {
            float4 ta[TP];  // (x, x', y, y')
            float4 tz[TP];  // (z, z', m, m')
        } t;
        double red[8][32];  // the groups' sums at the end of a unit
    };
    float4 soff[P2PW_CHUNK];  // source leaf's centre - target leaf's centre; w: first pair of the leaf - its
                              // first position in the chunk (as bits)
    uint8_t own[P2PW_MAP];    // leaf of each pair of the chunk
};

template <int TP>
__global__ void __launch_bounds__(32 * P2PW_WARPS, 4) k_p2p_mixed(DirList L, CellsView cv, P2pUnits U,
                                                                const float4* __restrict__ pairs, float soft2_1,
                                                                double* __restrict__ ax, double* __restrict__ ay,
                                                                double* __restrict__ az, double* __restrict__ pot) {
    constexpr int PPT = TP / 32;  // pairs staged per lane
    __shared__ P2pWarpSmem<TP> smem_w[P2PW_WARPS];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    P2pWarpSmem<TP>& S = smem_w[threadIdx.x >> 5];
    const float2 soft2 = make_float2(soft2_1, soft2_1);
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
        const double4 gc = cv.geo[c];
        const int nt = (int)min((uint32_t)P2P_NT, tn - t0);
        const int G = (nt + 1) >> 1;
        const int R = 32 / G;
        const int g = lane % G, rep = lane / G;
        const bool active = rep < R;
        const int i0 = g, i1 = min(g + G, nt - 1);  // (an odd last target is computed twice, written once)
        float x0, y0, z0, x1, y1, z1;
        {
            const float* tp = reinterpret_cast<const float*>(pairs) + 8 * (size_t)pair_base(tf, (uint32_t)c);
            const uint32_t b0 = t0 + i0, b1 = t0 + i1;
            const float* q0 = tp + 8 * (size_t)(b0 >> 1) + (b0 & 1);
            const float* q1 = tp + 8 * (size_t)(b1 >> 1) + (b1 & 1);
            x0 = q0[0]; y0 = q0[2]; z0 = q0[4];
            x1 = q1[0]; y1 = q1[2]; z1 = q1[4];
        }
        const float2 nx0 = make_float2(-x0, -x0), ny0 = make_float2(-y0, -y0), nz0 = make_float2(-z0, -z0);
        const float2 nx1 = make_float2(-x1, -x1), ny1 = make_float2(-y1, -y1), nz1 = make_float2(-z1, -z1);
        double a0x = 0, a0y = 0, a0z = 0, p0 = 0, a1x = 0, a1y = 0, a1z = 0, p1 = 0;
        // FP32 partial sums, added into the FP64 sums after the tile with which
        // they reach P2PM_FLUSH source pairs (and at the end): at most P2PM_FLUSH - 1
        // pairs and a tile's share, half of its pairs or less (R >= 2)
        float2 q0x{0, 0}, q0y{0, 0}, q0z{0, 0}, q0p{0, 0}, q1x{0, 0}, q1y{0, 0}, q1z{0, 0}, q1p{0, 0};
        int held = 0;
        auto flush = [&]() {
            a0x += (double)(q0x.x + q0x.y);
            a0y += (double)(q0y.x + q0y.y);
            a0z += (double)(q0z.x + q0z.y);
            p0 += (double)(q0p.x + q0p.y);
            a1x += (double)(q1x.x + q1x.y);
            a1y += (double)(q1y.x + q1y.y);
            a1z += (double)(q1z.x + q1z.y);
            p1 += (double)(q1p.x + q1p.y);
            q0x = q0y = q0z = q0p = q1x = q1y = q1z = q1p = make_float2(0.f, 0.f);
            held = 0;
        };
        for (uint32_t sc = beg; sc < end;) {
            const int ns = (int)min((uint32_t)P2PW_CHUNK, end - sc);
            __syncwarp();
            // the chunk's source leaves: all loads of a kind at once, then the
            // positions of their pairs (one warp scan per 32 leaves)
            int src[P2PW_CHUNK / 32];
            uint32_t np[P2PW_CHUNK / 32], pb[P2PW_CHUNK / 32];
#pragma unroll
            for (int h = 0; h < P2PW_CHUNK / 32; ++h) {
                const int q = lane + 32 * h;
                src[h] = q < ns ? (int)L.src[sc + q] : -1;
            }
#pragma unroll
            for (int h = 0; h < P2PW_CHUNK / 32; ++h) {
                np[h] = 0;
                pb[h] = 0;
                if (src[h] >= 0) {
                    np[h] = (cv.count[src[h]] + 1) >> 1;
                    pb[h] = pair_base(cv.first[src[h]], (uint32_t)src[h]);
                    const double4 gs = cv.geo[src[h]];
                    S.soff[lane + 32 * h] = make_float4((float)(gs.x - gc.x), (float)(gs.y - gc.y),
                                                        (float)(gs.z - gc.z), 0.f);
                }
            }
            uint32_t base = 0;
            int nl = 0, self_at = -1;  // leaves whose pairs fit in the table; the target leaf's first position
#pragma unroll
            for (int h = 0; h < P2PW_CHUNK / 32; ++h) {
                const int q = lane + 32 * h;
                uint32_t incl = np[h];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += t;
                }
                incl += base;
                const uint32_t excl = incl - np[h];
                const bool fits = src[h] >= 0 && (incl <= P2PW_MAP || (q == 0));
                nl += __popc(__ballot_sync(FULL, fits));
                if (fits) {
                    S.soff[q].w = __uint_as_float(pb[h] - excl);
                    if (src[h] == c) self_at = (int)excl;
                    if (incl <= P2PW_MAP)
                        for (uint32_t e = excl; e < incl; ++e) S.own[e] = (uint8_t)q;
                }
                if (fits) np[h] = incl;  // keeps the last leaf's end
                base = __shfl_sync(FULL, incl, 31);
            }
            // pairs of the nl leaves: the end of the last one
            uint32_t total = 0;
#pragma unroll
            for (int h = 0; h < P2PW_CHUNK / 32; ++h) {
                const uint32_t v = __shfl_sync(FULL, np[h], (nl - 1) & 31);
                if ((nl - 1) >> 5 == h) total = v;
            }
            const bool mapped = total <= P2PW_MAP;
            const int sp = __reduce_max_sync(FULL, self_at);
            __syncwarp();
            sc += nl;
            float4 ra[PPT], rz[PPT], ro[PPT];
            auto issue = [&](uint32_t b0) {  // load the pairs of the tile at b0
#pragma unroll
                for (int e = 0; e < PPT; ++e) {
                    const uint32_t p = b0 + lane + 32 * e;
                    if (p < total) {
                        ro[e] = S.soff[mapped ? S.own[p] : 0];
                        const float4* s = pairs + 2 * (size_t)(p + __float_as_uint(ro[e].w));
                        ra[e] = s[0];
                        rz[e] = s[1];
                    }
                }
            };
            issue(0);
            for (uint32_t b0 = 0; b0 < total; b0 += TP) {
                const int npair = (int)min((uint32_t)TP, total - b0);
                __syncwarp();
#pragma unroll
                for (int e = 0; e < PPT; ++e) {
                    const int p = lane + 32 * e;
                    if (p < npair) {
                        const float4 o = ro[e];
                        S.t.ta[p] = make_float4(ra[e].x + o.x, ra[e].y + o.x, ra[e].z + o.y, ra[e].w + o.y);
                        S.t.tz[p] = make_float4(rz[e].x + o.z, rz[e].y + o.z, rz[e].z, rz[e].w);
                    }
                }
                __syncwarp();
                issue(b0 + TP);
                if (active) {
                    const int last = sp + (int)((tn + 1) >> 1);  // the target leaf's own pairs: sp .. last - 1
                    if (sp < 0 || sp >= (int)b0 + npair || last <= (int)b0) {
#pragma unroll 1
                        for (int j = rep; j < npair; j += R) {
                            const float4 a = S.t.ta[j], b = S.t.tz[j];
                            p2p_pair(a, b, nx0, ny0, nz0, soft2, q0x, q0y, q0z, q0p);
                            p2p_pair(a, b, nx1, ny1, nz1, soft2, q1x, q1y, q1z, q1p);
                        }
                    } else {
                        // the target's own body is body t0 + i of the leaf
                        const int s0 = 2 * (sp - (int)b0) + (int)t0 + i0, s1 = 2 * (sp - (int)b0) + (int)t0 + i1;
                        for (int j = rep; j < npair; j += R) {
                            const float4 a = S.t.ta[j], b = S.t.tz[j];
                            float4 a0 = a, b0v = b, a1 = a, b1v = b;
                            if (j == (s0 >> 1)) mask_self(a0, b0v, s0 & 1, x0, y0, z0);
                            if (j == (s1 >> 1)) mask_self(a1, b1v, s1 & 1, x1, y1, z1);
                            p2p_pair(a0, b0v, nx0, ny0, nz0, soft2, q0x, q0y, q0z, q0p);
                            p2p_pair(a1, b1v, nx1, ny1, nz1, soft2, q1x, q1y, q1z, q1p);
                        }
                    }
                    held += (npair - rep + R - 1) / R;
                    if (held >= P2PM_FLUSH) flush();
                }
            }
        }
        flush();
        __syncwarp();
        S.red[0][lane] = a0x; S.red[1][lane] = a0y; S.red[2][lane] = a0z; S.red[3][lane] = p0;
        S.red[4][lane] = a1x; S.red[5][lane] = a1y; S.red[6][lane] = a1z; S.red[7][lane] = p1;
        __syncwarp();
        // outputs: nt targets x 4 components, each the sum over the R groups
        // in group order
        for (int o = lane; o < 4 * nt; o += 32) {
            const int t = o >> 2, comp = o & 3;
            const int gi = t < G ? t : t - G;  // target t = gi + half * G
            const int row = (t < G ? 0 : 4) + comp;
            double v = 0.0;
            for (int r = 0; r < R; ++r) v += S.red[row][r * G + gi];
            if (ns_all == 1) {
                double* out = comp == 0 ? ax : comp == 1 ? ay : comp == 2 ? az : pot;
                out[tf + t0 + t] = v;
            } else {
                reinterpret_cast<double*>(U.part + U.soff[c] + (size_t)share * tn + t0 + t)[comp] = v;
            }
        }
        __syncwarp();
    }
}

template <int TP>
static void launch_tile(int nsm, cudaStream_t s, DirList L, CellsView cv, P2pUnits U, const float4* pairs, float soft2,
                        double* ax, double* ay, double* az, double* pot) {
    // persistent blocks: as many as fit on an SM at once, no more than there are units
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_p2p_mixed<TP>, 32 * P2PW_WARPS, 0) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const unsigned need = (unsigned)std::min<uint64_t>(((uint64_t)U.nunits + P2PW_WARPS - 1) / P2PW_WARPS, 1u << 30);
    k_p2p_mixed<TP><<<std::max(1u, std::min(need, (unsigned)(nsm * per_sm))), 32 * P2PW_WARPS, 0, s>>>(
        L, cv, U, pairs, soft2, ax, ay, az, pot);
}

void launch_p2p_mixed(int tile, int nsm, cudaStream_t s, DirList L, int ncells, CellsView cv, P2pUnits U, size_t n,
                      const int32_t* body_leaf, const double* x, const double* y, const double* z, const double* m,
                      float4* pairs, float soft2, double* ax, double* ay, double* az, double* pot) {
    k_local_pairs<<<grid_for(n, 256), 256, 0, s>>>(n, body_leaf, cv, x, y, z, m, reinterpret_cast<float*>(pairs));
    // `tile` bodies per block of four warps: 64 pairs per warp's tile at 512
    if (tile <= 256) launch_tile<32>(nsm, s, L, cv, U, pairs, soft2, ax, ay, az, pot);
    else if (tile <= 512) launch_tile<64>(nsm, s, L, cv, U, pairs, soft2, ax, ay, az, pot);
    else launch_tile<128>(nsm, s, L, cv, U, pairs, soft2, ax, ay, az, pot);
    launch_p2p_combine(s, ncells, L, cv, U, ax, ay, az, pot);
}

}  // namespace fmmx
