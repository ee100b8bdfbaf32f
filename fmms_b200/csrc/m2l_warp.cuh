// Rotation M2L, one lane per directed translation, templated on the
// arithmetic type T (double for the plain form, float for the mixed form) and
// the expansion order P.
//
// Algorithm (the reference's RotCtx::m2l_pair/apply, rotation.rs:262-435,
// Dehnen 2014 A.6.1): back-rotate the source multipole with two x<->z swaps
// B_k around a z-rotation by -β, translate along z with the diagonal kernel
// F~_n^m = sum_k b_k^{-m} (n+k)!/R^{n+k+1}, rotate forward with B_n^T, and add
// into the destination's local expansion.
//
// B200 structure:
//  - A warp owns one destination cell; each lane takes every 32nd of its
//    sources, so 32 translations run side by side. A lane adds its results
//    into its own column of shared memory; the columns are summed once per
//    destination, in a fixed order (no atomics).
//  - Expansions of a real field satisfy v_{-m} = (-1)^m conj(v_m); so do all
//    intermediate vectors (rotations map real fields to real fields). Only
//    m >= 0 is kept, and each swap matvec splits into two real products,
//    Re(s) = P_k Re(u), Im(s) = Q_k Im(u) with
//    P_k[r][c] = B_k[r][c] + (-1)^c B_k[r][-c], Q_k[r][c] = B_k[r][c] - (-1)^c B_k[r][-c].
//    Both are zero in a parity pattern, and the imaginary part at m = 0 is zero.
//  - P is a template parameter and every table a constexpr, so each
//    coefficient is an immediate operand of the FMA that uses it (FP64 values
//    that do not fit one come from the constant bank). The tables used to be
//    read from __constant__ memory: 4,717 instructions per translation at
//    p = 10 (FP32), about 915 of them coefficient loads.
//  - What the algorithm's structure makes zero or cancels is left out by hand,
//    since IEEE arithmetic does not let the compiler do it: the axial step
//    couples only m <= min(k, P - k), so the second back product needs just
//    those rows and the first forward product just those columns; the factors
//    i^m of the two rotations cancel through the axial step; (n-m)!(n+m)! and
//    its inverses are folded into the first back product and the axial
//    coefficients, and the last one is applied once per destination, to the sum.
//  - Phases e^{imα}, e^{imβ} come from powers of (x + iy)/ρ_xy and
//    (z + iρ_xy)/R: no trigonometric calls.
//  - SCALED expansions (mixed form) carry M^_k = M_k / l_a^k and
//    F^_n = F_n l_b^{n+1}, l the cell's radius, so FP32 never overflows at
//    high order: the axial kernel becomes (n+k)! (l_a/R)^k (l_b/R)^{n+1}.
#pragma once

#include <type_traits>
#include <utility>

#include "common.cuh"
#include "kernels.h"

namespace fmmx {

__host__ __device__ constexpr int rot_hx(int n, int m) { return n * (n + 1) / 2 + m; }
#define ROTW_MAXP 16

// Swap matrices B_n (Dehnen 2014 eq 63; rotation.rs:136-211) of one degree and
// their real half-basis forms, built degree by degree at compile time.
struct SwapFull {
    double v[2 * ROTW_MAXP + 1][2 * ROTW_MAXP + 1];
};
constexpr SwapFull swap_next(const SwapFull& b, int n) {  // B_{n-1} -> B_n
    SwapFull o{};
    for (int mr = 0; mr <= 2 * n; ++mr) {
        const int mm = mr - n;
        const int row = mm == n ? 2 * n - 2 : mm == -n ? 0 : mr - 1;  // row of B_{n-1}
        const double s = mm == n ? 1.0 : mm == -n ? -1.0 : 0.0;
        for (int lc = 0; lc <= 2 * n; ++lc) {
            const double lm = lc >= 2 ? b.v[row][lc - 2] : 0.0;                    // l - 1
            const double l0 = lc >= 1 && lc <= 2 * n - 1 ? b.v[row][lc - 1] : 0.0;  // l
            const double lp = lc <= 2 * n - 2 ? b.v[row][lc] : 0.0;                // l + 1
            o.v[mr][lc] = s == 0.0 ? (lm - lp) * 0.5 : (lm + lp + 2.0 * s * l0) * 0.5;
        }
    }
    return o;
}
template <int N>
struct SwapOf {
    static constexpr SwapFull b = swap_next(SwapOf<N - 1>::b, N);
};
constexpr SwapFull swap_zero() {
    SwapFull o{};
    o.v[0][0] = 1.0;
    return o;
}
template <>
struct SwapOf<0> {
    static constexpr SwapFull b = swap_zero();
};

// half-basis entry (r, c) of B_k (or its transpose): the P form (IM = false)
// and the Q form (IM = true)
template <int K, bool TR, bool IM>
constexpr double half_entry(int r, int c) {
    const double a = TR ? SwapOf<K>::b.v[c + K][r + K] : SwapOf<K>::b.v[r + K][c + K];
    if (c == 0) return a;
    const double b = TR ? SwapOf<K>::b.v[-c + K][r + K] : SwapOf<K>::b.v[r + K][-c + K];
    const double sg = (c & 1) ? -1.0 : 1.0;
    return IM ? a - sg * b : a + sg * b;
}
// the zero pattern the products rely on: P[r][c] = 0 unless r + c + K is even,
// Q[r][c] = 0 (c >= 1) unless r >= 1 and r + c + K is odd
template <int K, bool TR>
constexpr bool half_pattern_ok() {
    for (int r = 0; r <= K; ++r)
        for (int c = 0; c <= K; ++c) {
            if (((r + c + K) & 1) != 0 && half_entry<K, TR, false>(r, c) != 0.0) return false;
            if (c >= 1 && !(r >= 1 && ((r + c + K) & 1) == 1) && half_entry<K, TR, true>(r, c) != 0.0) return false;
        }
    return true;
}
constexpr double rot_fact(int n) {
    double f = 1.0;
    for (int i = 2; i <= n; ++i) f *= (double)i;
    return f;
}
constexpr double rot_fm(int n, int m) { return rot_fact(n - m) * rot_fact(n + m); }  // (n-m)!(n+m)!

// Pair phases e^{imα}, e^{imβ} (m = 1..P): in the lane's shared-memory
// columns (FP64 at high order: registers are too few) or in registers.
template <typename T>
struct PhSmem {
    const cplx<T>* a;
    const cplx<T>* b;
    __device__ __forceinline__ cplx<T> A(int m) const { return a[32 * (m - 1)]; }
    __device__ __forceinline__ cplx<T> B(int m) const { return b[32 * (m - 1)]; }
};
template <typename T, int P>
struct PhRegs {
    cplx<T> a[P], b[P];
    __device__ __forceinline__ cplx<T> A(int m) const { return a[m - 1]; }
    __device__ __forceinline__ cplx<T> B(int m) const { return b[m - 1]; }
};

// Compiler barrier between degrees: it bounds the live registers where the
// expansion does not fit in them next to two degrees' temporaries.
template <typename T, int P>
__device__ __forceinline__ void degree_fence() {
    if constexpr (P > (sizeof(T) == 4 ? 10 : 6)) asm volatile("" ::: "memory");
}

// compile-time loop: f(integral_constant<m>) for m = M..N-1
template <int M, int N>
struct Unroll {
    template <class F>
    __device__ __forceinline__ static void run(F&& f) {
        if constexpr (M < N) {
            f(std::integral_constant<int, M>{});
            Unroll<M + 1, N>::run(f);
        }
    }
};

// orders m <= ROT_M that the axial step couples at degree k of an order-P expansion
__host__ __device__ constexpr int rot_mmax(int P, int k) { return k < P - k ? k : P - k; }

// One swap product of degree K: rows 0..NR-1 from columns 0..NC-1,
// Re(s) = P Re(v), Im(s) = Q Im(v), si[0] unused. TR: the matrices of B_K^T.
// FM: the columns carry the factor (K-c)!(K+c)! (the first back product).
template <typename T, int K, bool TR, bool FM, int NR, int NC, int N>
__device__ __forceinline__ void swap_product(const T (&vr)[N], const T (&vi)[N], T (&sr)[N], T (&si)[N]) {
    static_assert(half_pattern_ok<K, TR>(), "swap matrix pattern");
    Unroll<0, NR>::run([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        T a = T(0), b = T(0);
        Unroll<0, NC>::run([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr double f = FM ? rot_fm(K, q) : 1.0;
            if constexpr (((r + q + K) & 1) == 0) {
                constexpr double c = half_entry<K, TR, false>(r, q) * f;
                if constexpr (c != 0.0) a += T(c) * vr[q];
            }
            if constexpr (r >= 1 && q >= 1 && ((r + q + K) & 1) == 1) {
                constexpr double c = half_entry<K, TR, true>(r, q) * f;
                if constexpr (c != 0.0) b += T(c) * vi[q];
            }
        });
        sr[r] = a;
        si[r] = b;
    });
}

// The back-rotated multipole at the coupled orders: entry (k, m) at
// tr_off(k) + m, m <= rot_mmax(P, k); times (l_a/R)^k.
template <int P>
struct TOff {
    __host__ __device__ static constexpr int at(int k) {
        int s = 0;
        for (int j = 0; j < k; ++j) s += rot_mmax(P, j) + 1;
        return s;
    }
};
template <typename T, int P>
struct TRegs {
    T re[TOff<P>::at(P + 1)], im[TOff<P>::at(P + 1)];
};

template <typename T, int P, int K, bool FULL_LAYOUT, class PH>
__device__ __forceinline__ void back_degree(const cplx<T>* __restrict__ ms, const PH& ph, TRegs<T, P>& t, T sa,
                                            T& sak, T cap) {
    typedef cplx<T> Z;
    constexpr int N = K + 1;
    constexpr int NT = rot_mmax(P, K) + 1;  // rows the axial step reads
    constexpr int E = TOff<P>::at(K);
    // FP32 half layout: every cell starts on 16 bytes (the cell stride is
    // half_stride(P), even), so entry pairs that start on an even index load
    // as one float4
    Z Mv[N];
    constexpr bool PAIRS = sizeof(T) == 4 && !FULL_LAYOUT;
    constexpr int B0 = rot_hx(K, 0);
    Unroll<0, N>::run([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        if constexpr (PAIRS && ((B0 + j) & 1) == 0 && j + 1 < N) {
            const float4 v = *reinterpret_cast<const float4*>(ms + B0 + j);
            Mv[j] = mk<T>(v.x, v.y);
            Mv[j + 1] = mk<T>(v.z, v.w);
        } else if constexpr (!PAIRS || ((B0 + j) & 1) == 0 || j == 0) {
            Mv[j] = ms[FULL_LAYOUT ? (K * (K + 1) + j) : rot_hx(K, j)];
        }
    });
    if constexpr (K == 0) {
        t.re[E] = Mv[0].re;
    } else {
        T vr[N], vi[N], sr[N], si[N];
        vr[0] = Mv[0].re;
        vi[0] = T(0);
        Unroll<1, N>::run([&](auto mc) {  // u = (-i)^m e^{imα} conj(M)
            constexpr int m = decltype(mc)::value;
            const Z M = Mv[m], p = ph.A(m);
            const T a = p.re * M.re + p.im * M.im, b = p.im * M.re - p.re * M.im;
            if constexpr ((m & 3) == 0) { vr[m] = a; vi[m] = b; }
            else if constexpr ((m & 3) == 1) { vr[m] = b; vi[m] = -a; }
            else if constexpr ((m & 3) == 2) { vr[m] = -a; vi[m] = -b; }
            else { vr[m] = -b; vi[m] = a; }
        });
        swap_product<T, K, false, true, N, N, N>(vr, vi, sr, si);
        vr[0] = sr[0];
        Unroll<1, N>::run([&](auto rc) {
            constexpr int r = decltype(rc)::value;
            const Z p = ph.B(r);
            const T a = sr[r], b = si[r];
            vr[r] = a * p.re - b * p.im;
            vi[r] = a * p.im + b * p.re;
        });
        swap_product<T, K, false, false, NT, N, N>(vr, vi, sr, si);
        t.re[E] = sr[0] * sak;
        Unroll<1, NT>::run([&](auto rc) {
            constexpr int r = decltype(rc)::value;
            t.re[E + r] = sr[r] * sak;
            t.im[E + r] = si[r] * sak;
        });
    }
    sak = min(sak * sa, cap);
    degree_fence<T, P>();
}

template <typename T, int P, bool FULL_LAYOUT, class PH, int... Ks>
__device__ __forceinline__ void back_all(const cplx<T>* __restrict__ ms, const PH& ph, TRegs<T, P>& t, T sa, T cap,
                                         std::integer_sequence<int, Ks...>) {
    T sak = min(sa, cap);  // of degree 1 (degree 0 carries no scale)
    (back_degree<T, P, Ks, FULL_LAYOUT, PH>(ms, ph, t, Ks == 0 ? T(1) : sa, sak, cap), ...);
}

// Degree K of the translated expansion, formed where the forward rotation
// needs it: with the rotations' factors of i cancelled its swapped-in vector is
// g[m] = conj(sum_{k=m}^{P-K} t[k][m] (K+k)! / ((k-m)!(k+m)! (K-m)!(K+m)!)) (l_b/R)^{K+1}.
// Then the forward rotation, added into the lane's column without its last
// factor i^m (K-m)!(K+m)!.
template <typename T, int P, int K, class PH>
__device__ __forceinline__ void fwd_degree(const TRegs<T, P>& t, cplx<T>* __restrict__ col, const PH& ph, T& sbn, T sb,
                                           T cap) {
    typedef cplx<T> Z;
    constexpr int N = K + 1;
    constexpr int NM = rot_mmax(P, K) + 1;
    T vr[N], vi[N], sr[N], si[N];
    Unroll<0, NM>::run([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        T ar = T(0), ai = T(0);
        Unroll<m, P - K + 1>::run([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            if constexpr (m <= rot_mmax(P, k)) {
                constexpr T c = T(rot_fact(K + k) / rot_fm(k, m) / rot_fm(K, m));
                ar += t.re[TOff<P>::at(k) + m] * c;
                if constexpr (m >= 1) ai -= t.im[TOff<P>::at(k) + m] * c;
            }
        });
        vr[m] = ar * sbn;
        vi[m] = ai * sbn;
    });
    sbn = min(sbn * sb, cap);
    if constexpr (K == 0) {
        col[0].re += vr[0];
    } else {
        swap_product<T, K, true, false, N, NM, N>(vr, vi, sr, si);
        vr[0] = sr[0];
        vi[0] = T(0);
        Unroll<1, N>::run([&](auto rc) {  // q = conj(e^{irβ}) s
            constexpr int r = decltype(rc)::value;
            const Z p = ph.B(r);
            const T a = sr[r], b = si[r];
            vr[r] = a * p.re + b * p.im;
            vi[r] = b * p.re - a * p.im;
        });
        swap_product<T, K, true, false, N, N, N>(vr, vi, sr, si);
        col[32 * rot_hx(K, 0)].re += sr[0];
        Unroll<1, N>::run([&](auto rc) {  // out = e^{irα} t; i^r and the factorials follow on the sum
            constexpr int r = decltype(rc)::value;
            const Z p = ph.A(r);
            const T a = sr[r], b = si[r];
            Z o = col[32 * rot_hx(K, r)];
            o.re += a * p.re - b * p.im;
            o.im += a * p.im + b * p.re;
            col[32 * rot_hx(K, r)] = o;
        });
    }
    degree_fence<T, P>();
}

template <typename T, int P, class PH, int... Ks>
__device__ __forceinline__ void fwd_all(const TRegs<T, P>& t, cplx<T>* __restrict__ col, const PH& ph, T sb, T cap,
                                        std::integer_sequence<int, Ks...>) {
    T sbn = sb;
    (fwd_degree<T, P, Ks, PH>(t, col, ph, sbn, sb, cap), ...);
}

// (n-m)!(n+m)! on the half index, for the destination's sums
template <typename T>
struct FmTable {
    T v[(ROTW_MAXP + 1) * (ROTW_MAXP + 2) / 2];
};
template <typename T>
constexpr FmTable<T> make_fm_table() {
    FmTable<T> t{};
    for (int n = 0; n <= ROTW_MAXP; ++n)
        for (int m = 0; m <= n; ++m) t.v[rot_hx(n, m)] = T(rot_fm(n, m));
    return t;
}
static __device__ const FmTable<ROTW_T> g_rot_fm = make_fm_table<ROTW_T>();

// FP64 keeps the phases in registers up to this order (p = 10: 3.69 -> 3.48 ms
// at N = 2^18 against shared memory, which then holds one warp less per SM)
#define ROTW_PH64_MAXP 10
// `cap` bounds the scale powers of the normalised (mixed) form: a power only
// exceeds 1 where the moments it multiplies are exactly zero (a cell of radius
// 0), and the cap keeps that product 0 instead of 0 * inf.
template <typename T, bool SCALED>
__device__ __forceinline__ constexpr T rotw_cap() { return SCALED ? T(1e30) : T(INFINITY); }

template <typename T, int P>
constexpr bool rotw_ph_regs() { return sizeof(T) == 4 || P <= ROTW_PH64_MAXP; }

// The destination's sum over the lanes' columns, times i^m (n-m)!(n+m)!: lane
// l takes entries l, l + 32, ..., each starting at its own column so that the
// reads hit distinct banks.
template <typename T, int P, bool FULL_LAYOUT>
__device__ __forceinline__ void rotw_finish(int c, const cplx<T>* __restrict__ sbuf, cplx<T>* __restrict__ loc,
                                            int lane) {
    constexpr int H = (P + 1) * (P + 2) / 2;
    constexpr int DIM = (P + 1) * (P + 1);
    __syncwarp();
    for (int e = lane; e < H; e += 32) {
        T sr = T(0), si = T(0);
        const cplx<T>* row = sbuf + 32 * e;
#pragma unroll 8
        for (int l = 0; l < 32; ++l) {
            const cplx<T> v = row[(l + lane) & 31];
            sr += v.re;
            si += v.im;
        }
        int n = 0;
        while ((n + 1) * (n + 2) / 2 <= e) ++n;
        const int m = e - n * (n + 1) / 2;
        const T f = g_rot_fm.v[e];
        const T fr = sr * f, fi = si * f;
        const T re = (m & 1) ? ((m & 2) ? fi : -fi) : ((m & 2) ? -fr : fr);
        const T im = (m & 1) ? ((m & 2) ? -fr : fr) : ((m & 2) ? -fi : fi);
        if (FULL_LAYOUT) {
            cplx<T>* out = loc + (size_t)c * DIM;
            out[n * (n + 1) + m] = mk<T>(re, im);
            if (m > 0) {
                const T sg = (m & 1) ? T(-1) : T(1);
                out[n * (n + 1) - m] = mk<T>(sg * re, -sg * im);
            }
        } else {
            loc[(size_t)c * half_stride(P) + e] = mk<T>(re, im);
        }
    }
    __syncwarp();
}

template <typename T, int P>
constexpr size_t rotw_smem_per_warp() {
    return (size_t)32 * ((P + 1) * (P + 2) / 2 + (rotw_ph_regs<T, P>() ? 0 : 2 * P)) * sizeof(cplx<T>);
}

// Resident warps per SM: what the columns leave room for in 224 KB of shared
// memory (1 KB per block is the system's), and as many as the registers allow
// without spilling the expansion. FP32 keeps it, with the phases and two degrees'
// temporaries, in 128 registers up to P = 6 (16 warps), in 168 up to P = 10 (12
// warps) and in 255 above (8 warps; 9 of 224: P = 12 2.24 ms against 1.84). FP64
// uses 166 registers at P = 4 (12 warps) and 246 and more from P = 5 (8 warps);
// from P = 10 it spills at 255.
template <typename T, int P>
constexpr int rotw_warps_per_sm() {
    const int by_smem = (int)(224 * 1024 / (rotw_smem_per_warp<T, P>() + 1024));
    const int by_regs = sizeof(T) == 4 ? (P <= 6 ? 16 : P <= 10 ? 12 : 8) : (P <= 4 ? 12 : 8);
    return by_smem < by_regs ? by_smem : by_regs;
}

// Warps of a block: more than one run in step (see k_m2l_rotw).
template <typename T, int P>
constexpr int rotw_block_warps() {
    constexpr int w = rotw_warps_per_sm<T, P>();
    if (sizeof(T) == 4) return P <= 10 ? 1 : w;
    return P <= 9 ? 1 : P == 10 ? w / 2 : w;
}

// Geometry, phases and the back rotation of one translation (source cell src).
template <typename T, int P, bool SCALED, bool FULL_LAYOUT>
__device__ __forceinline__ void rotw_back(uint32_t src, double bx, double by, double bz, T lb, const CellsView& cv,
                                          const T* __restrict__ scale, const cplx<T>* __restrict__ mom,
                                          PhRegs<T, P>& phr, cplx<T>* pha, cplx<T>* phb, TRegs<T, P>& t, T& sb) {
    typedef cplx<T> Z;
    constexpr bool PH_REGS = rotw_ph_regs<T, P>();
    // geometry in FP64: r = s_B - z_A
    const double rx = bx - cv.cx[src], ry = by - cv.cy[src], rz = bz - cv.cz[src];
    const double rxy2 = rx * rx + ry * ry;
    const double iR = rsqrt(rxy2 + rz * rz);
    double ear = 1.0, eai = 0.0, rxy = 0.0;
    if (rxy2 > 0.0) {
        const double ir = rsqrt(rxy2);
        rxy = rxy2 * ir;
        ear = rx * ir;
        eai = ry * ir;
    }
    const Z ea = mk<T>((T)ear, (T)eai), eb = mk<T>((T)(rz * iR), (T)(rxy * iR));
    Z a = ea, b = eb;
#pragma unroll
    for (int m = 1; m <= P; ++m) {
        if (PH_REGS) {
            phr.a[m - 1] = a;
            phr.b[m - 1] = b;
        } else {
            pha[32 * (m - 1)] = a;
            phb[32 * (m - 1)] = b;
        }
        a = zmul(a, ea);
        b = zmul(b, eb);
    }
    T sa;  // per-degree scale factors of the axial kernel
    if (SCALED) {
        sa = (T)((double)scale[src] * iR);
        sb = (T)((double)lb * iR);
    } else {
        sa = (T)iR;
        sb = (T)iR;
    }
    const Z* ms = mom + (size_t)src * (FULL_LAYOUT ? (P + 1) * (P + 1) : half_stride(P));
    if constexpr (PH_REGS)
        back_all<T, P, FULL_LAYOUT>(ms, phr, t, sa, rotw_cap<T, SCALED>(), std::make_integer_sequence<int, P + 1>{});
    else
        back_all<T, P, FULL_LAYOUT>(ms, PhSmem<T>{pha, phb}, t, sa, rotw_cap<T, SCALED>(),
                                    std::make_integer_sequence<int, P + 1>{});
}

// Axial step and forward rotation, added into the lane's column.
template <typename T, int P, bool SCALED>
__device__ __forceinline__ void rotw_fwd(const TRegs<T, P>& t, const PhRegs<T, P>& phr, const cplx<T>* pha,
                                         const cplx<T>* phb, T sb, cplx<T>* col) {
    if constexpr (rotw_ph_regs<T, P>())
        fwd_all<T, P>(t, col, phr, sb, rotw_cap<T, SCALED>(), std::make_integer_sequence<int, P + 1>{});
    else
        fwd_all<T, P>(t, col, PhSmem<T>{pha, phb}, sb, rotw_cap<T, SCALED>(),
                      std::make_integer_sequence<int, P + 1>{});
}

// With a work counter the blocks are persistent and their warps pull
// destination cells from it; without one (work == nullptr) block b handles the
// destinations W b .. W b + W - 1, so every block is short-lived and the block
// scheduler can interleave kernels of higher-priority streams between them.
//
// W = 1: independent warps. W > 1 (high orders): each warp still works on a
// destination of its own, 32 sources (a chunk) at a time, but the block's warps
// meet at a barrier before each chunk and in its middle. The unrolled code of a
// chunk is larger than the instruction caches there (about 90 KB at p = 12),
// and warps in step fetch it once for all of them: FP64 p = 12, no_instruction
// stalls 3.9 -> 0.3 per issue.
// Measured, ms of this kernel at N = 2^18 (uniform cube, leaf 64, theta 0.5,
// 5.95 M translations), independent | all the SM's warps in step:
//   FP32  p = 8: 0.56 | 0.86   10: 1.14 | 1.63   11: 1.88 | 1.56   12: 3.07 | 1.84   14: 6.98 | 2.97   16: 14.5 | 5.5
//   FP64  p = 8: 1.33 | 1.78    9: 2.30 | 2.59   10: 3.37 | 3.81 (two blocks of 3: 3.00)   12: 10.0 | 6.3   14: 17.5 | 17.1
// so FP32 runs in step from p = 11 and FP64 from p = 10. The kernel before, with
// its tables in constant memory: FP32 p = 8 0.88, 10 1.82, 12 4.90, 14 8.70;
// FP64 p = 6 1.64, 8 3.76, 10 6.14, 12 17.9, 14 38.9 ms. The FP32 form is
// bound by issue and instruction latency (12 warps per SM, 168 registers), the
// FP64 form by latency at 2 to 8 warps per SM (shared memory for the columns).
// FP64 p = 14 takes twice p = 13 (17.1 and 8.6 ms): two warps of columns fit instead
// of three, half again as much is spilled (1.6 KB a thread), and two warps in step
// share each fetch between them instead of three (no_instruction 1.8 per issue).
template <typename T, int P, bool SCALED, bool FULL_LAYOUT, int W>
__global__ void __launch_bounds__(32 * W, (rotw_warps_per_sm<T, P>() / W))
    k_m2l_rotw(DirList L, int ncells, CellsView cv, const T* __restrict__ scale, const cplx<T>* __restrict__ mom,
               cplx<T>* __restrict__ loc, int* __restrict__ work) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    typedef cplx<T> Z;
    constexpr int H = (P + 1) * (P + 2) / 2;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Z* sbuf = reinterpret_cast<Z*>(smem_raw) + (size_t)wid * (rotw_smem_per_warp<T, P>() / sizeof(Z));
    Z* col = sbuf + lane;           // this lane's column: entry e at col[32 e]
    Z* pha = sbuf + 32 * H + lane;  // e^{imα}, m = 1..P (where not in registers)
    Z* phb = pha + 32 * P;          // e^{imβ}
    const uint32_t* __restrict__ srcs = L.src;
    auto clear = [&]() {
#pragma unroll 4
        for (int e = 0; e < H; ++e) col[32 * e] = mk<T>(T(0), T(0));
    };
    if constexpr (W == 1) {
        for (;;) {
            int c = blockIdx.x;
            if (work) {
                if (lane == 0) c = atomicAdd(work, 1);
                c = __shfl_sync(0xffffffffu, c, 0);
            }
            if (c >= ncells) break;
            const uint32_t beg = L.seg_begin[c], end = L.seg_end[c];
            if (beg < end) {
                const double bx = cv.cx[c], by = cv.cy[c], bz = cv.cz[c];
                const T lb = SCALED ? scale[c] : T(1);
                clear();
                for (uint32_t i = beg + lane; i < end; i += 32) {
                    PhRegs<T, P> phr;
                    TRegs<T, P> t;
                    T sb;
                    rotw_back<T, P, SCALED, FULL_LAYOUT>(srcs[i], bx, by, bz, lb, cv, scale, mom, phr, pha, phb, t, sb);
                    rotw_fwd<T, P, SCALED>(t, phr, pha, phb, sb, col);
                }
                rotw_finish<T, P, FULL_LAYOUT>(c, sbuf, loc, lane);
            }
            if (!work) break;
        }
    } else {
        int c = -1, nextc = work ? 0 : blockIdx.x * W + wid;
        uint32_t i = 0, end = 0;
        double bx = 0, by = 0, bz = 0;
        T lb = T(1);
        for (;;) {
            while (i >= end) {  // the next destination with sources
                if (c >= 0) rotw_finish<T, P, FULL_LAYOUT>(c, sbuf, loc, lane);
                c = -1;
                if (work && nextc < ncells) {
                    int g = 0;
                    if (lane == 0) g = atomicAdd(work, 1);
                    nextc = __shfl_sync(0xffffffffu, g, 0);
                }
                if (nextc >= ncells) break;
                i = L.seg_begin[nextc];
                end = L.seg_end[nextc];
                if (i < end) {
                    c = nextc;
                    bx = cv.cx[c];
                    by = cv.cy[c];
                    bz = cv.cz[c];
                    if (SCALED) lb = scale[c];
                    clear();
                }
                if (!work) nextc = ncells;
            }
            if (!__syncthreads_or(c >= 0)) break;  // no warp of the block has a destination left
            const bool active = c >= 0 && i + lane < end;
            PhRegs<T, P> phr;
            TRegs<T, P> t;
            T sb = T(0);
            if (active)
                rotw_back<T, P, SCALED, FULL_LAYOUT>(srcs[i + lane], bx, by, bz, lb, cv, scale, mom, phr, pha, phb, t,
                                                     sb);
            __syncthreads();
            if (active) rotw_fwd<T, P, SCALED>(t, phr, pha, phb, sb, col);
            i += 32;
        }
    }
}

}  // namespace fmmx
