// FP32 instantiation of the warp-per-destination rotation M2L (mixed form:
// size-normalised expansions, m >= 0 half layout).
#define ROTW_T float
#include "m2l_warp.cuh"
#include "rotw.h"

namespace fmmx {

template <int P>
static cudaError_t launch_p(DirList L, int nc, CellsView cv, const float* scale, const zf* mom, zf* loc, int* work,
                            int nsm, cudaStream_t s) {
    constexpr int W = rotw_block_warps<float, P>();
    constexpr size_t smem = W * rotw_smem_per_warp<float, P>();
    auto kern = k_m2l_rotw<float, P, true, false, W>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    constexpr int per_sm = rotw_warps_per_sm<float, P>() / W;
    kern<<<work ? nsm * per_sm : (unsigned)((nc + W - 1) / W), 32 * W, smem, s>>>(L, nc, cv, scale, mom, loc, work);
    return cudaGetLastError();
}

cudaError_t launch_rotw_f32(int p, DirList L, int nc, CellsView cv, const float* scale, const zf* mom, zf* loc,
                            int* work, int nsm, cudaStream_t s) {
    switch (p) {
#define CASE(P) \
    case P: return launch_p<P>(L, nc, cv, scale, mom, loc, work, nsm, s);
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10) CASE(11) CASE(12)
        CASE(13) CASE(14) CASE(15) CASE(16)
#undef CASE
    }
    return cudaErrorInvalidValue;
}

}  // namespace fmmx
