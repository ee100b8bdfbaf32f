// Host side of the warp rotation M2L: the launchers.
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace fmmx {

cudaError_t launch_rotw_f64(int p, DirList L, int nc, CellsView cv, const zd* mom, zd* loc, int* work, int nsm,
                            cudaStream_t s);
cudaError_t launch_rotw_f32(int p, DirList L, int nc, CellsView cv, const float* scale, const zf* mom, zf* loc,
                            int* work, int nsm, cudaStream_t s);
constexpr int kRotwMaxP = 16;

}  // namespace fmmx
