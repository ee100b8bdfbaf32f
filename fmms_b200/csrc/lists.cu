// Prefix sums of the engine, via CUB's single-pass device scan.
#include <cub/device/device_scan.cuh>

#include "common.cuh"
#include "kernels.h"

namespace fmmx {

namespace {
struct Add4 {
    __host__ __device__ uint4 operator()(const uint4& a, const uint4& b) const {
        return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    }
};
}  // namespace

size_t scan_u32_temp(int n) {
    size_t a = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, a, (const uint32_t*)nullptr, (uint32_t*)nullptr, n);
    return a;
}

cudaError_t scan_u32(void* tmp, size_t tmp_bytes, const uint32_t* in, uint32_t* out, int n, cudaStream_t s) {
    return cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, in, out, n, s);
}

size_t scan_u32x4_temp(int n) {
    size_t a = 0;
    cub::DeviceScan::ExclusiveScan(nullptr, a, (const uint4*)nullptr, (uint4*)nullptr, Add4(), make_uint4(0, 0, 0, 0),
                                   n);
    return a;
}

cudaError_t scan_u32x4(void* tmp, size_t tmp_bytes, const uint4* in, uint4* out, int n, cudaStream_t s) {
    return cub::DeviceScan::ExclusiveScan(tmp, tmp_bytes, in, out, Add4(), make_uint4(0, 0, 0, 0), n, s);
}

}  // namespace fmmx
