// Input rows of the grouped GEMMs in K order, as a block of a launch.
#pragma once

#include "tsp_common.cuh"

namespace tsp {

// Rows (FP32 or binary16) -> binary16 rows with the K order 0,2,1,3,4,6,5,7 inside each run of 8: the B operand of the
// gate-up GEMM, fetched from here by token id. 64 threads per row, four rows per block of 256 threads.
template <bool IN16>
__device__ __forceinline__ void rows_f16k_block(const void* x, uint64_t x_stride, uint32_t rows, uint32_t cols, __half* __restrict__ xk, uint64_t xk_stride,
                                                uint32_t* error, uint32_t block) {
    const uint32_t row = block * 4 + (threadIdx.x >> 6);
    if (row >= rows) return;
    const uint32_t t64 = threadIdx.x & 63;
    const char* src = reinterpret_cast<const char*>(x) + static_cast<uint64_t>(row) * x_stride;
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<char*>(xk) + static_cast<uint64_t>(row) * xk_stride);
    bool bad = false;
    for (uint32_t k8 = t64; k8 < cols / 8; k8 += 64) {
        uint32_t h[8];
        if (IN16) {
            const uint4 v = reinterpret_cast<const uint4*>(src)[k8];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                h[2 * i] = w[i] & 0xffffu; h[2 * i + 1] = w[i] >> 16;
                bad |= (w[i] & 0x7c00u) == 0x7c00u || (w[i] & 0x7c000000u) == 0x7c000000u;
            }
        } else {
            const float4 a = reinterpret_cast<const float4*>(src)[2 * k8], b = reinterpret_cast<const float4*>(src)[2 * k8 + 1];
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) { const __half hv = __float2half_rn(v[i]); bad |= !finite_f32(__half2float(hv)); h[i] = __half_as_ushort(hv); }
        }
        dst[k8] = make_uint4(h[0] | (h[2] << 16), h[1] | (h[3] << 16), h[4] | (h[6] << 16), h[5] | (h[7] << 16));
    }
    if (bad) raise_error(error, TSP_ERR_NONFINITE);
}

}  // namespace tsp
