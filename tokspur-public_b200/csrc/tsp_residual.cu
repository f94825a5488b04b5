// Hyper-connection residual read / write: the step either side of the MoE FFN sub-layer in every layer
// (MetalGraph::residual_read / residual_write, native/include/tokspur/graph.hpp:1056-1058; CPU forms operators.cpp:60-96).
// Element-wise FP32 work over [tokens][branches][channels] rows: bound by HBM bandwidth, one pass each.
#include <initializer_list>

#include "tsp_common.cuh"

namespace tsp {

// V channels per thread (4: one 16-byte load per branch and tensor, all of a thread's loads issued before the first use; 1: rows that
// are not whole 16-byte units). 2048 rows of 4 x 2048 channels, rows of the call before still in L2: read 55 -> 25 us, write 30 -> 21 us
// against one 4-byte load after another.
template <uint32_t V> struct Chan;
template <> struct Chan<4> { using T = float4; };
template <> struct Chan<1> { using T = float; };
__device__ __forceinline__ float& chan_at(float4& v, uint32_t i) { return reinterpret_cast<float*>(&v)[i]; }
__device__ __forceinline__ float& chan_at(float& v, uint32_t) { return v; }

constexpr uint32_t kResThreads = 128;
constexpr uint32_t kResBranches = 4;   // branches in flight per thread

// stable_sigmoid without its branch: one exponential of -|v|, one division; the same operations on the same operands
__device__ __forceinline__ float sigmoid_one_exp(float v) {
    const float e = expf(-fabsf(v));
    return (v >= 0.f ? 1.f : e) / (1.f + e);
}

// out[t][c] = sum_b normalized[t][b][c] * sigmoid(scores[t][b][c]) / branches      (branch order ascending, as the reference adds them)
// scales[t][b] = 2 * sigmoid(inject_logits[t][b] / branches)
template <uint32_t V>
__global__ void __launch_bounds__(kResThreads)
residual_read_kernel(const float* normalized, const float* scores, const float* inject_logits,
                     uint32_t branches, uint32_t channels, float* __restrict__ output, float* __restrict__ scales, uint32_t* error) {
    using T = typename Chan<V>::T;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t t = blockIdx.y, units = channels / V;
    const uint64_t row = static_cast<uint64_t>(t) * branches * units;
    const T* nrm = reinterpret_cast<const T*>(normalized);
    const T* scr = reinterpret_cast<const T*>(scores);
    const float inv = 1.f / static_cast<float>(branches);
    bool bad = false;
    for (uint32_t u = blockIdx.x * kResThreads + threadIdx.x; u < units; u += gridDim.x * kResThreads) {
        float acc[V];
#pragma unroll
        for (uint32_t i = 0; i < V; ++i) acc[i] = 0.f;
        for (uint32_t b0 = 0; b0 < branches; b0 += kResBranches) {
            T n[kResBranches], g[kResBranches];
#pragma unroll
            for (uint32_t b = 0; b < kResBranches; ++b) {
                const uint64_t at = row + static_cast<uint64_t>(min(b0 + b, branches - 1)) * units + u;
                n[b] = nrm[at]; g[b] = scr[at];
            }
#pragma unroll
            for (uint32_t b = 0; b < kResBranches; ++b)
                if (b0 + b < branches)
#pragma unroll
                    for (uint32_t i = 0; i < V; ++i) acc[i] += chan_at(n[b], i) * sigmoid_one_exp(chan_at(g[b], i)) * inv;
        }
        T o;
#pragma unroll
        for (uint32_t i = 0; i < V; ++i) { bad |= !finite_f32(acc[i]); chan_at(o, i) = acc[i]; }
        reinterpret_cast<T*>(output)[static_cast<uint64_t>(t) * units + u] = o;
    }
    if (blockIdx.x == 0)
        for (uint32_t b = threadIdx.x; b < branches; b += kResThreads) {
            const float s = 2.f * stable_sigmoid(inject_logits[static_cast<uint64_t>(t) * branches + b] * inv);
            bad |= !finite_f32(s);
            scales[static_cast<uint64_t>(t) * branches + b] = s;
        }
    if (bad) raise_error(error, TSP_ERR_NONFINITE);
}

// destination[t][b][c] = streams[t][b][c] + scales[t][b] * output[t][c]      (destination may be streams: a thread writes what it read)
// A thread takes NB branches of one unit; blockIdx.x counts (run of units, group of branches).
template <uint32_t V, uint32_t NB>
__global__ void __launch_bounds__(V == 4 ? 128 : 256)
residual_write_kernel(const float* streams, const float* output, const float* scales, uint32_t branches,
                      uint32_t channels, float* destination, uint32_t* error) {
    using T = typename Chan<V>::T;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t t = blockIdx.y, units = channels / V, groups = (branches + NB - 1) / NB;
    const uint32_t run = blockIdx.x / groups, b0 = (blockIdx.x - run * groups) * NB, u = run * blockDim.x + threadIdx.x;
    if (u >= units) return;
    const uint64_t row = static_cast<uint64_t>(t) * branches * units;
    bool bad = false;
    T o = reinterpret_cast<const T*>(output)[static_cast<uint64_t>(t) * units + u];
    T s[NB];
    float f[NB];
#pragma unroll
    for (uint32_t b = 0; b < NB; ++b) {
        const uint32_t bb = min(b0 + b, branches - 1);
        s[b] = reinterpret_cast<const T*>(streams)[row + static_cast<uint64_t>(bb) * units + u];
        f[b] = scales[static_cast<uint64_t>(t) * branches + bb];
    }
#pragma unroll
    for (uint32_t b = 0; b < NB; ++b) {
        if (b0 + b >= branches) break;
        T v;
#pragma unroll
        for (uint32_t i = 0; i < V; ++i) { chan_at(v, i) = fmaf(f[b], chan_at(o, i), chan_at(s[b], i)); bad |= !finite_f32(chan_at(v, i)); }
        reinterpret_cast<T*>(destination)[row + static_cast<uint64_t>(b0 + b) * units + u] = v;
    }
    if (bad) raise_error(error, TSP_ERR_NONFINITE);
}

static bool whole_units(uint32_t channels, std::initializer_list<const void*> rows) {
    if (channels % 4) return false;
    for (const void* r : rows) if (!aligned16(r)) return false;
    return true;
}

int launch_residual_read(const float* normalized, const float* scores, const float* inject_logits, uint32_t branches, uint32_t channels,
                         uint32_t tokens, float* output, float* scales, uint32_t* error, cudaStream_t st) {
    const bool v4 = whole_units(channels, {normalized, scores, output});
    const uint32_t units = v4 ? channels / 4 : channels;
    const dim3 grid((units + kResThreads - 1) / kResThreads, tokens);
    TSP_CUDA(launch_pdl(v4 ? residual_read_kernel<4> : residual_read_kernel<1>, grid, dim3(kResThreads), 0, st, normalized, scores, inject_logits, branches,
                        channels, output, scales, error));
    return TSP_OK;
}

int launch_residual_write(const float* streams, const float* output, const float* scales, uint32_t branches, uint32_t channels, uint32_t tokens,
                          float* destination, uint32_t* error, cudaStream_t st) {
    const bool v4 = whole_units(channels, {streams, output, destination});
    const uint32_t threads = v4 ? 128 : 256, units = v4 ? channels / 4 : channels, runs = (units + threads - 1) / threads;
    // One branch per thread while that is about one wave of blocks: 64 rows of 4 x 2560 1.7 us against 2.0 with four branches per thread, 256
    // rows of 4 x 2048 4.8 us against 3.5. (Every branch in one thread: 64 rows of 16 x 4096 7.2 us, now 4.2; 2000 rows of 4 x 2050 43 us, now 27.)
    const bool single = static_cast<uint64_t>(runs) * branches * tokens <= 8u * 148u;
    const dim3 grid(runs * (single ? branches : (branches + 3) / 4), tokens);
    auto kernel = v4 ? (single ? residual_write_kernel<4, 1> : residual_write_kernel<4, 4>) : (single ? residual_write_kernel<1, 1> : residual_write_kernel<1, 4>);
    TSP_CUDA(launch_pdl(kernel, grid, dim3(threads), 0, st, streams, output, scales, branches, channels, destination, error));
    return TSP_OK;
}

}  // namespace tsp
