// A dense Q8_0 matrix (or a gate / up pair with SwiGLU) times a few token rows, spread over many small blocks: the shared expert of a decode
// batch, as blocks of the launches that route the batch and build its tables (tsp_route.cu). Those launches leave most of the chip idle and
// the shared expert waits for neither.
//
// In launches of its own after the routed ones the shared expert ran on 8 (512 hidden units) and 16 (2048 channels) of 148 SMs, whole rows
// of K per SM, 128 matrix rows at a time: 24 and 12 us of a layer of 13 rows.
//
// A group of 16 MMA rows (8 gate + 8 up rows, or 16 plain rows) is shared by `sl` warps, each with runs of 256 columns (eight 34-byte blocks =
// 272 bytes a row): the run's bytes go to shared memory with 16-byte copies, all in flight at once, and the activations straight from global
// memory into the MMA's registers, as binary16 high and low halves (binary16 rows: as they are). Codes enter as exact binary16 integers,
// the block scale is applied to the FP32 sum of a block, sums of the warps meet in shared memory in the order of K.
#pragma once

#include "tsp_common.cuh"

namespace tsp {

constexpr uint32_t kQ8RunBytes = 272, kQ8RunCols = 256;
constexpr uint32_t kQ8WarpBytes = 16 * kQ8RunBytes;   // one run of a warp's 16 rows

struct Q8Rows {
    const uint8_t *a, *b;                 // GGUF rows; b: the up matrix (gate-up only)
    uint32_t rows, cols, row_bytes;
    const void* x; uint64_t x_stride;     // token rows, FP32 or binary16
    float* out; uint64_t out_stride;
    uint32_t tokens, sl, blocks;          // warps that share a group of rows; blocks of the launch that work on this matrix (0: none)
    uint32_t* error;
};
__host__ __device__ constexpr uint32_t q8_rows_smem(uint32_t warps) { return warps * (kQ8WarpBytes + 32u * 16u); }

// Eight codes starting at byte `p` (even, not a multiple of four: ODD_WORD) -> pairs (0,2), (1,3), (4,6), (5,7) as binary16 integers
template <bool ODD_WORD>
__device__ __forceinline__ void q8_rows_codes(const uint8_t* p, uint32_t (&out)[4]) {
    uint32_t c0, c1;
    if (ODD_WORD) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(p - 2);
        c0 = __funnelshift_r(w[0], w[1], 16); c1 = __funnelshift_r(w[1], w[2], 16);
    } else {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
        c0 = w[0]; c1 = w[1];
    }
    const __half2 k1152 = __float2half2_rn(1152.f);
    c0 ^= 0x80808080u; c1 ^= 0x80808080u;   // 0x6400 | (code + 128) = 1152 + code
    const uint32_t w[4] = {__byte_perm(c0, 0x64646464u, 0x4240), __byte_perm(c0, 0x64646464u, 0x4341),
                           __byte_perm(c1, 0x64646464u, 0x4240), __byte_perm(c1, 0x64646464u, 0x4341)};
#pragma unroll
    for (int i = 0; i < 4; ++i) { const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&w[i]), k1152); out[i] = *reinterpret_cast<const uint32_t*>(&v); }
}

// Block `block` of p.blocks, called by all threads of a block of WARPS warps (or more: the others only meet the barrier)
template <bool GATEUP, bool X16, uint32_t WARPS>
__device__ __forceinline__ void q8_rows_block(const Q8Rows& p, uint32_t block, uint8_t* smem) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    constexpr uint32_t RW = GATEUP ? 8u : 16u;
    const uint32_t per_block = WARPS / p.sl, row_blocks = (p.rows / RW + per_block - 1) / per_block;
    const uint32_t tile = block / row_blocks, group = (block - tile * row_blocks) * per_block + warp / p.sl, part = warp % p.sl;
    const uint32_t r0 = group * RW, token0 = tile * 8u, count = min(p.tokens - token0, 8u);
    const bool live = warp < WARPS && r0 < p.rows;   // whole warps
    uint8_t* const mine = smem + warp * kQ8WarpBytes;
    float4* const red = reinterpret_cast<float4*>(smem + WARPS * kQ8WarpBytes);
    float total[4] = {0.f, 0.f, 0.f, 0.f};
    if (live) {
        bool bad = false;
        const char* xrow = reinterpret_cast<const char*>(p.x) + static_cast<uint64_t>(token0 + min(g, count - 1u)) * p.x_stride;
        const bool row = g < count;
        for (uint32_t run = part; run < p.cols / kQ8RunCols; run += p.sl) {
            for (uint32_t i = lane; i < 16u * 17u; i += 32) {
                const uint32_t r = i / 17u, c = i - r * 17u;
                const uint8_t* src = (GATEUP && r >= 8 ? p.b + static_cast<uint64_t>(r0 + r - 8u) * p.row_bytes : p.a + static_cast<uint64_t>(r0 + r) * p.row_bytes) +
                                     run * kQ8RunBytes + c * 16u;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(mine + r * kQ8RunBytes + c * 16u)), "l"(src) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            const uint32_t k0 = run * kQ8RunCols + t * 8u;
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                // this lane's activations of four blocks, on their way with the weights
                uint4 x0[4], x1[X16 ? 1 : 4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t k = k0 + (half * 4u + j) * 32u;
                    if (X16) x0[j] = *reinterpret_cast<const uint4*>(xrow + k * 2u);
                    else { x0[j] = *reinterpret_cast<const uint4*>(xrow + k * 4u); x1[X16 ? 0 : j] = *reinterpret_cast<const uint4*>(xrow + k * 4u + 16u); }
                }
                if (half == 0) {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    __syncwarp();
                }
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t blk = half * 4u + j;
                    const uint8_t* pa = mine + g * kQ8RunBytes + blk * 34u;
                    const uint8_t* pb = pa + 8u * kQ8RunBytes;
                    uint32_t A[4], B[4], xh[4], xl[4];
                    if (blk & 1u) { q8_rows_codes<false>(pa + 2 + 8 * t, A); q8_rows_codes<false>(pb + 2 + 8 * t, B); }
                    else { q8_rows_codes<true>(pa + 2 + 8 * t, A); q8_rows_codes<true>(pb + 2 + 8 * t, B); }
                    if (X16) {
                        const uint32_t w[4] = {x0[j].x, x0[j].y, x0[j].z, x0[j].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) bad |= row && ((w[e] & 0x7c00u) == 0x7c00u || (w[e] & 0x7c000000u) == 0x7c000000u);
                        xh[0] = __byte_perm(w[0], w[1], 0x5410); xh[1] = __byte_perm(w[0], w[1], 0x7632);
                        xh[2] = __byte_perm(w[2], w[3], 0x5410); xh[3] = __byte_perm(w[2], w[3], 0x7632);
                    } else {
                        const uint4 y = x1[X16 ? 0 : j];
                        const float v[8] = {__uint_as_float(x0[j].x), __uint_as_float(x0[j].z), __uint_as_float(x0[j].y), __uint_as_float(x0[j].w),
                                            __uint_as_float(y.x), __uint_as_float(y.z), __uint_as_float(y.y), __uint_as_float(y.w)};   // order 0,2,1,3
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
                            const float2 f = __half22float2(h);
                            bad |= row && (!finite_f32(f.x) || !finite_f32(f.y));   // binary16's range is this encoding's range of activations
                            const __half2 l = __floats2half2_rn(v[2 * e] - f.x, v[2 * e + 1] - f.y);
                            xh[e] = *reinterpret_cast<const uint32_t*>(&h); xl[e] = *reinterpret_cast<const uint32_t*>(&l);
                        }
                    }
                    float acc[4];
                    mma_f16_16816_zero(acc, A[0], B[0], A[1], B[1], xh[0], xh[1]);
                    mma_f16_16816(acc, A[2], B[2], A[3], B[3], xh[2], xh[3]);
                    if (!X16) {
                        mma_f16_16816(acc, A[0], B[0], A[1], B[1], xl[0], xl[1]);
                        mma_f16_16816(acc, A[2], B[2], A[3], B[3], xl[2], xl[3]);
                    }
                    const float fA = half_bits_to_float(*reinterpret_cast<const uint16_t*>(pa)), fB = half_bits_to_float(*reinterpret_cast<const uint16_t*>(pb));
                    total[0] = fmaf(fA, acc[0], total[0]); total[1] = fmaf(fA, acc[1], total[1]);
                    total[2] = fmaf(fB, acc[2], total[2]); total[3] = fmaf(fB, acc[3], total[3]);
                }
            }
            __syncwarp();   // the run's bytes are read before the next run's land
        }
        if (bad) raise_error(p.error, TSP_ERR_NONFINITE);
        if (part) red[warp * 32u + lane] = make_float4(total[0], total[1], total[2], total[3]);
    }
    __syncthreads();
    if (!live || part) return;
    for (uint32_t k = 1; k < p.sl; ++k) {
        const float4 v = red[(warp + k) * 32u + lane];
        total[0] += v.x; total[1] += v.y; total[2] += v.z; total[3] += v.w;
    }
    bool bad = false;
#pragma unroll
    for (uint32_t q = 0; q < 2; ++q) {   // token rows 2t, 2t + 1
        const uint32_t j = 2 * t + q;
        if (j >= count) continue;
        float* o = reinterpret_cast<float*>(reinterpret_cast<char*>(p.out) + static_cast<uint64_t>(token0 + j) * p.out_stride) + r0 + g;
        if (GATEUP) {
            const float v = stable_silu(total[q]) * total[2 + q];
            bad |= !finite_f32(v);
            *o = v;
        } else {
            bad |= !finite_f32(total[q]) | !finite_f32(total[2 + q]);
            o[0] = total[q]; o[8] = total[2 + q];
        }
    }
    if (bad) raise_error(p.error, TSP_ERR_NONFINITE);
}

// The shared expert of a decode batch as the layer hands it to the prologue: GGUF Q8_0 matrices, hidden rows of hidden * 4 bytes, output rows of
// channels * 4 bytes; `up`, `down` and `done` are the prologue's.
struct DecodeDense {
    const uint8_t *gate_w, *up_w, *down_w;
    uint32_t hidden, channels;
    const void* x; uint64_t x_stride;
    float *h, *out;
    uint32_t* error;
    bool x16 = false, done = false;
    Q8Rows up{}, down{};
};

// Geometry for blocks of `warps` warps: as many warps per group of rows as K has runs, a power of two
static inline void q8_rows_plan(Q8Rows& p, bool gate_up, uint32_t warps) {
    const uint32_t runs = p.cols / kQ8RunCols;
    for (p.sl = 1; p.sl * 2 <= runs && p.sl * 2 <= (warps < 8 ? warps : 8u);) p.sl *= 2;
    const uint32_t groups = p.rows / (gate_up ? 8u : 16u), per_block = warps / p.sl;
    p.blocks = (groups + per_block - 1) / per_block * ((p.tokens + 7u) / 8u);
}

}  // namespace tsp
