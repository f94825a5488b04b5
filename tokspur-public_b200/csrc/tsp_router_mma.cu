// Router projection for batches on the 5th-generation tensor cores (tcgen05) at FP32 precision:
//   logits[t][e] = sum_c W[e][c] * x[t][c],  W and x FP32.
//
// Each FP32 value is the exact sum of three bfloat16 values (h = the value rounded to nearest, m = the rest rounded to nearest, l = what is
// left: 8 + 8 + 8 significant bits and their signs), and a product is taken as six of its nine partial products:
// hh + (hm + mh + mm + hl + lh). |m| <= 2^-8 |v| and |l| <= 2^-17 |v|, so what is left out, ml + lm + ll, stays within 2^-24 of the product
// (2^-28 on average) and has either sign. (Parts cut off instead of rounded leave out up to 2^-21, always towards zero.) Values below
// 2^-109 lose low bits: the last part ends where bfloat16 does, at 2^-133. Products of bfloat16 values are exact in FP32. The tensor core adds into FP32 with truncation,
// which over 2048 columns would cost more than the FP32 chain it replaces (128 truncated additions); so the hh sums run over 256
// columns at most, in one of two accumulators that the epilogue warps empty into FP32 registers (rounded to nearest) while the other
// fills. The five small products, 2^-8 of the result, share one accumulator for the whole K extent.
//
// What bounds it: shared memory and the conversion. A (128 token rows) is therefore staged in tensor memory: 16x256b stores take the
// values as coalesced 16-byte loads leave them in the lanes; only B (64 matrix rows) passes through shared memory, which the six
// products of a K step read six times (48 KB per 64 columns at 128 bytes a cycle; with A there too it would be 144 KB).
//
// Measured with 512 matrix rows of 2048 columns (the FP32 FMA kernels before: 64-255 token rows 248 us, 256-1024 rows 154 us, 2048 rows
// 283 us): 33 us up to 1024 rows, 39 us at 2048, and the error against 64-bit sums falls from 8.1e-7 to 2.4e-7 (relative, 2-norm;
// 3.4e-7 with parts cut off).
// Loading two chunks ahead instead of one changed nothing (43 us at 2048 rows): the six products set the pace.
//
// Warps: 0..2 convert B, 3 issues the MMAs, 4..7 and 8..11 convert A (even and odd K chunks), 12..15 epilogue.
#include "tsp_common.cuh"

namespace tsp {

constexpr uint32_t kRmM = 128, kRmN = 64, kRmK = 64;   // tile: token rows, matrix rows, columns per stage
constexpr uint32_t kRmStages = 3, kRmBlock = 4;         // stages in flight; chunks per hh accumulation (256 columns)
constexpr uint32_t kRmThreads = 16 * 32;
constexpr uint32_t kRmPlane = kRmN * 128;               // bytes of one bfloat16 plane of a B chunk
constexpr uint32_t kRmSmem = 1024 + kRmStages * 3 * kRmPlane + 1024;
// tensor memory: hh accumulators [0, 64) and [64, 128), small products [128, 192), A stages of three planes of 32 columns from 192
constexpr uint32_t kRmSmall = 2 * kRmN, kRmA = 3 * kRmN;
static_assert(kRmA + kRmStages * 96 <= 512, "tensor memory");

// two FP32 values -> their three bfloat16 parts as packed pairs (`a` in the low half)
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    // the largest bfloat16 in the place of an infinity: a finite value above it keeps its rest, an infinity leaves one in `m`
    asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(b), "f"(a));
    const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xffff0000u);    // exact
    m = bf16_pair(ra, rb);
    l = bf16_pair(ra - __uint_as_float(m << 16), rb - __uint_as_float(m & 0xffff0000u));         // exact, at most 8 bits left
}

// 16 lanes x 16 columns: thread t holds columns 8 s + 2 (t % 4), + 1 of lanes t / 4 (r[4 s], r[4 s + 1]) and t / 4 + 8 (r[4 s + 2], r[4 s + 3])
__device__ __forceinline__ void tmem_st_16x256_x2(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void rm_tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
// four K steps of 16: D (+)= A[tensor memory] * B[shared memory], bfloat16
__device__ __forceinline__ void rm_mma4(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t accumulate) {
    constexpr uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);   // descriptor: 1024 bytes per eight rows, version 1, 128-byte swizzle
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kRmN >> 3) << 17) | ((kRmM >> 4) << 24);   // FP32 += bf16 x bf16
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
        asm volatile("{\n\t.reg .pred q;\n\t.reg .b64 b;\n\tsetp.ne.b32 q, %4, 0;\n\tmov.b64 b, {%2, %5};\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, q;\n\t}"
                     ::"r"(d), "r"(a + k * 8), "r"(b_lo + k * 2), "r"(idesc), "r"(accumulate | k), "n"(hi) : "memory");
}
__device__ __forceinline__ void rm_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool rm_wait(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, 1u << 21)); }

// four columns k .. k + 3 of a row, zeros past its end; V: rows are whole 16-byte units
template <bool V>
__device__ __forceinline__ float4 rm_load4(const float* row, uint32_t k, uint32_t cols) {
    if (V) return k < cols ? *reinterpret_cast<const float4*>(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(k < cols ? row[k] : 0.f, k + 1 < cols ? row[k + 1] : 0.f, k + 2 < cols ? row[k + 2] : 0.f, k + 3 < cols ? row[k + 3] : 0.f);
}

template <bool V>
__global__ void __launch_bounds__(kRmThreads, 1)
router_mma_kernel(const float* w, uint32_t rows, uint32_t cols, const float* extra, const float* x, uint64_t x_stride, uint32_t tokens, float* __restrict__ out,
                  uint64_t out_stride, float* __restrict__ extra_out, uint32_t* error) {
    pdl_launch_dependents();
    // The extra row (the shared expert's gate, one dot product per token): the blocks past the matrix's columns of blocks, a warp per token in turn,
    // with the sums of gemv_f32_kernel. A launch of its own behind this one took 6 to 8 us; one wave of this launch leaves SMs idle.
    if (blockIdx.x * kRmN >= rows) {
        pdl_wait();
        const uint32_t end = min(tokens, (blockIdx.y + 1) * kRmM);
        for (uint32_t t = blockIdx.y * kRmM + (threadIdx.x >> 5); t < end; t += kRmThreads / 32) {
            const float acc = f32_dot_row(extra, reinterpret_cast<const float*>(reinterpret_cast<const char*>(x) + static_cast<uint64_t>(t) * x_stride), cols, threadIdx.x & 31u);
            if ((threadIdx.x & 31u) == 0) {
                if (!finite_f32(acc)) raise_error(error, TSP_ERR_NONFINITE);
                extra_out[t] = acc;
            }
        }
        return;
    }
    extern __shared__ uint8_t rm_raw[];
    uint8_t* sm = rm_raw + ((1024u - (smem_u32(rm_raw) & 1023u)) & 1023u);
    uint64_t *full = reinterpret_cast<uint64_t*>(sm), *empty = full + kRmStages, *main_full = empty + kRmStages, *main_empty = main_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + 512);
    uint8_t* const bst = sm + 1024;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kRmStages; ++s) { mbar_init(&full[s], 3 + 4); mbar_init(&empty[s], 1); }
        for (uint32_t s = 0; s < 2; ++s) { mbar_init(&main_full[s], 1); mbar_init(&main_empty[s], 4); }
        mbar_fence_init();
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    pdl_wait();   // everything above touched shared and tensor memory only

    const uint32_t t0 = blockIdx.y * kRmM, r0 = blockIdx.x * kRmN;
    const uint32_t chunks = (cols + kRmK - 1) / kRmK, blocks = (chunks + kRmBlock - 1) / kRmBlock;
    bool ok = true;
    if (warp < 3) {
        // =========================== B: 64 matrix rows, 16 bytes per lane, sixteen lanes per row ===========================
        constexpr uint32_t NR = (kRmN / 2 + 2) / 3;   // a warp takes every third pair of rows
        const uint32_t k4 = lane & 15u, rr = 2 * warp + (lane >> 4);   // rows rr, rr + 6, ...
        float4 v[NR];
        auto fetch = [&](uint32_t c) {
#pragma unroll
            for (uint32_t i = 0; i < NR; ++i)
                v[i] = rm_load4<V>(w + static_cast<uint64_t>(min(r0 + min(rr + 6 * i, kRmN - 1), rows - 1)) * cols, c * kRmK + k4 * 4, cols);
        };
        fetch(0);
        uint32_t st = 0, ph = 0;
        for (uint32_t c = 0; c < chunks; ++c) {
            ok = rm_wait(&empty[st], ph ^ 1u);
            if (!ok) break;
            uint8_t* base = bst + st * 3 * kRmPlane + (k4 & 1u) * 8u;
#pragma unroll
            for (uint32_t i = 0; i < NR; ++i) {
                const uint32_t row = rr + 6 * i;
                if (row >= kRmN) break;
                uint2 h, m, l;
                split3(v[i].x, v[i].y, h.x, m.x, l.x); split3(v[i].z, v[i].w, h.y, m.y, l.y);
                uint8_t* d = base + row * 128u + (((k4 >> 1) ^ (row & 7u)) << 4);   // 128-byte swizzle
                *reinterpret_cast<uint2*>(d) = h; *reinterpret_cast<uint2*>(d + kRmPlane) = m; *reinterpret_cast<uint2*>(d + 2 * kRmPlane) = l;
            }
            if (c + 1 < chunks) fetch(c + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[st]);
            if (++st == kRmStages) { st = 0; ph ^= 1u; }
        }
    } else if (warp >= 4 && warp < 12) {
        // =========================== A: 128 token rows, a warp 32 of them, four lanes (64 bytes) per row ===========================
        const uint32_t group = (warp - 4) >> 2, quarter = warp & 3u;
        const float* src[4];   // rows lane / 4 + 8 i of the warp's quarter
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)
            src[i] = reinterpret_cast<const float*>(reinterpret_cast<const char*>(x) + static_cast<uint64_t>(min(t0 + quarter * 32u + (lane >> 2) + 8 * i, tokens - 1)) * x_stride);
        float4 v[8];   // half a warp's rows: [row / row + 8][four K steps of 16]
        auto fetch = [&](uint32_t c, uint32_t h) {
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) v[i] = rm_load4<V>(src[2 * h + (i >> 2)], c * kRmK + (i & 3u) * 16 + (lane & 3u) * 4, cols);
        };
        if (group < chunks) fetch(group, 0);
        for (uint32_t c = group; c < chunks; c += 2) {
            const uint32_t st = c % kRmStages, ph = (c / kRmStages) & 1u;
            ok = rm_wait(&empty[st], ph ^ 1u);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (uint32_t h2 = 0; h2 < 2; ++h2) {
                const uint32_t dst = tmem + ((quarter * 32u + h2 * 16u) << 16) + kRmA + st * 96u;
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {   // two K steps of 16
                    uint32_t h[8], m[8], l[8];
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {   // (K step, row / row + 8)
                        const float4 f = v[(i >> 1) + 2 * q + 4 * (i & 1u)];
                        split3(f.x, f.y, h[2 * i], m[2 * i], l[2 * i]);
                        split3(f.z, f.w, h[2 * i + 1], m[2 * i + 1], l[2 * i + 1]);
                    }
                    tmem_st_16x256_x2(dst + q * 16, h); tmem_st_16x256_x2(dst + 32 + q * 16, m); tmem_st_16x256_x2(dst + 64 + q * 16, l);
                }
                if (h2 == 0) fetch(c, 1);
                else if (c + 2 < chunks) fetch(c + 2, 0);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[st]);
        }
    } else if (warp == 3) {
        // =========================== MMA issuer ===========================
        const uint32_t b0 = ((smem_u32(bst) & 0x3FFFFu) >> 4) | (1u << 16);
        uint32_t st = 0, ph = 0;
        for (uint32_t c = 0; c < chunks; ++c) {
            const uint32_t blk = c / kRmBlock, buf = blk & 1u;
            if (c % kRmBlock == 0) {   // the epilogue has emptied this accumulator (used two blocks ago)
                ok = rm_wait(&main_empty[buf], ((blk >> 1) & 1u) ^ 1u);
                if (!ok) break;
            }
            ok = rm_wait(&full[st], ph);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint32_t a = tmem + kRmA + st * 96u, b = b0 + st * (3 * kRmPlane >> 4), bm = b + (kRmPlane >> 4), bl = b + (2 * kRmPlane >> 4);
                rm_mma4(tmem + buf * kRmN, a, b, c % kRmBlock);
                rm_mma4(tmem + kRmSmall, a, bm, c);
                rm_mma4(tmem + kRmSmall, a + 32, b, 1);
                rm_mma4(tmem + kRmSmall, a + 32, bm, 1);
                rm_mma4(tmem + kRmSmall, a, bl, 1);
                rm_mma4(tmem + kRmSmall, a + 64, b, 1);
                rm_commit(&empty[st]);
                if (c % kRmBlock == kRmBlock - 1 || c + 1 == chunks) rm_commit(&main_full[buf]);
            }
            __syncwarp();
            if (++st == kRmStages) { st = 0; ph ^= 1u; }
        }
    } else {
        // =========================== epilogue: a thread owns a token row ===========================
        const uint32_t quarter = warp & 3u, t = t0 + quarter * 32u + lane;
        const uint32_t lane_base = tmem + ((quarter * 32u) << 16);
        float acc[kRmN];
#pragma unroll
        for (uint32_t j = 0; j < kRmN; ++j) acc[j] = 0.f;
        auto add = [&](uint32_t col) {
#pragma unroll
            for (uint32_t h = 0; h < kRmN / 16; ++h) {
                uint32_t v[16];
                rm_tmem_ld16(lane_base + col + h * 16, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) acc[h * 16 + j] += __uint_as_float(v[j]);
            }
        };
        for (uint32_t blk = 0; blk < blocks; ++blk) {
            const uint32_t buf = blk & 1u;
            ok = rm_wait(&main_full[buf], (blk >> 1) & 1u);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            add(buf * kRmN);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&main_empty[buf]);
        }
        if (ok) {
            add(kRmSmall);   // the last block's commit covers every MMA before it
            bool bad = false;
            if (t < tokens) {
                float* orow = reinterpret_cast<float*>(reinterpret_cast<char*>(out) + static_cast<uint64_t>(t) * out_stride) + r0;
                const bool vec = (reinterpret_cast<uintptr_t>(orow) & 15u) == 0;
#pragma unroll
                for (uint32_t j = 0; j < kRmN; j += 4) {
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) bad |= r0 + j + i < rows && !finite_f32(acc[j + i]);
                    if (vec && r0 + j + 4 <= rows) *reinterpret_cast<float4*>(orow + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                    else {
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) if (r0 + j + i < rows) orow[j + i] = acc[j + i];
                    }
                }
            }
            if (bad) raise_error(error, TSP_ERR_NONFINITE);
        }
    }
    if (!ok && lane == 0) raise_error(error, TSP_ERR_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 3) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

template <bool V>
static int launch_router_mma_t(const float* w, uint32_t rows, uint32_t cols, const float* extra, const float* x, uint64_t x_stride, uint32_t tokens, float* out,
                               uint64_t out_stride, float* extra_out, uint32_t* error, cudaStream_t st) {
    static thread_local SmemAttrCache configured;   // per kernel instantiation, keyed by device
    TSP_CUDA(ensure_dynamic_smem(router_mma_kernel<V>, configured, kRmSmem));
    const dim3 grid((rows + kRmN - 1) / kRmN + (extra ? 1u : 0u), (tokens + kRmM - 1) / kRmM);
    TSP_CUDA(launch_pdl(router_mma_kernel<V>, grid, dim3(kRmThreads), kRmSmem, st, w, rows, cols, extra, x, x_stride, tokens, out, out_stride, extra_out, error));
    return TSP_OK;
}

int launch_router_mma(const float* w, uint32_t rows, uint32_t cols, const float* extra, const float* x, uint64_t x_stride, uint32_t tokens, float* out,
                      uint64_t out_stride, float* extra_out, uint32_t* error, cudaStream_t st) {
    const bool v4 = cols % 4 == 0 && (reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(x) | x_stride) % 16 == 0;
    if (v4) return launch_router_mma_t<true>(w, rows, cols, extra, x, x_stride, tokens, out, out_stride, extra_out, error, st);
    return launch_router_mma_t<false>(w, rows, cols, extra, x, x_stride, tokens, out, out_stride, extra_out, error, st);
}

}  // namespace tsp
