// Decode-size routed / dense projections over the five-bit encodings of the reference's model: Q5_K (176-byte super-blocks of
// 256 weights; gate and up tensors) and Q5_1 (24-byte blocks of 32 weights; down tensors), plain GGUF rows.
//
// Two kernels: tiles of up to eight token rows (every routed launch) take warp-level MMAs on the five-bit codes (gemv_k5_mma_kernel, below);
// dense batches of more rows and shapes that are not whole warps or too long take FP32 FMAs on exactly rounded weights:
//
// A block takes one token tile and a run of weight rows. It first stages the tile's FP32 activation rows in shared memory
// (32-value groups padded to 36 values, so that 32 lanes reading 16 bytes each at a group stride touch every bank equally). Then
// the lanes of a warp spread over the K extent of one weight row (gate-up: the gate row and the up row of one hidden unit): a
// lane takes one 32-weight group at a time with 16-byte loads that are contiguous across the warp, decodes it to the exactly
// rounded FP32 weights (numeric.cpp:38-50: d * sc * q and dmin * mn are exact in FP32, so one FMA gives the reference's rounded
// value), multiplies with the staged activations and keeps one FP32 sum per token; the lanes' sums are added with shuffles.
// Weight bytes are read once per (tile, row).
#include <cuda.h>

#include "tsp_common.cuh"

namespace tsp {

int get_tensor_map_bytes(const void* base, uint32_t rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box,
                         bool swizzle128, CUtensorMap* out);

constexpr uint32_t kK5MaxTokens = 16;   // token rows of a tile (8 per routed tile, 16 for dense row batches)
constexpr uint32_t kK5Threads = 256;    // eight warps
constexpr uint32_t kK5BlockRows = 64;   // weight rows (hidden units) per block and tile

struct K5Params {
    const uint8_t* a_base; const uint8_t* a_base_hi; const uint8_t* b_base; const uint8_t* b_base_hi;
    uint64_t expert_stride; uint32_t split, experts;
    uint32_t rows, cols, row_bytes;
    const float* x; uint64_t x_stride_bytes; uint32_t in_div;
    const uint32_t* token_map; const uint32_t* counts; const uint32_t* tasks;
    uint32_t tokens, tile_tokens;
    // MMA kernel
    uint32_t wpu;             // warps that share a unit, each with a part of its K extent (a power of two, no more than there are K steps)
    uint32_t slots;           // (unit, K part) sums of a batch that shared memory holds
    uint32_t copies, copy_lines, mat_bytes, stage_bytes, stages;   // a unit's matrix: copies of copy_lines lines, padded to mat_bytes; ring of stages
    uint32_t off_sx, off_red, off_stage;
    uint32_t lanes_per_row;   // lanes that share one weight row: the largest power of two <= min(32, groups)
    float* out; uint64_t out_stride_bytes;
    uint32_t* error;
    uint32_t staging;         // what staging the rows of a tile costs, in units
};

// byte k of `q` as a float: 0x4B0000bb is 2^23 + bb, the subtraction is exact (no integer-to-float conversion instruction)
template <uint32_t K>
__device__ __forceinline__ float byte_f32(uint32_t q) { return __uint_as_float(__byte_perm(q, 0x4b000000u, 0x7440u + K)) - 8388608.f; }

// One 32-weight group of a row, fetched with wide loads and then read four weights at a time: get(i4, w) gives weights
// 4 i4 .. 4 i4 + 3 of the group as the exactly rounded FP32 values.
template <uint32_t TYPE> struct Group5;
template <> struct Group5<13u> {   // Q5_K: header (d, dmin, twelve factor bytes), 32 bytes of fifth bits, 128 bytes of nibbles
    float s, m; uint32_t qs[8], qh[8]; uint32_t shift, g; bool finite;
    __device__ __forceinline__ Group5(const uint8_t* row, uint32_t grp) {
        const uint8_t* block = row + (grp >> 3) * 176u;
        g = grp & 7u;
        const uint4 h = *reinterpret_cast<const uint4*>(block);
        const uint4 h0 = reinterpret_cast<const uint4*>(block + 16)[0], h1 = reinterpret_cast<const uint4*>(block + 16)[1];
        const uint4 q0 = reinterpret_cast<const uint4*>(block + 48 + (g >> 1) * 32)[0], q1 = reinterpret_cast<const uint4*>(block + 48 + (g >> 1) * 32)[1];
        qh[0] = h0.x; qh[1] = h0.y; qh[2] = h0.z; qh[3] = h0.w; qh[4] = h1.x; qh[5] = h1.y; qh[6] = h1.z; qh[7] = h1.w;
        qs[0] = q0.x; qs[1] = q0.y; qs[2] = q0.z; qs[3] = q0.w; qs[4] = q1.x; qs[5] = q1.y; qs[6] = q1.z; qs[7] = q1.w;
        // factors of group g from the header words (y, z, w = the twelve packed bytes), numeric.cpp:25-31
        const uint32_t sh = 8u * (g & 3u);
        const uint32_t by = (h.y >> sh) & 255u, bz = (h.z >> sh) & 255u, bw = (h.w >> sh) & 255u;
        const uint32_t sc = g < 4 ? (by & 63u) : ((bw & 15u) | ((by >> 6) << 4));
        const uint32_t mn = g < 4 ? (bz & 63u) : ((bw >> 4) | ((bz >> 6) << 4));
        const float d = half_bits_to_float(h.x & 0xffffu), dmin = half_bits_to_float(h.x >> 16);
        s = d * static_cast<float>(sc); m = -(dmin * static_cast<float>(mn));   // both exact
        shift = 4u * (g & 1u);
        finite = finite_f32(d) && finite_f32(dmin);
    }
    __device__ __forceinline__ void get(uint32_t i4, float (&w)[4]) const {
        const uint32_t q = ((qs[i4] >> shift) & 0x0f0f0f0fu) | (((qh[i4] >> g) & 0x01010101u) << 4);
        w[0] = fmaf(s, byte_f32<0>(q), m); w[1] = fmaf(s, byte_f32<1>(q), m); w[2] = fmaf(s, byte_f32<2>(q), m); w[3] = fmaf(s, byte_f32<3>(q), m);
    }
};
template <> struct Group5<7u> {    // Q5_1: d, m, 32 fifth bits, 16 bytes of nibbles
    float d, m; uint32_t qh; uint32_t qs[4]; bool finite;
    __device__ __forceinline__ Group5(const uint8_t* row, uint32_t grp) {
        const uint2* block = reinterpret_cast<const uint2*>(row + grp * 24u);   // 24-byte blocks of 8-byte aligned rows: three 8-byte loads
        const uint2 h = block[0], q01 = block[1], q23 = block[2];
        d = half_bits_to_float(h.x & 0xffffu); m = half_bits_to_float(h.x >> 16);
        qh = h.y;
        qs[0] = q01.x; qs[1] = q01.y; qs[2] = q23.x; qs[3] = q23.y;
        finite = finite_f32(d) && finite_f32(m);
    }
    __device__ __forceinline__ void get(uint32_t i4, float (&w)[4]) const {
        // weight i: nibble (i / 16) of byte i % 16, fifth bit = bit i of qh
        const uint32_t hb = (qh >> (4u * i4)) & 15u;
        // the four fifth bits spread to bit 4 of each byte: bit k of hb -> bit 8 k + 4
        const uint32_t q = ((qs[i4 & 3u] >> (4u * (i4 >> 2))) & 0x0f0f0f0fu) | (((hb * 0x00204081u) & 0x01010101u) << 4);
        w[0] = fmaf(d, byte_f32<0>(q), m); w[1] = fmaf(d, byte_f32<1>(q), m); w[2] = fmaf(d, byte_f32<2>(q), m); w[3] = fmaf(d, byte_f32<3>(q), m);
    }
};

// The FP32 sums of one weight row (gate-up: gate and up row) per `lpr` lanes for `count` token rows: at(j, grp, i4) gives four activations,
// put(j, v) takes a finished output on the row's first lane. Whole warps; a lane of no live row computes along.
template <uint32_t TYPE, bool GATEUP, uint32_t MT, class At, class Put>
__device__ __forceinline__ bool k5_row_f32(const uint8_t* rowA, const uint8_t* rowB, uint32_t groups, uint32_t lpr, uint32_t lig, uint32_t count, At at, Put put) {
    bool ok = true;
    float accA[MT], accB[GATEUP ? MT : 1];
#pragma unroll
    for (uint32_t j = 0; j < MT; ++j) { accA[j] = 0.f; if (GATEUP) accB[j] = 0.f; }
    for (uint32_t grp = lig; grp < groups; grp += lpr) {
        const Group5<TYPE> ga(rowA, grp), gb(rowB, grp);
        ok &= ga.finite & gb.finite;
#pragma unroll
        for (uint32_t i4 = 0; i4 < 8; ++i4) {
            float wa[4], wb[4] = {0.f, 0.f, 0.f, 0.f};
            ga.get(i4, wa);
            if (GATEUP) gb.get(i4, wb);
#pragma unroll
            for (uint32_t j = 0; j < MT; ++j) {
                if (j >= count) break;
                const float4 v = at(j, grp, i4);
                accA[j] = fmaf(wa[0], v.x, accA[j]); accA[j] = fmaf(wa[1], v.y, accA[j]); accA[j] = fmaf(wa[2], v.z, accA[j]); accA[j] = fmaf(wa[3], v.w, accA[j]);
                if (GATEUP) { accB[j] = fmaf(wb[0], v.x, accB[j]); accB[j] = fmaf(wb[1], v.y, accB[j]); accB[j] = fmaf(wb[2], v.z, accB[j]); accB[j] = fmaf(wb[3], v.w, accB[j]); }
            }
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < MT; ++j) {
        if (j >= count) break;
        float a = accA[j], b = GATEUP ? accB[j] : 0.f;
        for (uint32_t o = lpr >> 1; o > 0; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); if (GATEUP) b += __shfl_xor_sync(0xffffffffu, b, o); }
        // silu with the branch-stable sigmoid (operators.cpp:28-36)
        if (lig == 0) put(j, GATEUP ? (a >= 0.f ? a / (1.f + expf(-a)) : a * expf(a) / (1.f + expf(a))) * b : a);
    }
    return ok;
}

// MT: token rows of a tile at most (8 for routed tiles, 16 for dense row batches of more than 8 rows).
// Shared memory: the tile's rows as [token][group][9 float4] (eight of data, one of padding).
template <uint32_t TYPE, bool GATEUP, uint32_t MT>
__global__ void __launch_bounds__(kK5Threads) gemv_k5_kernel(const K5Params p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float4 k5_xs[];
    __shared__ const float4* s_x[kK5MaxTokens];   // the tile's input rows
    __shared__ float* s_out[kK5MaxTokens];        // and its output rows
    __shared__ uint32_t s_tile[3];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t n_tiles = p.token_map ? p.tasks[0] : (p.tokens + p.tile_tokens - 1) / p.tile_tokens;
    const uint32_t groups = p.cols / 32u;
    const uint32_t lpr = p.lanes_per_row, rpw = 32u / lpr;    // lanes per row, rows per warp
    const uint32_t sub = lane / lpr, lig = lane & (lpr - 1u); // this lane's row of the warp's rows, its first group
    const uint32_t row0 = blockIdx.x * kK5BlockRows;
    for (uint32_t tile = blockIdx.y; tile < n_tiles; tile += gridDim.y) {   // uniform over the block
        __syncthreads();   // the previous tile's rows are no longer read
        if (threadIdx.x == 0) {
            uint32_t expert = 0, start = tile * p.tile_tokens, count = 0;
            if (p.token_map) {
                expert = p.tasks[2 + 2 * tile];
                start = p.tasks[3 + 2 * tile];
                if (expert < p.experts) { const uint32_t c = p.counts[expert]; count = c > start ? min(c - start, p.tile_tokens) : 0u; }
                else expert = 0;
            } else if (start < p.tokens) count = min(p.tokens - start, p.tile_tokens);
            s_tile[0] = expert; s_tile[1] = start; s_tile[2] = count;
        }
        __syncthreads();
        const uint32_t expert = s_tile[0], start = s_tile[1], count = min(s_tile[2], MT);
        if (count == 0) continue;   // uniform
        if (threadIdx.x < count) {
            const uint32_t rid = p.token_map ? p.token_map[static_cast<uint64_t>(expert) * p.tokens + start + threadIdx.x] : start + threadIdx.x;
            s_x[threadIdx.x] = reinterpret_cast<const float4*>(reinterpret_cast<const char*>(p.x) + static_cast<uint64_t>(rid / p.in_div) * p.x_stride_bytes);
            s_out[threadIdx.x] = reinterpret_cast<float*>(reinterpret_cast<char*>(p.out) + static_cast<uint64_t>(rid) * p.out_stride_bytes);
        }
        __syncthreads();
        // stage the activation rows: consecutive threads read consecutive 16-byte pieces of a row
        for (uint32_t i = threadIdx.x; i < count * groups * 8u; i += kK5Threads) {
            const uint32_t j = i / (groups * 8u), rem = i - j * groups * 8u;
            k5_xs[(j * groups + (rem >> 3)) * 9u + (rem & 7u)] = s_x[j][rem];
        }
        __syncthreads();
        const bool hi = expert >= p.split;
        const uint64_t eoff = static_cast<uint64_t>(hi ? expert - p.split : expert) * p.expert_stride;
        const uint8_t* baseA = (hi ? p.a_base_hi : p.a_base) + eoff;
        const uint8_t* baseB = GATEUP ? (hi ? p.b_base_hi : p.b_base) + eoff : baseA;
        bool ok = true;
        // the warps take the block's rows in turn, `rpw` rows at a time (uniform trip count over the warp: shuffles inside)
        for (uint32_t rb = row0 + warp * rpw; rb < row0 + kK5BlockRows && rb < p.rows; rb += (kK5Threads / 32u) * rpw) {
            const uint32_t r = rb + sub;
            const bool live = r < p.rows && r < row0 + kK5BlockRows;
            const uint8_t* rowA = baseA + static_cast<uint64_t>(live ? r : rb) * p.row_bytes;
            const uint8_t* rowB = baseB + static_cast<uint64_t>(live ? r : rb) * p.row_bytes;
            ok &= k5_row_f32<TYPE, GATEUP, MT>(
                rowA, rowB, groups, lpr, lig, count, [&](uint32_t j, uint32_t grp, uint32_t i4) { return k5_xs[(j * groups + grp) * 9u + i4]; },
                [&](uint32_t j, float v) {   // a non-finite activation makes the sums it enters non-finite (0 * inf is NaN)
                    if (!live) return;
                    if (!finite_f32(v)) raise_error(p.error, TSP_ERR_NONFINITE);
                    s_out[j][r] = v;
                });
        }
        if (!ok) raise_error(p.error, TSP_ERR_NONFINITE);
    }
}

// ---------------------------------------------------------------------------------------------
// The same projections on warp-level MMAs (m16n8k16, binary16 operands, FP32 accumulators) for tiles of up to 8 token rows.
//
// What bounded the kernel above: with one or two routes per expert it is all decoding (about five instructions a weight) between
// dependent load latencies. Here the five-bit codes enter the MMA as binary16 integers code - 16 (three or four operations per pair),
// the group's scale s and offset 16 s + m are applied to FP32 sums, the offset through the group's FP32 activation sum. Centred codes
// keep both terms as small as the weights themselves; with codes 0..31 a weight near zero is the difference of two large terms.
// Activations enter as binary16 high + low halves after a power-of-two scaling of the row's largest to [2^14, 2^15): the pair keeps 22 bits of
// every value, down to 2^-25 after scaling (2^-39 of the row's largest), for rows anywhere in FP32's range.
// One block per SM: sixteen consumer warps and a producer warp. Work is counted in units of 8 hidden units (8 gate + 8 up rows) or 16 plain rows of
// one tile; a block takes a contiguous run of them, so that it stages a tile's rows once for all of its units there. A unit's bytes are one
// contiguous run per matrix: one tensor copy each, as 128-byte lines under the 128-byte swizzle (row strides of 1408 or 384 bytes would put
// eight rows on the same banks), several units ahead. `wpu` warps share a unit, each a part of the K extent (one step of it in most shapes), and
// a batch of units is added up behind a barrier.
// What bounded the kernel before, when each warp loaded whole rows into registers: the L1 data pipe (58 % of its cycles for gate-up, 70 % for down:
// every load touched eight lines), the integer pipe, warps with a fourth unit where 3.1 were their share. Whole layer of 512 experts of
// 512 x 2048, ten per token: 13 rows 190 -> 153 us, 64 rows 498 -> 370 us. Now: issue on 65 % of the cycles, the integer pipe busy on 53 %.
// The groups of a step are summed by themselves before they join the total: one chain over K of 2048 was further from 64-bit sums
// (2.1e-7, relative 2-norm) than the FP32 kernel (1.5e-7).
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kKmWarps = 16, kKmThreads = (kKmWarps + 4) * 32;   // consumer warps; + the producer's warpgroup (one warp of it works)
// Registers after the hand-over between the warpgroups (setmaxnreg): the consumers' request waits for what the producers give back, so
// kKmWarps * (kKmConsRegs - launch) <= 4 * (launch - kKmProdRegs) must hold for the count at launch (96). launch_km() checks the compiled kernel.
constexpr int kKmConsRegs = 112, kKmProdRegs = 24;
constexpr uint32_t kKmParts = 8;       // warps that share a unit at most
constexpr uint32_t kKmStages = 16;     // units in flight at most
constexpr uint32_t kKmTable = 32;      // tiles whose routing data a block keeps in shared memory
struct alignas(64) K5Maps { CUtensorMap m[4]; };   // matrix A low ids, high ids, matrix B the same: [128 B][line][expert]

// 16 rows x 32 columns of codes (two K steps of 16) against 8 token rows: acc = (codes - 16) x scaled activations
__device__ __forceinline__ void k5_group_mma(float (&acc)[4], const uint32_t (&a)[4], const uint32_t (&b)[4], const uint8_t* x) {
    const uint4 v = *reinterpret_cast<const uint4*>(x);
    mma_f16_16816_zero(acc, a[0], b[0], a[1], b[1], v.x, v.y);
    mma_f16_16816(acc, a[2], b[2], a[3], b[3], v.z, v.w);
}
// four code bytes in the low five bits of each byte of `c` -> two pairs of binary16 integers code - 16 (bytes 0, 2 and bytes 1, 3). The kernel is
// bound by the integer pipe (two cycles an instruction): bytes widen to 0x64bb = 1024 + code with one permutation per pair, where masks and shifts
// took 46 integer instructions per group of 32 columns and 16 rows; the subtraction on the FMA pipe is exact.
__device__ __forceinline__ void k5_codes(uint32_t c, uint32_t& even, uint32_t& odd) {
    const uint32_t e = __byte_perm(c, 0x64646464u, 0x4240), o = __byte_perm(c, 0x64646464u, 0x4341);
    const __half2 k1040 = __float2half2_rn(1040.f);
    const __half2 he = __hsub2(*reinterpret_cast<const __half2*>(&e), k1040), ho = __hsub2(*reinterpret_cast<const __half2*>(&o), k1040);
    even = *reinterpret_cast<const uint32_t*>(&he); odd = *reinterpret_cast<const uint32_t*>(&ho);
}

// byte `lin` of a run of lines that a copy with the 128-byte swizzle laid down at a multiple of 1024
__device__ __forceinline__ uint32_t km_swizzle(uint32_t lin) { return lin ^ (((lin >> 7) & 7u) << 4); }

template <uint32_t I> struct KmIndex { static constexpr uint32_t value = I; };
// Codes - 16, scale (an exact product) and offset 16 scale + m (one rounding; RAW: m alone) of the groups of a step, for this lane's row. get<G>() is
// called by whole warps.
template <uint32_t TYPE> struct KmStep;
// Q5_K: a step is one 256-weight super-block of a row. Lane t of the four that share the row works out groups 2t and 2t + 1; the others read them
// by shuffles (the kernel is bound by the integer pipe, where byte-to-float steps and factor unpacking would be repeated four times).
template <> struct KmStep<13u> {
    static constexpr uint32_t kGroups = 8, kBytes = 176;
    static constexpr uint32_t kLoads = 6;
    __device__ __forceinline__ static void offsets(uint32_t lin, uint32_t t, uint32_t (&at)[kLoads]) {   // lin: the step's first byte in the unit's matrix
        at[0] = km_swizzle(lin); at[1] = km_swizzle(lin + 16 + t * 8);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) at[2 + j] = km_swizzle(lin + 48 + j * 32 + t * 8);
    }
    uint4 hd; uint2 qh, qs[4];
    __device__ __forceinline__ void load(const uint8_t* m, const uint32_t (&at)[kLoads]) {
        hd = *reinterpret_cast<const uint4*>(m + at[0]);
        qh = *reinterpret_cast<const uint2*>(m + at[1]);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) qs[j] = *reinterpret_cast<const uint2*>(m + at[2 + j]);
    }
    float f[2], m[2]; uint2 qh4;
    template <bool RAW = false> __device__ __forceinline__ bool header(uint32_t t) {
        // 6-bit factors 2t, 2t + 1 of the scales and minima (numeric.cpp:25-31) in bytes 0 and 1
        const uint32_t sh = 16u * (t & 1u), y = hd.y >> sh, z = hd.z >> sh, w = hd.w >> sh;
        const uint32_t sc = t < 2 ? y & 0x3f3fu : (w & 0x0f0fu) | ((y >> 2) & 0x3030u), mn = t < 2 ? z & 0x3f3fu : ((w >> 4) & 0x0f0fu) | ((z >> 2) & 0x3030u);
        const float d = half_bits_to_float(hd.x & 0xffffu), dmin = half_bits_to_float(hd.x >> 16);
        f[0] = d * byte_f32<0>(sc); f[1] = d * byte_f32<1>(sc);
        const float m0 = -(dmin * byte_f32<0>(mn)), m1 = -(dmin * byte_f32<1>(mn));   // exact
        m[0] = RAW ? m0 : fmaf(16.f, f[0], m0); m[1] = RAW ? m1 : fmaf(16.f, f[1], m1);
        qh4 = make_uint2(qh.x >> 4, qh.y >> 4);
        return finite_f32(d) && finite_f32(dmin);
    }
    template <uint32_t G, bool RAW = false> __device__ __forceinline__ void get(uint32_t, uint32_t (&a)[4], float& fg, float& mg) const {
        constexpr uint32_t J = G >> 1, HI = G & 1u;
        const uint2 h = G < 4 ? qh : qh4;
        constexpr uint32_t M = 0x01010101u << (G & 3u), S = 16u >> (G & 3u);
        k5_codes(((HI ? qs[J].x >> 4 : qs[J].x) & 0x0f0f0f0fu) | ((h.x & M) * S), a[0], a[1]);
        k5_codes(((HI ? qs[J].y >> 4 : qs[J].y) & 0x0f0f0f0fu) | ((h.y & M) * S), a[2], a[3]);
        fg = __shfl_sync(0xffffffffu, f[HI], J, 4);
        mg = __shfl_sync(0xffffffffu, m[HI], J, 4);
    }
};
// Q5_1: a step is four 32-weight blocks of a row
template <> struct KmStep<7u> {
    static constexpr uint32_t kGroups = 4, kBytes = 96;
    static constexpr uint32_t kLoads = 8;
    __device__ __forceinline__ static void offsets(uint32_t lin, uint32_t t, uint32_t (&at)[kLoads]) {
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) { at[j] = km_swizzle(lin + 24 * j); at[4 + j] = km_swizzle(lin + 24 * j + 8 + t * 4); }
    }
    uint2 hd[4]; uint32_t qs[4];
    __device__ __forceinline__ void load(const uint8_t* m, const uint32_t (&at)[kLoads]) {
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) { hd[j] = *reinterpret_cast<const uint2*>(m + at[j]); qs[j] = *reinterpret_cast<const uint32_t*>(m + at[4 + j]); }
    }
    template <bool RAW = false> __device__ __forceinline__ bool header(uint32_t) const {
        __half2 top = __half2half2(__ushort_as_half(0));   // the largest magnitude of scales and minima; NaN where one is
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) top = __hmax2_nan(top, __habs2(*reinterpret_cast<const __half2*>(&hd[j].x)));
        const uint32_t w = *reinterpret_cast<const uint32_t*>(&top);
        return (w & 0x7c00u) != 0x7c00u && (w & 0x7c000000u) != 0x7c000000u;
    }
    // lane t: low nibbles of its word = weights 4t .. 4t + 3, high nibbles = 16 + 4t ..; fifth bits: bits 4t .. and 16 + 4t .. of the bit word,
    // bit k spread to bit 4 of byte k (the partial products of the multiplication do not meet)
    template <uint32_t G, bool RAW = false> __device__ __forceinline__ void get(uint32_t t, uint32_t (&a)[4], float& f, float& m) const {
        const uint32_t bits = hd[G].y >> (4u * t);
        k5_codes((qs[G] & 0x0f0f0f0fu) | (((bits & 15u) * 0x02040810u) & 0x10101010u), a[0], a[1]);
        k5_codes(((qs[G] >> 4) & 0x0f0f0f0fu) | ((((bits >> 16) & 15u) * 0x02040810u) & 0x10101010u), a[2], a[3]);
        const float m0 = half_bits_to_float(hd[G].x >> 16);
        f = half_bits_to_float(hd[G].x & 0xffffu); m = RAW ? m0 : fmaf(16.f, f, m0);
    }
};

// Rows that the split would not serve take FP32 sums of exactly rounded weights, from the same bytes in shared memory, part of K by part of K: rows
// with a run of eight values, not all zero, that are all below 1 after scaling (2^-14 of the row's largest or less). The halves end at
// 2^-25, so in every run that stays on the MMAs the values are good to 2^-25 of its largest, as good as FP32's own rounding of that one,
// whatever outlier is beside it. Infinities and NaN go the same way, and a row's path depends on that row alone. Normally distributed rows never
// get there. Layers whose input rows all hold an outlier of 5000 (whole rows of weights read again from global memory per unit / now / the FP32
// kernel): 13 rows 406 / 206 / 231 us, 64 rows on 16 experts 755 / 229 / 323 us.
constexpr float kKmNarrow = 1.f;

// What a tile's rows need in shared memory
struct KmTile {
    const float* x[8]; float* out[8]; float scale[8], inv[8];
    alignas(8) uint8_t wide[8];   // rows that take FP32 sums
};

// Out of line: the rare path takes no registers from the loop above it. This warp's part of K of one unit for the wide rows of the tile, up to four
// at a time, into their places of the unit's sums. linA, linB: the lane's rows' first bytes.
template <uint32_t TYPE>
__device__ __noinline__ void k5_wide_unit(const KmTile* tile, const uint8_t* mA, const uint8_t* mB, uint32_t linA, uint32_t linB, uint32_t part, uint32_t wpu,
                                          uint32_t steps, uint32_t count, float* sums) {
    using Step = KmStep<TYPE>;
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    for (uint32_t j = 0; j < count;) {
        uint32_t n = 0, list = 0;   // the next wide rows, four bits each
        for (; j < count && n < 4; ++j) if (tile->wide[j]) list |= j << (4u * n++);
        if (!n) break;
        float acc[4][2] = {};
        for (uint32_t st = part; st < steps; st += wpu) {
            uint32_t at[Step::kLoads];
            Step a, b;
            Step::offsets(linA + st * Step::kBytes, t, at); a.load(mA, at);
            Step::offsets(linB + st * Step::kBytes, t, at); b.load(mB, at);
            a.template header<true>(t); b.template header<true>(t);   // not finite: the loop above has reported it
            auto one = [&](auto gi) {
                constexpr uint32_t G = decltype(gi)::value;
                uint32_t ca[4], cb[4];
                float fa, ma, fb, mb, wa[8], wb[8];
                a.template get<G, true>(t, ca, fa, ma); b.template get<G, true>(t, cb, fb, mb);
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) {   // pairs (0, 2), (1, 3), (4, 6), (5, 7) of the lane's eight columns
                    const float2 va = __half22float2(*reinterpret_cast<const __half2*>(&ca[q])), vb = __half22float2(*reinterpret_cast<const __half2*>(&cb[q]));
                    const uint32_t i = (q >> 1) * 4u + (q & 1u);
                    wa[i] = fmaf(fa, va.x + 16.f, ma); wa[i + 2] = fmaf(fa, va.y + 16.f, ma);
                    wb[i] = fmaf(fb, vb.x + 16.f, mb); wb[i + 2] = fmaf(fb, vb.y + 16.f, mb);
                }
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    if (k >= n) break;
                    const float4* src = reinterpret_cast<const float4*>(tile->x[(list >> (4u * k)) & 15u] + (st * Step::kGroups + G) * 32u);
                    const float4 x0 = src[TYPE == 13u ? 2 * t : t], x1 = src[TYPE == 13u ? 2 * t + 1 : 4 + t];
                    const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) { acc[k][0] = fmaf(wa[i], x[i], acc[k][0]); acc[k][1] = fmaf(wb[i], x[i], acc[k][1]); }
                }
            };
            one(KmIndex<0>{}); one(KmIndex<1>{}); one(KmIndex<2>{}); one(KmIndex<3>{});
            if constexpr (Step::kGroups == 8) { one(KmIndex<4>{}); one(KmIndex<5>{}); one(KmIndex<6>{}); one(KmIndex<7>{}); }
        }
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t row = (list >> (4u * k)) & 15u;
#pragma unroll
            for (uint32_t q = 0; q < 2; ++q) {
                acc[k][q] += __shfl_xor_sync(0xffffffffu, acc[k][q], 1);
                acc[k][q] += __shfl_xor_sync(0xffffffffu, acc[k][q], 2);
                if (k < n && t == row >> 1) sums[lane * 4u + 2u * q + (row & 1u)] = acc[k][q];
            }
        }
    }
}

// Shared memory (from a multiple of 1024): barriers, tile table, high halves [8][x_stride], low halves [8][x_stride], group sums [group][8] (of the
// scaled values), partial sums [unit of a batch][K part][lane][4], stages [matrix][lines].
// WHOLE: where whole blocks per tile come out shorter than an even split, each tile gets as many blocks as there are for all. An even split has blocks
// that straddle tiles and stage the rows of both, a chain of loads and barriers worth p.staging units (about 2.5 us): a few units of short rows
// take no longer than that. 256 x 512 of 16 experts: 72 tiles 16 -> 11 us, 16 tiles 10.4 -> 7.5. With fewer than one and a half units per block few
// blocks straddle (12 tiles of 16 units 6.8 us, whole blocks 7.4).
__device__ __forceinline__ uint2 km_whole(uint32_t n_tiles, uint32_t tile_units, uint32_t staging) {   // first unit and number of units of this block
    const uint32_t n_units = n_tiles * tile_units, share = n_units / gridDim.x, rest = n_units - share * gridDim.x;
    const uint32_t per_tile = n_tiles ? gridDim.x / n_tiles : 0u;   // 0: more tiles than blocks
    if (per_tile && 2u * n_units >= 3u * gridDim.x && (tile_units + per_tile - 1u) / per_tile < share + staging) {   // uniform over the grid
        const uint32_t tile = blockIdx.x / per_tile, sub = blockIdx.x - tile * per_tile, from = tile_units * sub / per_tile;
        return tile < n_tiles ? make_uint2(tile * tile_units + from, tile_units * (sub + 1u) / per_tile - from) : make_uint2(0u, 0u);
    }
    const uint32_t more = rest * blockIdx.x / gridDim.x;   // the remainder spread over the blocks
    return make_uint2(share * blockIdx.x + more, share + rest * (blockIdx.x + 1u) / gridDim.x - more);
}
template <uint32_t TYPE, bool GATEUP, bool WHOLE>
__global__ void __launch_bounds__(kKmThreads, 1) gemv_k5_mma_kernel(const __grid_constant__ K5Maps maps, const K5Params p) {
    pdl_launch_dependents();
    extern __shared__ uint8_t km_raw[];
    __shared__ KmTile tl;
    __shared__ uint32_t s_top[8][kKmWarps];
    uint8_t* const km = km_raw + ((1024u - (smem_u32(km_raw) & 1023u)) & 1023u);
    uint64_t* const full = reinterpret_cast<uint64_t*>(km);
    uint64_t* const empty = full + kKmStages;
    uint32_t* const tt = reinterpret_cast<uint32_t*>(km + 256);             // [kKmTable + 1][12]: expert, first route, count, -, route ids; the last for a tile beyond
    uint8_t* const xhi = km + 2048;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t groups = p.cols / 32u, x_stride = p.cols * 2u + 64u;
    float* const sx = reinterpret_cast<float*>(km + p.off_sx);
    float4* const red = reinterpret_cast<float4*>(km + p.off_red);
    uint8_t* const ring = km + p.off_stage;
    constexpr uint32_t RW = GATEUP ? 8u : 16u, NMAT = GATEUP ? 2u : 1u;     // rows of one matrix per unit
    using Step = KmStep<TYPE>;
    const uint32_t S = p.stages;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < S; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], p.wpu); }
        mbar_fence_init();
    }
    pdl_wait();   // everything above touched shared memory only
    const uint32_t n_tiles = p.token_map ? p.tasks[0] : (p.tokens + 7u) / 8u;
    const uint32_t tile_units = p.rows / RW;     // whole: the launcher asks for it
    const uint64_t n_units = static_cast<uint64_t>(n_tiles) * tile_units;
    const uint64_t unit0 = WHOLE ? km_whole(n_tiles, tile_units, p.staging).x : n_units * blockIdx.x / gridDim.x;
    const uint32_t units = WHOLE ? km_whole(n_tiles, tile_units, p.staging).y : static_cast<uint32_t>(n_units * (blockIdx.x + 1) / gridDim.x - unit0);
    const uint32_t tile0 = WHOLE ? static_cast<uint32_t>(unit0) / tile_units : static_cast<uint32_t>(unit0 / tile_units);   // the run's first tile and unit in it
    const uint32_t first0 = WHOLE ? static_cast<uint32_t>(unit0) - tile0 * tile_units : static_cast<uint32_t>(unit0 % tile_units);
    // expert, first route and count of a tile (count 0: an entry that names no expert)
    auto look_up = [&](uint32_t tile, uint32_t& expert, uint32_t& start, uint32_t& count) {
        expert = 0; start = tile * 8u; count = 0;
        if (p.token_map) {
            const uint32_t e = p.tasks[2 + 2 * tile];
            start = p.tasks[3 + 2 * tile];
            if (e < p.experts) { const uint32_t c = p.counts[e]; expert = e; count = c > start ? min(c - start, 8u) : 0u; }
        } else if (start < p.tokens) count = min(p.tokens - start, 8u);
    };
    auto fill = [&](uint32_t* entry, uint32_t tile, uint32_t slot) {   // eight threads per entry
        uint32_t expert, start, count;
        look_up(tile, expert, start, count);
        if (slot == 0) { entry[0] = expert; entry[1] = start; entry[2] = count; }
        if (slot < count) entry[4 + slot] = p.token_map ? p.token_map[static_cast<uint64_t>(expert) * p.tokens + start + slot] : start + slot;
    };
    // the first tiles of the run, fetched at once: three dependent loads each
    for (uint32_t i = threadIdx.x; i < kKmTable * 8u; i += kKmThreads)
        if (tile0 + (i >> 3) < n_tiles && (i >> 3) * static_cast<uint64_t>(tile_units) < static_cast<uint64_t>(units) + first0) fill(tt + (i >> 3) * 12u, tile0 + (i >> 3), i & 7u);
    __syncthreads();

    if (warp >= kKmWarps) {
        // ------------------------------ producer warp ------------------------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kKmProdRegs));
        if (warp > kKmWarps) return;
        uint32_t stage = 0, phase = 0, filled = 0;
        bool ok = true;
        uint32_t tile = tile0, first = first0;
        for (uint32_t done = 0; done < units && ok; ++tile, first = 0) {
            const uint32_t seg = done;
            done = min(units, done + (tile_units - first));
            uint32_t expert, start, count;
            if (tile - tile0 < kKmTable) { expert = tt[(tile - tile0) * 12u]; count = tt[(tile - tile0) * 12u + 2]; }
            else look_up(tile, expert, start, count);
            if (count == 0) continue;
            const bool hi = expert >= p.split;
            const int el = static_cast<int>(hi ? expert - p.split : expert);
            for (uint32_t u = seg; u < done && ok; ++u, ++filled) {
                if (filled >= S) ok = __all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1u));
                if (!ok) { if (lane == 0) raise_error(p.error, TSP_ERR_TIMEOUT); break; }
                uint8_t* dst = ring + stage * p.stage_bytes;
                const uint32_t line = (first + u - seg) * (p.copies * p.copy_lines);
                if (elect_one()) {
                    mbar_arrive_expect_tx(&full[stage], NMAT * p.copies * p.copy_lines * 128u);
                    for (uint32_t m = 0; m < NMAT; ++m)
                        for (uint32_t c = 0; c < p.copies; ++c)
                            asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                                         ::"r"(smem_u32(dst + m * p.mat_bytes + c * p.copy_lines * 128u)), "l"(reinterpret_cast<uint64_t>(&maps.m[2 * m + (hi ? 1 : 0)])),
                                           "r"(smem_u32(&full[stage])), "r"(0), "r"(static_cast<int>(line + c * p.copy_lines)), "r"(el) : "memory");
                }
                __syncwarp();
                if (++stage == S) { stage = 0; phase ^= 1u; }
            }
        }
        return;
    }

    // -------------------------------- consumer warps --------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kKmConsRegs));
    constexpr uint32_t CT = kKmWarps * 32;
    const uint32_t steps = groups / Step::kGroups, wpu = p.wpu, part = warp & (wpu - 1u), ngroups = kKmWarps / wpu;
    const uint32_t my_steps = (steps - part + wpu - 1u) / wpu, batch = p.slots / wpu;   // K steps part, part + wpu, ...
    uint32_t mine = warp / wpu;                  // this warp's next unit of the run
    uint32_t filled = 0;                         // units brought before this tile's
    bool ready = true;                           // no wait has expired
    uint32_t atA[Step::kLoads], atB[Step::kLoads];   // (gate-up: the same for both matrices)
    Step::offsets(g * p.row_bytes + part * Step::kBytes, t, atA);
    if (!GATEUP) Step::offsets((g + 8u) * p.row_bytes + part * Step::kBytes, t, atB);
    uint32_t tile = tile0, first = first0;
    for (uint32_t done = 0; done < units; ++tile, first = 0) {   // uniform over the block
        const uint32_t seg = done, row0 = first;
        done = min(units, done + (tile_units - first));
        named_bar_sync(1, CT);                // the previous tile's rows are no longer read
        uint32_t* entry = tt + min(tile - tile0, kKmTable) * 12u;
        if (tile - tile0 >= kKmTable) {
            if (threadIdx.x < 8) fill(entry, tile, threadIdx.x);
            named_bar_sync(1, CT);
        }
        const uint32_t expert = entry[0], count = entry[2];
        if (count == 0) {   // uniform
            while (mine < done) mine += ngroups;
            continue;
        }
        const bool packed = count <= 4;   // low halves of row j in row j + 4: one pass instead of two
        // scale: a power of two from the row's largest magnitude
        for (uint32_t j = 0; j < count; ++j) {
            const uint4* x = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(p.x) + static_cast<uint64_t>(entry[4 + j] / p.in_div) * p.x_stride_bytes);
            uint32_t top = 0;
            for (uint32_t i = threadIdx.x; i < p.cols / 4u; i += CT) {
                const uint4 v = x[i];
                top = max(max(max(v.x & 0x7fffffffu, v.y & 0x7fffffffu), max(v.z & 0x7fffffffu, v.w & 0x7fffffffu)), top);
            }
            top = __reduce_max_sync(0xffffffffu, top);
            if (lane == 0) s_top[j][warp] = top;
        }
        named_bar_sync(1, CT);
        if (warp < 8) {
            uint32_t top = warp < count && lane < kKmWarps ? s_top[warp][lane] : 0u;
            top = __reduce_max_sync(0xffffffffu, top) >> 23;   // biased exponent of the largest magnitude
            if (lane == 0) {
                const uint32_t e = top >= 255u ? 127u : min(268u - top, 253u);   // not finite: a wide row
                tl.wide[warp] = warp < count && top >= 255u;
                tl.scale[warp] = __uint_as_float(e << 23); tl.inv[warp] = __uint_as_float((254u - e) << 23);
                if (warp < count) {
                    const uint32_t rid = entry[4 + warp];
                    tl.x[warp] = reinterpret_cast<const float*>(reinterpret_cast<const char*>(p.x) + static_cast<uint64_t>(rid / p.in_div) * p.x_stride_bytes);
                    tl.out[warp] = reinterpret_cast<float*>(reinterpret_cast<char*>(p.out) + static_cast<uint64_t>(rid) * p.out_stride_bytes);
                }
            }
        }
        named_bar_sync(1, CT);
        // stage: a thread takes the eight values that lane tq of a group multiplies, in the MMA's order
        for (uint32_t i = threadIdx.x; i < count * groups * 4u; i += CT) {
            const uint32_t j = i / (groups * 4u), rem = i - j * groups * 4u, grp = rem >> 2, tq = rem & 3u;
            const float4* src = reinterpret_cast<const float4*>(tl.x[j] + grp * 32u);
            const float4 f0 = src[TYPE == 13u ? 2 * tq : tq], f1 = src[TYPE == 13u ? 2 * tq + 1 : 4 + tq];
            const float sc = tl.scale[j];
            const float v[8] = {f0.x * sc, f0.z * sc, f0.y * sc, f0.w * sc, f1.x * sc, f1.z * sc, f1.y * sc, f1.w * sc};   // order 0,2,1,3
            uint32_t h[8], l[8];
            float sum = 0.f;
            const float most = fmaxf(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))),
                                     fmaxf(fmaxf(fabsf(v[4]), fabsf(v[5])), fmaxf(fabsf(v[6]), fabsf(v[7]))));
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const __half hv = __float2half_rn(v[q]);
                h[q] = __half_as_ushort(hv);
                l[q] = __half_as_ushort(__float2half_rn(v[q] - __half2float(hv)));
                sum += v[q];
            }
            if (most < kKmNarrow && most > 0.f) tl.wide[j] = 1;
            uint8_t* dst = xhi + j * x_stride + grp * 64u + tq * 16u;
            *reinterpret_cast<uint4*>(dst) = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
            *reinterpret_cast<uint4*>(dst + (packed ? 4u : 8u) * x_stride) = make_uint4(l[0] | (l[1] << 16), l[2] | (l[3] << 16), l[4] | (l[5] << 16), l[6] | (l[7] << 16));
            // count * groups * 4 is a multiple of four: the four lanes of a group are all here or none is
            const uint32_t quad = 0xfu << (lane & 28u);
            sum += __shfl_xor_sync(quad, sum, 1);
            sum += __shfl_xor_sync(quad, sum, 2);
            if (tq == 0) {
                sx[grp * 8u + j] = sum;
                if (packed) sx[grp * 8u + 4u + j] = 0.f;   // the offset's sum enters once, in the token's first column
            }
        }
        named_bar_sync(1, CT);
        const uint2 wide8 = *reinterpret_cast<const uint2*>(tl.wide);
        const bool wide = (wide8.x | wide8.y) != 0;   // some row of the tile
        const uint8_t* xh = xhi + g * x_stride + t * 16u;
        const float* sp = sx + 2 * t;
        uint32_t stage = (filled + mine - seg) % S, phase = ((filled + mine - seg) / S) & 1u;   // of this warp's next unit
        for (uint32_t b0 = seg; b0 < done; b0 += batch) {   // uniform over the block
            const uint32_t b1 = min(done, b0 + batch);
            for (; mine < b1; mine += ngroups) {
                if (ready) {
                    ready = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase));
                    if (!ready && lane == 0) raise_error(p.error, TSP_ERR_TIMEOUT);
                }
                const uint8_t* mA = ring + stage * p.stage_bytes;
                const uint8_t* mB = mA + (GATEUP ? p.mat_bytes : 0u);
                float total[4] = {0.f, 0.f, 0.f, 0.f};
                bool ok = true;
                auto work = [&](auto packed_tile) {   // two copies: as a run-time choice the second pass was predicated and issued all the same
                    constexpr bool PACKED = decltype(packed_tile)::value != 0;
                    for (uint32_t st = 0; st < my_steps; ++st) {
                        const uint32_t step = part + st * wpu;
                        if (my_steps > 1) {
                            Step::offsets(g * p.row_bytes + step * Step::kBytes, t, atA);
                            if (!GATEUP) Step::offsets((g + 8u) * p.row_bytes + step * Step::kBytes, t, atB);
                        }
                        Step a, b;
                        a.load(mA, atA); b.load(mB, GATEUP ? atA : atB);
                        ok &= a.header(t) & b.header(t);
                        float sum[4] = {0.f, 0.f, 0.f, 0.f}, low[4] = {0.f, 0.f, 0.f, 0.f};   // low: the low halves' sums of a tile that is not packed
                        auto one = [&](auto gi) {
                            constexpr uint32_t G = decltype(gi)::value;
                            uint32_t ca[4], cb[4];
                            float fa, ma, fb, mb, acc[4];
                            a.template get<G>(t, ca, fa, ma); b.template get<G>(t, cb, fb, mb);
                            const uint32_t grp = step * Step::kGroups + G;
                            k5_group_mma(acc, ca, cb, xh + grp * 64u);
                            if (!PACKED) {
                                float al[4];
                                k5_group_mma(al, ca, cb, xh + 8u * x_stride + grp * 64u);
                                low[0] = fmaf(fa, al[0], low[0]); low[1] = fmaf(fa, al[1], low[1]);
                                low[2] = fmaf(fb, al[2], low[2]); low[3] = fmaf(fb, al[3], low[3]);
                            }
                            const float2 s = *reinterpret_cast<const float2*>(sp + grp * 8u);
                            sum[0] = fmaf(fa, acc[0], fmaf(ma, s.x, sum[0])); sum[1] = fmaf(fa, acc[1], fmaf(ma, s.y, sum[1]));
                            sum[2] = fmaf(fb, acc[2], fmaf(mb, s.x, sum[2])); sum[3] = fmaf(fb, acc[3], fmaf(mb, s.y, sum[3]));
                        };
                        one(KmIndex<0>{}); one(KmIndex<1>{}); one(KmIndex<2>{}); one(KmIndex<3>{});
                        if constexpr (Step::kGroups == 8) { one(KmIndex<4>{}); one(KmIndex<5>{}); one(KmIndex<6>{}); one(KmIndex<7>{}); }
                        // high and low sums of a step meet here; packed: lane t ^ 2 holds the token's other column. The same additions either way:
                        // a row's result does not depend on how many rows share its tile
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q) total[q] += sum[q] + (PACKED ? __shfl_xor_sync(0xffffffffu, sum[q], 2) : low[q]);
                    }
                };
                if (packed) work(KmIndex<1>{});
                else work(KmIndex<0>{});
                float4* const sums = red + ((mine - b0) * wpu + part) * 32u;
                sums[lane] = make_float4(total[0], total[1], total[2], total[3]);
                if (wide)   // uniform over the block
                    k5_wide_unit<TYPE>(&tl, mA, mB, g * p.row_bytes, (GATEUP ? g : g + 8u) * p.row_bytes, part, wpu, steps, count, reinterpret_cast<float*>(sums));
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[stage]);
                stage += ngroups;
                while (stage >= S) { stage -= S; phase ^= 1u; }
                if (!ok) raise_error(p.error, TSP_ERR_NONFINITE);
            }
            named_bar_sync(1, CT);
            for (uint32_t u = b0 + warp; u < b1 && ready; u += kKmWarps) {
                const uint32_t r0 = (row0 + u - seg) * RW;
                float4 total = red[(u - b0) * wpu * 32u + lane];
                for (uint32_t k = 1; k < wpu; ++k) {
                    const float4 v = red[((u - b0) * wpu + k) * 32u + lane];
                    total.x += v.x; total.y += v.y; total.z += v.z; total.w += v.w;
                }
                // this lane: token rows 2t, 2t + 1; rows g of matrix A (x, y) and of matrix B / g + 8 (z, w)
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    const uint32_t j = 2 * t + q;
                    if (j >= count) continue;
                    const float inv = wide && tl.wide[j] ? 1.f : tl.inv[j], va = (q ? total.y : total.x) * inv, vb = (q ? total.w : total.z) * inv;
                    float* o = tl.out[j] + r0 + g;
                    if (GATEUP) {
                        const float v = (va >= 0.f ? va / (1.f + expf(-va)) : va * expf(va) / (1.f + expf(va))) * vb;
                        if (!finite_f32(v)) raise_error(p.error, TSP_ERR_NONFINITE);
                        *o = v;
                    } else {
                        if (!finite_f32(va) || !finite_f32(vb)) raise_error(p.error, TSP_ERR_NONFINITE);
                        o[0] = va; o[8] = vb;
                    }
                }
            }
            named_bar_sync(1, CT);   // the sums of the batch are read
        }
        filled += done - seg;
    }
}

// Exactly rounded FP32 weights of one matrix (test hook)
template <uint32_t TYPE>
__global__ void __launch_bounds__(256) dequant_k5_kernel(const uint8_t* __restrict__ m, uint64_t groups, float* __restrict__ out, uint32_t* error) {
    const uint64_t grp = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x;
    if (grp >= groups) return;
    // Group5 indexes blocks from the pointer it is given: hand it this group's own block
    const Group5<TYPE> g(TYPE == 13u ? m + (grp >> 3) * 176u : m + grp * 24u, TYPE == 13u ? static_cast<uint32_t>(grp & 7u) : 0u);
    float4* dst = reinterpret_cast<float4*>(out + grp * 32);
#pragma unroll
    for (uint32_t i4 = 0; i4 < 8; ++i4) { float w[4]; g.get(i4, w); dst[i4] = make_float4(w[0], w[1], w[2], w[3]); }
    if (!g.finite) raise_error(error, TSP_ERR_NONFINITE);
}

int launch_dequant_k5(uint32_t type, const uint8_t* m, uint64_t elements, float* out, uint32_t* error, cudaStream_t st) {
    const uint64_t groups = elements / 32;
    const unsigned grid = static_cast<unsigned>((groups + 255) / 256);
    if (type == TSP_TYPE_Q5_K) dequant_k5_kernel<13u><<<grid, 256, 0, st>>>(m, groups, out, error);
    else dequant_k5_kernel<7u><<<grid, 256, 0, st>>>(m, groups, out, error);
    TSP_CUDA(cudaGetLastError());
    return TSP_OK;
}

template <uint32_t TYPE, bool GATEUP, bool WHOLE>
static int launch_km(const K5Maps& maps, const K5Params& p, size_t smem, int grid, cudaStream_t st) {
    static thread_local int regs_ok = -1;   // the register hand-over adds up for this build
    if (regs_ok < 0) {
        cudaFuncAttributes fa{};
        TSP_CUDA(cudaFuncGetAttributes(&fa, gemv_k5_mma_kernel<TYPE, GATEUP, WHOLE>));
        regs_ok = (fa.numRegs >= kKmProdRegs && static_cast<int>(kKmWarps) * (kKmConsRegs - fa.numRegs) <= 4 * (fa.numRegs - kKmProdRegs)) ? 1 : 0;
    }
    if (!regs_ok) return fail(TSP_E_CUDA, "five-bit projection kernel: the compiled register count does not allow the producer/consumer register hand-over");
    static thread_local SmemAttrCache configured;   // per kernel instantiation, keyed by device
    TSP_CUDA(ensure_dynamic_smem(gemv_k5_mma_kernel<TYPE, GATEUP, WHOLE>, configured, smem));
    TSP_CUDA(launch_pdl(gemv_k5_mma_kernel<TYPE, GATEUP, WHOLE>, dim3(grid), dim3(kKmThreads), smem, st, maps, p));
    return TSP_OK;
}

template <uint32_t TYPE, bool GATEUP, uint32_t MT>
static int launch_k5(const K5Params& p, dim3 grid, size_t smem, cudaStream_t st) {
    static thread_local SmemAttrCache configured;   // per kernel instantiation, keyed by device
    TSP_CUDA(ensure_dynamic_smem(gemv_k5_kernel<TYPE, GATEUP, MT>, configured, smem));
    TSP_CUDA(launch_pdl(gemv_k5_kernel<TYPE, GATEUP, MT>, grid, dim3(kK5Threads), smem, st, p));
    return TSP_OK;
}

int launch_gemv_k5(const tsp_matrix_set* a, const tsp_matrix_set* b, bool gateup, const float* x, uint64_t x_stride_bytes, uint32_t in_div,
                   uint32_t tokens, const uint32_t* token_map, const uint32_t* counts, const uint32_t* tasks, float* out,
                   uint64_t out_stride_bytes, int nc, uint32_t* error, cudaStream_t st) {
    if (a->layout != TSP_LAYOUT_GGUF) return fail(TSP_E_TYPE, "five-bit encodings are read as plain GGUF rows only");
    if (nc != 1 && nc != 2) return fail(TSP_E_ARG, "five-bit projection: tiles hold 8 or 16 token rows");
    K5Params p{};
    p.a_base = static_cast<const uint8_t*>(a->base);
    p.a_base_hi = static_cast<const uint8_t*>(a->base_hi ? a->base_hi : a->base);
    if (gateup) {
        p.b_base = static_cast<const uint8_t*>(b->base);
        p.b_base_hi = static_cast<const uint8_t*>(b->base_hi ? b->base_hi : b->base);
    }
    p.expert_stride = a->expert_stride;
    p.split = a->split < a->experts ? a->split : a->experts;
    p.experts = a->experts;
    p.rows = a->rows; p.cols = a->cols;
    p.row_bytes = a->type == TSP_TYPE_Q5_K ? a->cols / 256 * 176 : a->cols / 32 * 24;
    p.x = x; p.x_stride_bytes = x_stride_bytes; p.in_div = in_div ? in_div : 1;
    p.token_map = token_map; p.counts = counts; p.tasks = tasks;
    p.tokens = tokens; p.tile_tokens = 8u * static_cast<uint32_t>(nc);
    p.out = out; p.out_stride_bytes = out_stride_bytes; p.error = error;
    const uint32_t groups = a->cols / 32;
    const int sms = sm_count();
    if (sms <= 0) return fail(TSP_E_CUDA, "no usable CUDA device");
    p.lanes_per_row = 1;
    while (p.lanes_per_row * 2 <= groups && p.lanes_per_row < 32) p.lanes_per_row *= 2;
    // Tiles of up to 8 rows take the MMA kernel where a unit's rows are whole, K is whole steps and the tile's rows leave room for two units in
    // flight (up to 3328 columns); dense batches of more rows (16 per tile) and the other shapes keep the FP32 FMA kernel.
    const uint32_t dense_tiles = (tokens + p.tile_tokens - 1) / p.tile_tokens, rw = gateup ? 8u : 16u;
    const uint32_t km_groups = a->type == TSP_TYPE_Q5_K ? 8u : 4u;
    if (nc == 1 && a->rows % rw == 0 && groups % km_groups == 0 && a->cols <= 3328) {
        for (p.wpu = 1; p.wpu < kKmParts && groups / km_groups >= 2u * p.wpu;) p.wpu *= 2;
        const uint32_t lines = rw * p.row_bytes / 128u;   // whole: eight rows of 176 or 96 bytes a step
        p.staging = min(4000u / a->cols, 5u);             // 2.5 us against 0.6 ns a column, and half a microsecond for a unit of few
        p.copies = (lines + 255u) / 256u;                 // a box holds 256 lines at most; 16 rows are an even number of lines
        p.copy_lines = lines / p.copies;
        p.mat_bytes = (lines * 128u + 1023u) & ~1023u;
        p.stage_bytes = (gateup ? 2u : 1u) * p.mat_bytes;
        const uint32_t budget = 225 * 1024;               // of the 227 KB, the static tile record and the alignment of the base taken off
        p.off_sx = 2048u + 16u * (a->cols * 2u + 64u);
        p.off_red = p.off_sx + groups * 32u;
        for (p.slots = 128; p.slots > kKmParts && p.off_red + p.slots * 512u + (kKmWarps / p.wpu > 4u ? kKmWarps / p.wpu : 4u) * p.stage_bytes > budget;) p.slots /= 2;   // units in flight before long batches
        p.off_stage = (p.off_red + p.slots * 512u + 1023u) & ~1023u;
        // The warps that share a unit take every unit_groups-th one. A whole number of such rounds in the ring: the unit that had a unit's stage before
        // it was then read by the same warps, so that a wait is never a phase of the barrier too early.
        const uint32_t unit_groups = kKmWarps / p.wpu;
        p.stages = (budget - p.off_stage) / p.stage_bytes;
        p.stages = (p.stages < kKmStages ? p.stages : kKmStages) / unit_groups * unit_groups;
        if (p.copies * p.copy_lines != lines || p.stages < 2) return fail(TSP_E_ARG, "five-bit projection: no room for the weight rows in shared memory");
        K5Maps maps;
        const uint32_t n_lo = p.split ? p.split : 1u, n_hi = p.experts > p.split ? p.experts - p.split : 1u;
        for (uint32_t m = 0; m < (gateup ? 2u : 1u); ++m)
            for (uint32_t hi = 0; hi < 2; ++hi) {
                const uint64_t dims[3] = {128, static_cast<uint64_t>(a->rows) * p.row_bytes / 128u, hi ? n_hi : n_lo};
                const uint64_t strides[2] = {128, a->experts > 1 ? a->expert_stride : 16};
                const uint32_t box[3] = {128, p.copy_lines, 1};
                if (int rc = get_tensor_map_bytes(m ? (hi ? p.b_base_hi : p.b_base) : (hi ? p.a_base_hi : p.a_base), 3, dims, strides, box, true, &maps.m[2 * m + hi])) return rc;
            }
        if (!gateup) { maps.m[2] = maps.m[0]; maps.m[3] = maps.m[1]; }
        const size_t km_smem = p.off_stage + static_cast<size_t>(p.stages) * p.stage_bytes + 1024;
        // Whole blocks per tile: routed batches whose tiles are little work beside a staging (up to 32 units of 512 columns). Larger ones gain little and pay
        // 0.2 to 0.4 us a launch for the choice, as batches of a few rows do; 2048 columns in this form's arithmetic came out 2.5 % slower.
        const bool whole = token_map && tokens >= 8 && a->rows / rw * a->cols <= 16384u;
#define TSP_KM(T, G) (whole ? launch_km<T, G, true>(maps, p, km_smem, sms, st) : launch_km<T, G, false>(maps, p, km_smem, sms, st))
        if (a->type == TSP_TYPE_Q5_K) return gateup ? TSP_KM(13u, true) : TSP_KM(13u, false);
        return gateup ? TSP_KM(7u, true) : TSP_KM(7u, false);
#undef TSP_KM
    }
    const size_t smem = static_cast<size_t>(p.tile_tokens) * groups * 9 * sizeof(float4);
    if (smem > 200 * 1024) return fail(TSP_E_ARG, "five-bit projection: %u columns x %u token rows do not fit the activation staging", a->cols, p.tile_tokens);
    // routed launches learn their tile count on the device: a fixed number of block rows walks the tiles (a routed launch has at
    // most 64 routes per token row, one tile each at worst)
    const uint64_t routed_cap = static_cast<uint64_t>(tokens) * 64u;
    const uint32_t walkers = static_cast<uint32_t>(routed_cap < 4u * static_cast<uint32_t>(sms) ? routed_cap : 4u * static_cast<uint32_t>(sms));
    const dim3 grid((a->rows + kK5BlockRows - 1) / kK5BlockRows, token_map ? walkers : (dense_tiles < 1024u ? dense_tiles : 1024u));
    if (a->type == TSP_TYPE_Q5_K) {
        if (gateup) return nc == 1 ? launch_k5<13u, true, 8u>(p, grid, smem, st) : launch_k5<13u, true, 16u>(p, grid, smem, st);
        return nc == 1 ? launch_k5<13u, false, 8u>(p, grid, smem, st) : launch_k5<13u, false, 16u>(p, grid, smem, st);
    }
    if (gateup) return nc == 1 ? launch_k5<7u, true, 8u>(p, grid, smem, st) : launch_k5<7u, true, 16u>(p, grid, smem, st);
    return nc == 1 ? launch_k5<7u, false, 8u>(p, grid, smem, st) : launch_k5<7u, false, 16u>(p, grid, smem, st);
}

}  // namespace tsp
