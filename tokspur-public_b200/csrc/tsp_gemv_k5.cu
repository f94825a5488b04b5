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
#include "tsp_common.cuh"

namespace tsp {

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
    uint32_t item_warps;      // MMA kernel, SPLIT: warps of a block that take rows of an item
    uint32_t lanes_per_row;   // lanes that share one weight row: the largest power of two <= min(32, groups)
    float* out; uint64_t out_stride_bytes;
    uint32_t* error;
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
// A warp owns 8 hidden units (8 gate + 8 up rows) or 16 plain rows over the whole K, its weights loaded straight into registers one
// step ahead (a row's bytes are read by the four lanes that use them: 32-byte pieces); blocks of eight warps walk (tile, row block)
// items, two blocks per SM, so that one streams while the other stages its rows.
// The groups of a step are summed by themselves before they join the total: one chain over K of 2048 was further from 64-bit sums
// (2.1e-7, relative 2-norm) than the FP32 kernel (1.5e-7).
// Measured against the FP32 kernel, whole layer of 512 experts of 512 x 2048, ten per token: 13 rows 228 -> 187 us, 64 rows 644 -> 492 us.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kKmWarps = 8;

// 16 rows x 32 columns of codes (two K steps of 16) against 8 token rows: acc = (codes - 16) x scaled activations
__device__ __forceinline__ void k5_group_mma(float (&acc)[4], const uint32_t (&a)[4], const uint32_t (&b)[4], const uint8_t* x) {
    const uint4 v = *reinterpret_cast<const uint4*>(x);
    mma_f16_16816_zero(acc, a[0], b[0], a[1], b[1], v.x, v.y);
    mma_f16_16816(acc, a[2], b[2], a[3], b[3], v.z, v.w);
}
// four code bytes: nibbles in the low half of each byte of `q`, fifth bits at bit 4 of each byte of `h` (other bits are noise)
__device__ __forceinline__ void k5_codes(uint32_t q, uint32_t h, uint32_t& even, uint32_t& odd) {
    const uint32_t c = (q & 0x0f0f0f0fu) | (h & 0xf0f0f0f0u);
    // 0x6400 | code = 1024 + code; the subtraction is exact
    const uint32_t e = (c & 0x001f001fu) | 0x64006400u, o = ((c >> 8) & 0x001f001fu) | 0x64006400u;
    const __half2 k1040 = __float2half2_rn(1040.f);
    const __half2 he = __hsub2(*reinterpret_cast<const __half2*>(&e), k1040), ho = __hsub2(*reinterpret_cast<const __half2*>(&o), k1040);
    even = *reinterpret_cast<const uint32_t*>(&he); odd = *reinterpret_cast<const uint32_t*>(&ho);
}
template <int S> __device__ __forceinline__ uint32_t shl_s(uint32_t v) { return S >= 0 ? v << (S >= 0 ? S : 0) : v >> (S < 0 ? -S : 0); }

template <uint32_t I> struct KmIndex { static constexpr uint32_t value = I; };
template <uint32_t TYPE> struct KmStep;
// Q5_K: a step is one 256-weight super-block of a row
template <> struct KmStep<13u> {
    static constexpr uint32_t kGroups = 8, kBytes = 176;
    uint4 hd; uint2 qh, qs[4];
    __device__ __forceinline__ void load(const uint8_t* blk, uint32_t t) {
        hd = *reinterpret_cast<const uint4*>(blk);
        qh = *reinterpret_cast<const uint2*>(blk + 16 + t * 8);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) qs[j] = *reinterpret_cast<const uint2*>(blk + 48 + j * 32 + t * 8);
    }
    uint32_t sc[2], mn[2]; float d, dmin;   // 6-bit factors as bytes (numeric.cpp:25-31)
    __device__ __forceinline__ bool header() {
        sc[0] = hd.y & 0x3f3f3f3fu; mn[0] = hd.z & 0x3f3f3f3fu;
        sc[1] = (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);
        mn[1] = ((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u);
        d = half_bits_to_float(hd.x & 0xffffu); dmin = half_bits_to_float(hd.x >> 16);
        return finite_f32(d) && finite_f32(dmin);
    }
    // code pairs, scale (an exact product) and offset (one rounding) of group G
    template <uint32_t G> __device__ __forceinline__ void group(uint32_t, uint32_t (&a)[4], float& f, float& m) const {
        constexpr uint32_t J = G >> 1, HI = G & 1u;
        k5_codes(HI ? qs[J].x >> 4 : qs[J].x, shl_s<4 - static_cast<int>(G)>(qh.x), a[0], a[1]);
        k5_codes(HI ? qs[J].y >> 4 : qs[J].y, shl_s<4 - static_cast<int>(G)>(qh.y), a[2], a[3]);
        f = d * byte_f32<G & 3u>(sc[G >> 2]);
        m = fmaf(16.f, f, -(dmin * byte_f32<G & 3u>(mn[G >> 2])));
    }
};
// Q5_1: a step is four 32-weight blocks of a row
template <> struct KmStep<7u> {
    static constexpr uint32_t kGroups = 4, kBytes = 96;
    uint2 hd[4]; uint32_t qs[4];
    __device__ __forceinline__ void load(const uint8_t* blk, uint32_t t) {
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            hd[j] = *reinterpret_cast<const uint2*>(blk + 24 * j);
            qs[j] = *reinterpret_cast<const uint32_t*>(blk + 24 * j + 8 + t * 4);
        }
    }
    __device__ __forceinline__ bool header() const {
        bool ok = true;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) ok &= (hd[j].x & 0x7c00u) != 0x7c00u && (hd[j].x & 0x7c000000u) != 0x7c000000u;
        return ok;
    }
    // lane t: low nibbles of its word = weights 4t .. 4t + 3, high nibbles = 16 + 4t ..; fifth bits: bits 4t .. and 16 + 4t .. of the bit word,
    // bit k spread to bit 4 of byte k (the partial products of the multiplication do not meet)
    template <uint32_t G> __device__ __forceinline__ void group(uint32_t t, uint32_t (&a)[4], float& f, float& m) const {
        const uint32_t bits = hd[G].y >> (4u * t);
        k5_codes(qs[G], (bits & 15u) * 0x02040810u, a[0], a[1]);
        k5_codes(qs[G] >> 4, ((bits >> 16) & 15u) * 0x02040810u, a[2], a[3]);
        f = half_bits_to_float(hd[G].x & 0xffffu); m = fmaf(16.f, f, half_bits_to_float(hd[G].x >> 16));
    }
};

// Rows that the split would not serve take the FP32 sums (k5_row_f32, by the warp that has the matrix rows, straight from global memory): rows
// with a run of eight values, not all zero, that are all below 1 after scaling (2^-14 of the row's largest or less). The halves end at
// 2^-25, so in every run that stays on the MMAs the values are good to 2^-25 of its largest, as good as FP32's own rounding of that one,
// whatever outlier is beside it. Infinities and NaN go the same way, and a row's path depends on that row alone. Normally distributed rows never
// get there. Layers whose input rows all hold an outlier of 5000 (the limit at 2^-10 and one row at a time / now / the FP32 kernel): 13 rows
// 492 / 264 / 231 us, 64 rows on 16 experts 949 / 297 / 323 us.
constexpr float kKmNarrow = 1.f;

// What a tile's rows need in shared memory, and what the rare path below reads of the launch (from here, so that the kernel keeps nothing for it)
struct KmTile {
    const float* x[8]; float* out[8]; float scale[8], inv[8];
    alignas(8) uint8_t wide[8];   // rows that take FP32 sums
    uint32_t row_bytes, groups, lanes_per_row; uint32_t* error;
};

// Out of line: the rare path takes no registers from the loop above it. Up to four token rows at a time; out row r of the warp's `rows` at r0 + r.
template <uint32_t TYPE, bool GATEUP>
__device__ __noinline__ void k5_wide_rows(const KmTile* tile, const uint8_t* rowsA, const uint8_t* rowsB, uint32_t count, uint32_t r0) {
    const uint32_t lpr = tile->lanes_per_row, groups = tile->groups, row_bytes = tile->row_bytes, rows = GATEUP ? 8u : 16u;
    const uint32_t lane = threadIdx.x & 31u, rpw = 32u / lpr, sub = lane / lpr, lig = lane & (lpr - 1u);
    bool ok = true;
    for (uint32_t j = 0; j < count;) {
        uint32_t n = 0, list = 0;   // the next wide rows, four bits each
        for (; j < count && n < 4; ++j) if (tile->wide[j]) list |= j << (4u * n++);
        if (!n) break;
        for (uint32_t rb = 0; rb < rows; rb += rpw) {
            const uint32_t r = rb + sub;
            const bool live = r < rows;
            const uint32_t at = (live ? r : rb) * row_bytes;
            const bool weights = k5_row_f32<TYPE, GATEUP, 4u>(
                rowsA + at, rowsB + at, groups, lpr, lig, n,
                [&](uint32_t k, uint32_t grp, uint32_t i4) { return reinterpret_cast<const float4*>(tile->x[(list >> (4u * k)) & 15u])[grp * 8u + i4]; },
                [&](uint32_t k, float v) {
                    if (!live) return;
                    ok = ok && finite_f32(v);
                    tile->out[(list >> (4u * k)) & 15u][r0 + r] = v;
                });
            ok = ok && weights;
        }
    }
    if (!ok) raise_error(tile->error, TSP_ERR_NONFINITE);
}

// Shared memory: high halves [8][x_stride], low halves [8][x_stride], group sums [group][8] (of the scaled values)
// SPLIT: only the first item_warps warps of a block take rows (all of them stage).
template <uint32_t TYPE, bool GATEUP, bool SPLIT>
__global__ void __launch_bounds__(kKmWarps * 32, 2) gemv_k5_mma_kernel(const K5Params p) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) uint8_t km_smem[];
    __shared__ KmTile tl;
    if (threadIdx.x == 0) { tl.row_bytes = p.row_bytes; tl.groups = p.cols / 32u; tl.lanes_per_row = p.lanes_per_row; tl.error = p.error; }   // read behind barriers
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t groups = p.cols / 32u, x_stride = p.cols * 2u + 64u;
    uint8_t* const xhi = km_smem;
    float* const sx = reinterpret_cast<float*>(km_smem + 16u * x_stride);
    constexpr uint32_t RW = GATEUP ? 8u : 16u;   // rows of one matrix per warp
    using Step = KmStep<TYPE>;
    const uint32_t steps = groups / Step::kGroups;
    pdl_wait();
    const uint32_t n_tiles = p.token_map ? p.tasks[0] : (p.tokens + 7u) / 8u;
    const uint32_t item_rows = RW * (SPLIT ? p.item_warps : kKmWarps), row_items = (p.rows + item_rows - 1) / item_rows;
    const uint32_t n_items = n_tiles * row_items;
    for (uint32_t item = blockIdx.x; item < n_items; item += gridDim.x) {   // uniform over the block
        const uint32_t tile = item / row_items, r0 = (item - tile * row_items) * item_rows + warp * RW;
        uint32_t expert = 0, start = tile * 8u, count = 0;
        if (p.token_map) {
            expert = p.tasks[2 + 2 * tile];
            start = p.tasks[3 + 2 * tile];
            if (expert < p.experts) { const uint32_t c = p.counts[expert]; count = c > start ? min(c - start, 8u) : 0u; }
            else expert = 0;
        } else if (start < p.tokens) count = min(p.tokens - start, 8u);
        if (count == 0) continue;   // uniform
        const bool packed = count <= 4;   // low halves of row j in row j + 4: one pass instead of two
        const bool hi = expert >= p.split;
        const uint64_t eoff = static_cast<uint64_t>(hi ? expert - p.split : expert) * p.expert_stride;
        const uint8_t* baseA = (hi ? p.a_base_hi : p.a_base) + eoff;
        const bool live = (!SPLIT || warp < p.item_warps) && r0 < p.rows;   // whole warps: rows are a multiple of RW
        const uint32_t rowA = (live ? r0 : 0u) + g;
        const uint8_t* wA = baseA + static_cast<uint64_t>(rowA) * p.row_bytes;
        const uint8_t* wB = GATEUP ? (hi ? p.b_base_hi : p.b_base) + eoff + static_cast<uint64_t>(rowA) * p.row_bytes
                                   : baseA + static_cast<uint64_t>(rowA + 8u) * p.row_bytes;
        Step nA, nB;
        if (!SPLIT || live) { nA.load(wA, t); nB.load(wB, t); }   // on their way while the rows are staged
        __syncthreads();                  // the previous item's rows are no longer read
        if (warp < count) {               // warp j: route id and scale of token row j
            const uint32_t rid = p.token_map ? p.token_map[static_cast<uint64_t>(expert) * p.tokens + start + warp] : start + warp;
            const float* x = reinterpret_cast<const float*>(reinterpret_cast<const char*>(p.x) + static_cast<uint64_t>(rid / p.in_div) * p.x_stride_bytes);
            uint32_t top = 0;
            for (uint32_t i = lane; i < p.cols / 4u; i += 32) {
                const uint4 v = reinterpret_cast<const uint4*>(x)[i];
                top = max(max(max(v.x & 0x7fffffffu, v.y & 0x7fffffffu), max(v.z & 0x7fffffffu, v.w & 0x7fffffffu)), top);
            }
            top = __reduce_max_sync(0xffffffffu, top) >> 23;   // biased exponent of the largest magnitude
            if (lane == 0) {
                const uint32_t e = top >= 255u ? 127u : min(268u - top, 253u);   // not finite: a wide row
                tl.wide[warp] = top >= 255u;
                tl.scale[warp] = __uint_as_float(e << 23); tl.inv[warp] = __uint_as_float((254u - e) << 23);
                tl.x[warp] = x;
                tl.out[warp] = reinterpret_cast<float*>(reinterpret_cast<char*>(p.out) + static_cast<uint64_t>(rid) * p.out_stride_bytes);
            }
        } else if (lane == 0) tl.wide[warp] = 0;
        __syncthreads();
        // stage: a thread takes the eight values that lane tq of a group multiplies, in the MMA's order
        for (uint32_t i = threadIdx.x; i < count * groups * 4u; i += kKmWarps * 32) {
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
        __syncthreads();
        if (!live) continue;
        const uint2 wide8 = *reinterpret_cast<const uint2*>(tl.wide);
        const bool wide = (wide8.x | wide8.y) != 0;   // some row of the tile
        float total[4] = {0.f, 0.f, 0.f, 0.f}, low[4] = {0.f, 0.f, 0.f, 0.f};   // low: the low halves' sums of a tile that is not packed
        bool ok = true;
        const uint8_t* xh = xhi + g * x_stride + t * 16u;
        const float* sp = sx + 2 * t;
        for (uint32_t st = 0; st < steps; ++st) {
            Step a = nA, b = nB;
            if (st + 1 < steps) { nA.load(wA + (st + 1) * Step::kBytes, t); nB.load(wB + (st + 1) * Step::kBytes, t); }
            ok &= a.header() & b.header();
            float part[4] = {0.f, 0.f, 0.f, 0.f}, part_low[4] = {0.f, 0.f, 0.f, 0.f};   // this step's groups: short chains of additions
            auto one = [&](auto gi) {
                constexpr uint32_t G = decltype(gi)::value;
                uint32_t ca[4], cb[4];
                float fa, ma, fb, mb, acc[4];
                a.template group<G>(t, ca, fa, ma); b.template group<G>(t, cb, fb, mb);
                const uint32_t grp = st * Step::kGroups + G;
                k5_group_mma(acc, ca, cb, xh + grp * 64u);
                if (!packed) {
                    float al[4];
                    k5_group_mma(al, ca, cb, xh + 8u * x_stride + grp * 64u);
                    part_low[0] = fmaf(fa, al[0], part_low[0]); part_low[1] = fmaf(fa, al[1], part_low[1]);
                    part_low[2] = fmaf(fb, al[2], part_low[2]); part_low[3] = fmaf(fb, al[3], part_low[3]);
                }
                const float2 s = *reinterpret_cast<const float2*>(sp + grp * 8u);
                part[0] = fmaf(fa, acc[0], fmaf(ma, s.x, part[0])); part[1] = fmaf(fa, acc[1], fmaf(ma, s.y, part[1]));
                part[2] = fmaf(fb, acc[2], fmaf(mb, s.x, part[2])); part[3] = fmaf(fb, acc[3], fmaf(mb, s.y, part[3]));
            };
            one(KmIndex<0>{}); one(KmIndex<1>{}); one(KmIndex<2>{}); one(KmIndex<3>{});
            if constexpr (Step::kGroups == 8) { one(KmIndex<4>{}); one(KmIndex<5>{}); one(KmIndex<6>{}); one(KmIndex<7>{}); }
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) { total[q] += part[q]; if (!packed) low[q] += part_low[q]; }
        }
        if (packed) {   // lane t ^ 2 holds the token's other column
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) total[q] += __shfl_xor_sync(0xffffffffu, total[q], 2);
        } else {   // the same sum: a row's result does not depend on how many rows share its tile
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) total[q] += low[q];
        }
        if (!ok) raise_error(p.error, TSP_ERR_NONFINITE);
        // this lane: token rows 2t, 2t + 1; rows g of matrix A (total[0..1]) and of matrix B / g + 8 (total[2..3])
#pragma unroll
        for (uint32_t q = 0; q < 2; ++q) {
            const uint32_t j = 2 * t + q;
            if (j >= count || (wide && tl.wide[j])) continue;
            const float inv = tl.inv[j], va = total[q] * inv, vb = total[2 + q] * inv;
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
        if (wide)   // uniform over the block
            k5_wide_rows<TYPE, GATEUP>(&tl, wA - static_cast<uint64_t>(g) * p.row_bytes, (GATEUP ? wB : wA) - static_cast<uint64_t>(g) * p.row_bytes, count, r0);
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

template <uint32_t TYPE, bool GATEUP, bool SPLIT>
static int launch_km_t(const K5Params& p, size_t smem, int grid, cudaStream_t st) {
    static thread_local SmemAttrCache configured;   // per kernel instantiation, keyed by device
    TSP_CUDA(ensure_dynamic_smem(gemv_k5_mma_kernel<TYPE, GATEUP, SPLIT>, configured, smem));
    TSP_CUDA(launch_pdl(gemv_k5_mma_kernel<TYPE, GATEUP, SPLIT>, dim3(grid), dim3(kKmWarps * 32), smem, st, p));
    return TSP_OK;
}
template <uint32_t TYPE, bool GATEUP>
static int launch_km(const K5Params& p, size_t smem, int grid, cudaStream_t st) {
    return p.item_warps < kKmWarps ? launch_km_t<TYPE, GATEUP, true>(p, smem, grid, st) : launch_km_t<TYPE, GATEUP, false>(p, smem, grid, st);
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
    // Tiles of up to 8 rows take the MMA kernel where a warp's rows are whole and two blocks' rows fit an SM's shared memory (up to 3328
    // columns); dense batches of more rows (16 per tile) and the other shapes keep the FP32 FMA kernel.
    // A dense launch of fewer than half as many items as SMs takes fewer warps per item: eight would leave most SMs idle (one row of Q5_1
    // 2048 x 512: 7.0 us on 16 SMs, the FP32 kernel's 32 blocks 5.5; 4.3 us on 128). Routed launches learn their items on the device; with the
    // count of warps a variable there, too, a layer of 64 rows took 506 us instead of 491.
    const uint32_t row_warps = (a->rows + (gateup ? 7u : 15u)) / (gateup ? 8u : 16u), dense_tiles = (tokens + p.tile_tokens - 1) / p.tile_tokens;
    for (p.item_warps = kKmWarps; !token_map && p.item_warps > 1 && 2ull * dense_tiles * ((row_warps + p.item_warps - 1) / p.item_warps) <= static_cast<uint32_t>(sms);) p.item_warps /= 2;
    const size_t km_smem = 16u * (a->cols * 2u + 64u) + groups * 32u;
    if (nc == 1 && a->rows % (gateup ? 8 : 16) == 0 && groups % (a->type == TSP_TYPE_Q5_K ? 8 : 4) == 0 && km_smem <= 110 * 1024) {
        if (a->type == TSP_TYPE_Q5_K) return gateup ? launch_km<13u, true>(p, km_smem, 2 * sms, st) : launch_km<13u, false>(p, km_smem, 2 * sms, st);
        return gateup ? launch_km<7u, true>(p, km_smem, 2 * sms, st) : launch_km<7u, false>(p, km_smem, 2 * sms, st);
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
