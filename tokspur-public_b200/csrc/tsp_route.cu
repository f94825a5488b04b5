// Router top-k, stable token permutation, gated combine and the activation edge conversions.
// All integer results (ids, token_map, counts, tasks) are deterministic and independent of
// scheduling: no atomics decide an order anywhere.
#include "tsp_common.cuh"
#include "tsp_q8_rows.cuh"
#include "tsp_route_row.cuh"
#include "tsp_rows_f16k.cuh"

namespace tsp {

// ---------------------------------------------------------------------------------------------
// route: one warp per token row. Selection order is (logit descending, id ascending), i.e. the
// total order of route_reference (routing.cpp:15-18). Logits are compared as FP32, which orders
// exactly as the reference's doubles do because the conversion is exact.
// Weights are evaluated in double so that they round to the same FP32 as the reference's.
// ---------------------------------------------------------------------------------------------
constexpr int kRouteWarps = 4;  // at most; fewer when a row of logits is long, to stay inside 48 KB of shared memory

// One warp routes one token row; `row` is the warp's scratch of `experts` floats in shared memory.
// `margins` (optional): margins[token] = logit of the last selected expert - logit of the best expert left out (+inf when every
// expert is selected): how far the selection is from changing under a perturbation of the logits.
__device__ __forceinline__ void route_row(float* row, const float* src, uint32_t token, uint32_t experts, uint32_t selected,
                                          uint32_t mode, int normalize, uint32_t* __restrict__ ids, float* __restrict__ weights,
                                          uint32_t* error, uint32_t lane, float* __restrict__ margins = nullptr) {
    bool bad = false;
    for (uint32_t e = lane; e < experts; e += 32) {
        const float v = src[e];
        bad |= !finite_f32(v);
        row[e] = v;
    }
    bad = __any_sync(0xffffffffu, bad);
    __syncwarp();
    uint32_t* out_ids = ids + static_cast<uint64_t>(token) * selected;
    float* out_w = weights + static_cast<uint64_t>(token) * selected;
    if (bad) {  // reference: FormatError("nonfinite router logit"); here: flag and publish a harmless row
        if (lane == 0) raise_error(error, TSP_ERR_NONFINITE);
        for (uint32_t r = lane; r < selected; r += 32) { out_ids[r] = r; out_w[r] = 0.f; }
        if (margins && lane == 0) margins[token] = 0.f;
        return;
    }
    // full-softmax denominator (only when not renormalising over the selection)
    double all_sum = 0;
    float row_max = -INFINITY;
    for (uint32_t e = lane; e < experts; e += 32) row_max = fmaxf(row_max, row[e]);
    for (int o = 16; o; o >>= 1) row_max = fmaxf(row_max, __shfl_xor_sync(0xffffffffu, row_max, o));
    if (mode == TSP_ROUTER_SOFTMAX && !normalize) {
        // ascending-id order of additions as in the reference loop, made deterministic by a serial lane-0 pass
        if (lane == 0) for (uint32_t e = 0; e < experts; ++e) all_sum += exp(static_cast<double>(row[e]) - static_cast<double>(row_max));
        all_sum = __shfl_sync(0xffffffffu, all_sum, 0);
    }
    // lane r keeps the logit of rank r (ranks >= 32 in a second slot); the double-precision activations are then
    // evaluated once per rank, in parallel across lanes, instead of once per rank by every lane
    float my_logit = 0.f, my_logit_hi = 0.f;
    for (uint32_t r = 0; r < selected; ++r) {
        float best = -INFINITY;
        uint32_t best_id = 0xffffffffu;
        for (uint32_t e = lane; e < experts; e += 32) {
            const float v = row[e];
            if (v > best) { best = v; best_id = e; }  // ascending scan keeps the lowest id on ties
        }
        for (int o = 16; o; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, best_id, o);
            if (ov > best || (ov == best && oi < best_id)) { best = ov; best_id = oi; }
        }
        if ((r & 31u) == lane) { if (r < 32) my_logit = best; else my_logit_hi = best; }
        if (lane == 0) { out_ids[r] = best_id; row[best_id] = -INFINITY; }
        __syncwarp();
    }
    if (margins) {   // one more round: the best logit among the experts left out
        float next = -INFINITY;
        for (uint32_t e = lane; e < experts; e += 32) next = fmaxf(next, row[e]);
        for (int o = 16; o; o >>= 1) next = fmaxf(next, __shfl_xor_sync(0xffffffffu, next, o));
        const uint32_t last = selected - 1;
        const float last_logit = __shfl_sync(0xffffffffu, last < 32 ? my_logit : my_logit_hi, last & 31u);
        if (lane == 0) margins[token] = selected < experts ? last_logit - next : INFINITY;
    }
    const double mx = row_max;
    auto activate = [&](float logit) -> double {
        const double l = logit;
        if (mode == TSP_ROUTER_SOFTMAX) return exp(l - mx);
        if (normalize) return exp(-softplus_f64(-l) + softplus_f64(-mx));
        return sigmoid_f64(l);
    };
    const double my_act = lane < selected ? activate(my_logit) : 0.0;
    const double my_act_hi = lane + 32 < selected ? activate(my_logit_hi) : 0.0;
    double sel_sum = my_act + my_act_hi;   // fixed butterfly order: deterministic, within an ulp of the rank-order sum
    for (int o = 16; o; o >>= 1) sel_sum += __shfl_xor_sync(0xffffffffu, sel_sum, o);
    double denominator = mode == TSP_ROUTER_SIGMOID ? 1.0 : all_sum;
    if (normalize) denominator = sel_sum;
    if (!(denominator > 0) || isinf(denominator)) {
        if (lane == 0) raise_error(error, TSP_ERR_NONFINITE);
        denominator = 1.0;
    }
    if (lane < selected) out_w[lane] = static_cast<float>(my_act / denominator);
    if (lane + 32 < selected) out_w[lane + 32] = static_cast<float>(my_act_hi / denominator);
}

__global__ void __launch_bounds__(kRouteWarps * 32)
route_kernel(const float* logits, uint64_t stride_bytes, uint32_t tokens, uint32_t experts,
             uint32_t selected, uint32_t mode, int normalize, uint32_t* __restrict__ ids,
             float* __restrict__ weights, uint32_t* error, float* __restrict__ margins) {
    pdl_launch_dependents();
    pdl_wait();

    extern __shared__ float route_smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t token = blockIdx.x * (blockDim.x >> 5) + warp;
    if (token >= tokens) return;
    const float* src = reinterpret_cast<const float*>(reinterpret_cast<const char*>(logits) + token * stride_bytes);
    if (experts <= 512 && normalize && !margins) route_row_regs(src, token, experts, selected, mode, ids, weights, error, lane);
    else route_row(route_smem + warp * experts, src, token, experts, selected, mode, normalize, ids, weights, error, lane, margins);
}

// ---------------------------------------------------------------------------------------------
// permutation: one block per expert compacts, in ascending token order, the routes that name it.
// ---------------------------------------------------------------------------------------------
constexpr int kPermuteThreads = 512;
constexpr uint32_t kPermuteExperts = 2;   // experts per block: a token's ids are read once for all of them

__global__ void __launch_bounds__(kPermuteThreads)
grouped_routes_kernel(const uint32_t* ids, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t first, int local_only,
                      uint32_t* __restrict__ token_map, uint32_t* __restrict__ counts, uint32_t* error) {
    pdl_launch_dependents();
    pdl_wait();

    __shared__ uint32_t totals[kPermuteExperts][kPermuteThreads / 32];
    const uint32_t e0 = blockIdx.x * kPermuteExperts, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t accumulated[kPermuteExperts];
#pragma unroll
    for (uint32_t q = 0; q < kPermuteExperts; ++q) accumulated[q] = 0;
    for (uint32_t base = 0; base < tokens; base += kPermuteThreads) {
        const uint32_t token = base + tid;
        uint32_t slot[kPermuteExperts], matches[kPermuteExperts];
#pragma unroll
        for (uint32_t q = 0; q < kPermuteExperts; ++q) { slot[q] = 0; matches[q] = 0; }
        if (token < tokens) {
            for (uint32_t i = 0; i < selected; ++i) {
                // ids are global; this launch owns experts [first, first + experts). With local_only, routes to other
                // owners are simply not this rank's business; without it they are an index error.
                const uint32_t id = ids[static_cast<uint64_t>(token) * selected + i] - first;
                if (id >= experts && blockIdx.x == 0 && !local_only) raise_error(error, TSP_ERR_INDEX);
#pragma unroll
                for (uint32_t q = 0; q < kPermuteExperts; ++q)
                    if (id == e0 + q) { slot[q] = i; ++matches[q]; }
            }
        }
        uint32_t prefix[kPermuteExperts];
#pragma unroll
        for (uint32_t q = 0; q < kPermuteExperts; ++q) {
            if (matches[q] > 1) raise_error(error, TSP_ERR_INDEX);
            const uint32_t ballot = __ballot_sync(0xffffffffu, matches[q] == 1);
            prefix[q] = __popc(ballot & ((1u << lane) - 1u));
            if (lane == 0) totals[q][warp] = __popc(ballot);
        }
        __syncthreads();
#pragma unroll
        for (uint32_t q = 0; q < kPermuteExperts; ++q) {
            uint32_t before = 0, chunk = 0;
            for (uint32_t i = 0; i < kPermuteThreads / 32; ++i) { if (i < warp) before += totals[q][i]; chunk += totals[q][i]; }
            if (matches[q] == 1 && e0 + q < experts)
                token_map[static_cast<uint64_t>(e0 + q) * tokens + accumulated[q] + before + prefix[q]] = token * selected + slot[q];
            accumulated[q] += chunk;
        }
        __syncthreads();
    }
    if (tid < kPermuteExperts && e0 + tid < experts) {
        uint32_t c = 0;
#pragma unroll
        for (uint32_t q = 0; q < kPermuteExperts; ++q) if (q == tid) c = accumulated[q];
        counts[e0 + tid] = c;
    }
}

// tasks = {live_tiles, routes, (expert, start) pairs in ascending expert order, 0xffffffff padding}
__global__ void __launch_bounds__(256)
grouped_tasks_kernel(const uint32_t* counts, uint32_t tokens, uint32_t experts, uint32_t selected,
                     uint32_t tile, uint32_t bound, int local_only, uint32_t* __restrict__ tasks, uint32_t* error) {
    pdl_launch_dependents();
    pdl_wait();

    extern __shared__ uint32_t offsets[];  // experts + 1
    const uint32_t tid = threadIdx.x;
    __shared__ uint32_t warp_tiles[8], warp_routes[8];
    // block-wide exclusive scan of tiles per expert, in chunks of 256 experts
    uint32_t carry_tiles = 0, carry_routes = 0;
    for (uint32_t base = 0; base < experts; base += 256) {
        const uint32_t e = base + tid;
        uint32_t c = 0, n = 0;
        if (e < experts) {
            c = counts[e];
            if (c > tokens) raise_error(error, TSP_ERR_INDEX);
            n = (min(c, tokens) + tile - 1) / tile;
        }
        uint32_t incl_n = n, incl_c = c;
        const uint32_t lane = tid & 31, warp = tid >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t tn = __shfl_up_sync(0xffffffffu, incl_n, o), tc = __shfl_up_sync(0xffffffffu, incl_c, o);
            if (lane >= static_cast<uint32_t>(o)) { incl_n += tn; incl_c += tc; }
        }
        if (lane == 31) { warp_tiles[warp] = incl_n; warp_routes[warp] = incl_c; }
        __syncthreads();
        uint32_t before_n = 0, total_n = 0, total_c = 0;
        for (uint32_t i = 0; i < 8; ++i) { if (i < warp) before_n += warp_tiles[i]; total_n += warp_tiles[i]; total_c += warp_routes[i]; }
        if (e < experts) offsets[e] = carry_tiles + before_n + incl_n - n;
        carry_tiles += total_n;
        carry_routes += total_c;
        __syncthreads();
    }
    if (tid == 0) {
        offsets[experts] = carry_tiles;
        tasks[0] = min(carry_tiles, bound);
        tasks[1] = carry_routes;
        if (carry_tiles > bound || (!local_only && carry_routes != tokens * selected) || carry_routes > tokens * selected) raise_error(error, TSP_ERR_INDEX);
    }
    for (uint32_t i = tid; i < bound; i += 256) { tasks[2 + 2 * i] = 0xffffffffu; tasks[3 + 2 * i] = 0xffffffffu; }
    __syncthreads();
    for (uint32_t e = tid; e < experts; e += 256) {
        const uint32_t n = (min(counts[e], tokens) + tile - 1) / tile;
        for (uint32_t i = 0; i < n; ++i) {
            const uint32_t at = offsets[e] + i;
            if (at < bound) { tasks[2 + 2 * at] = e; tasks[3 + 2 * at] = i * tile; }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Decode-size prologue of a batch of <= 1024 token rows in TWO launches: (1) routing, one warp per token over as many blocks
// as that takes, with the binary16 -> FP32 copy of the input rows done by the remaining blocks of the same launch (one block
// routing 64 rows alone is bound by its own issue rate: measured 25.7 us); (2) permutation + tile table in one block. The
// tables are the ones the separate kernels above produce, bit for bit: the per-expert token order comes from a bit mask of
// the tokens that name the expert (bit t set = token t routes here), so position = number of lower set bits: no atomics
// decide an order.
// ---------------------------------------------------------------------------------------------
constexpr int kPrologueThreads = 1024;
constexpr int kPrologueRouteWarps = 4;
constexpr uint32_t kPrologueTokens = 1024, kPrologueExperts = 1024;

// DENSE: 0 no dense expert; 1, 2: blocks past the conversion blocks work on the gate / up pair of a dense Q8_0 expert, from FP32 / binary16 rows
constexpr uint32_t kRouteDenseWarps = 8, kTablesDenseWarps = 16;

template <int DENSE>
__global__ void __launch_bounds__(DENSE ? kRouteDenseWarps * 32 : kPrologueRouteWarps * 32)
decode_route_kernel(const float* logits, uint64_t logits_stride, uint32_t tokens, uint32_t experts, uint32_t selected,
                    uint32_t mode, int normalize, uint32_t route_blocks, uint32_t nconv, uint32_t* __restrict__ ids, float* __restrict__ weights,
                    const __half* x16, uint64_t x16_stride, float* __restrict__ x32, uint64_t x32_stride, uint32_t channels,
                    const Q8Rows dense, uint32_t* error) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float pro_smem[];          // [warps][experts] routing rows of the shared-memory form; the dense blocks' weights
    pdl_wait();
    if (DENSE && blockIdx.x >= route_blocks + nconv) {
        q8_rows_block<true, DENSE == 2, kRouteDenseWarps>(dense, blockIdx.x - route_blocks - nconv, reinterpret_cast<uint8_t*>(pro_smem));
        return;
    }
    if (blockIdx.x >= route_blocks) {   // the conversion blocks: binary16 rows -> FP32 rows (exact)
        const uint32_t per_row = channels / 4;   // four values per thread step
        for (uint32_t i = (blockIdx.x - route_blocks) * blockDim.x + threadIdx.x; i < tokens * per_row; i += nconv * blockDim.x) {
            const uint32_t row = i / per_row, c4 = i - row * per_row;
            const uint2 h = *reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(x16) + row * x16_stride + c4 * 8ull);
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&h.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&h.y));
            *reinterpret_cast<float4*>(reinterpret_cast<char*>(x32) + row * x32_stride + c4 * 16ull) = make_float4(a.x, a.y, b.x, b.y);
        }
        return;
    }
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t t = blockIdx.x * kPrologueRouteWarps + warp;
    if ((DENSE && warp >= kPrologueRouteWarps) || t >= tokens) return;
    const float* row = reinterpret_cast<const float*>(reinterpret_cast<const char*>(logits) + t * logits_stride);
    if (experts <= 512 && normalize) route_row_regs(row, t, experts, selected, mode, ids, weights, error, lane);
    else route_row(pro_smem + warp * experts, row, t, experts, selected, mode, normalize, ids, weights, error, lane);
}

// Permutation + tile table of up to 1024 token rows in ONE block: a mask of the rows that name each expert (`words` 32-bit words per
// expert in shared memory), positions = number of lower set bits. ids are global; this launch owns experts [first, first + experts);
// with local_only, routes to other owners are skipped, without it they are an index error.
// DENSE: blocks 1 .. work on the down matrix of a dense Q8_0 expert (512 threads; up to 512 experts, one per thread).
template <bool DENSE>
__global__ void __launch_bounds__(DENSE ? kTablesDenseWarps * 32 : kPrologueThreads)
tables_kernel(const uint32_t* ids, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t tile, uint32_t first, int local_only,
              uint32_t words, uint32_t* __restrict__ token_map, uint32_t* __restrict__ counts, uint32_t* __restrict__ tasks, const Q8Rows dense, uint32_t* error) {
    pdl_launch_dependents();
    // [experts][stride] masks (an odd stride: lanes with different experts and one word index hit different banks), then [experts][stride]
    // running counts of the words before each word. (With a stride of 32 words and a walk over the words per route, 1003 rows took 100 us; 14 us now.)
    extern __shared__ __align__(16) uint32_t tables_mask[];
    if (DENSE && blockIdx.x > 0) {
        pdl_wait();
        q8_rows_block<false, false, kTablesDenseWarps>(dense, blockIdx.x - 1, reinterpret_cast<uint8_t*>(tables_mask));
        return;
    }
    const uint32_t stride = words | 1u;
    uint16_t* const before_word = reinterpret_cast<uint16_t*>(tables_mask + experts * stride);
    __shared__ uint32_t warp_tiles[32], warp_routes[32];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    for (uint32_t i = tid; i < experts * stride; i += blockDim.x) tables_mask[i] = 0u;
    const uint32_t routes = tokens * selected;
    const uint32_t bound = routes / tile + experts;
    pdl_wait();   // the ids come from the previous launch; everything above touched shared memory only
    __syncthreads();
    for (uint32_t i = tid; i < routes; i += blockDim.x) {
        const uint32_t t = i / selected, e = ids[i] - first;
        if (e >= experts) { if (!local_only) raise_error(error, TSP_ERR_INDEX); continue; }
        const uint32_t bit = 1u << (t & 31u);
        if (atomicOr(&tables_mask[e * stride + (t >> 5)], bit) & bit) raise_error(error, TSP_ERR_INDEX);   // an expert named twice by one token
    }
    for (uint32_t i = tid; i < bound; i += blockDim.x) { tasks[2 + 2 * i] = 0xffffffffu; tasks[3 + 2 * i] = 0xffffffffu; }
    __syncthreads();
    // tile table: exclusive scan of tiles per expert over the block (experts <= blockDim.x)
    uint32_t c = 0, n = 0;
    if (tid < experts) {
        for (uint32_t w = 0; w < words; ++w) { before_word[tid * stride + w] = static_cast<uint16_t>(c); c += __popc(tables_mask[tid * stride + w]); }
        n = (c + tile - 1) / tile;
        counts[tid] = c;
    }
    uint32_t incl_n = n, incl_c = c;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t tn = __shfl_up_sync(0xffffffffu, incl_n, o), tc = __shfl_up_sync(0xffffffffu, incl_c, o);
        if (lane >= static_cast<uint32_t>(o)) { incl_n += tn; incl_c += tc; }
    }
    if (lane == 31) { warp_tiles[warp] = incl_n; warp_routes[warp] = incl_c; }
    __syncthreads();   // also orders the padding of the tile table above before the entries below
    for (uint32_t i = tid; i < routes; i += blockDim.x) {
        const uint32_t t = i / selected, e = ids[i] - first;
        if (e >= experts) continue;
        const uint32_t at = e * stride + (t >> 5);
        token_map[static_cast<uint64_t>(e) * tokens + before_word[at] + __popc(tables_mask[at] & ((1u << (t & 31u)) - 1u))] = i;
    }
    uint32_t before = 0, total_n = 0, total_c = 0;
    for (uint32_t i = 0; i < nwarps; ++i) { if (i < warp) before += warp_tiles[i]; total_n += warp_tiles[i]; total_c += warp_routes[i]; }
    if (tid == 0) {
        tasks[0] = min(total_n, bound);
        tasks[1] = total_c;
        if (total_n > bound || (!local_only && total_c != routes) || total_c > routes) raise_error(error, TSP_ERR_INDEX);
    }
    if (tid < experts) {
        const uint32_t at0 = before + incl_n - n;
        for (uint32_t i = 0; i < n; ++i) {
            const uint32_t at = at0 + i;
            if (at < bound) { tasks[2 + 2 * at] = tid; tasks[3 + 2 * at] = i * tile; }
        }
    }
}

// The same tables of larger batches by ONE cluster of eight blocks, each with the masks of an eighth of the rows (whole words): a block counts its
// experts, reads the other blocks' counts through distributed shared memory, and so knows every expert's total, its own first position in each and
// the scan over experts. offsets (optional): first permuted position of every expert, their total, four zeroed counters (tsp_moe_route_offsets).
// Latency of a few round trips whatever the batch. A block per pair of experts that reads all routes took 45 us for 4096 rows of ten (512
// experts) of Zipf loads and 35 us of even ones, the one-block form 14 us for 1003, the scans behind them 6 and 2 us more; 15 and 6.5 us now. Up to 256 rows
// the one block is as fast (257 rows 5.8 / 5.2 us).
constexpr uint32_t kTablesCluster = 8;
__device__ __forceinline__ uint32_t dsmem_u32(const uint32_t* own, uint32_t rank) {   // the word at the same place in another block's shared memory
    uint32_t addr, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(own)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kPrologueThreads)
tables_cluster_kernel(const uint32_t* ids, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t tile, uint32_t first, int local_only,
                      uint32_t words, uint32_t* __restrict__ token_map, uint32_t* __restrict__ counts, uint32_t* __restrict__ tasks, uint32_t* __restrict__ offsets,
                      uint32_t* error) {
    pdl_launch_dependents();
    // [experts] counts of this block, [experts][stride] masks, [experts][stride] running counts of the words before each word, then first positions
    extern __shared__ __align__(16) uint32_t tables_mask[];
    const uint32_t stride = words | 1u;
    uint32_t* const own = tables_mask;
    uint32_t* const mask = own + experts;
    uint32_t* const base = mask + experts * stride;
    uint16_t* const before_word = reinterpret_cast<uint16_t*>(base + experts);
    __shared__ uint32_t warp_tiles[32], warp_routes[32];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5, rank = blockIdx.x;
    for (uint32_t i = tid; i < experts * stride; i += blockDim.x) mask[i] = 0u;
    const uint32_t t0 = rank * words * 32u, t1 = min(tokens, t0 + words * 32u);   // this block's rows
    const uint32_t r0 = t0 * selected, r1 = max(t0, t1) * selected;
    const uint32_t routes = tokens * selected, bound = routes / tile + experts;
    pdl_wait();   // the ids come from the previous launch; everything above touched shared memory only
    __syncthreads();
    for (uint32_t i = r0 + tid; i < r1; i += blockDim.x) {
        const uint32_t t = i / selected - t0, e = ids[i] - first;
        if (e >= experts) { if (!local_only) raise_error(error, TSP_ERR_INDEX); continue; }
        const uint32_t bit = 1u << (t & 31u);
        if (atomicOr(&mask[e * stride + (t >> 5)], bit) & bit) raise_error(error, TSP_ERR_INDEX);   // an expert named twice by one token
    }
    for (uint32_t i = rank * blockDim.x + tid; i < bound; i += kTablesCluster * blockDim.x) { tasks[2 + 2 * i] = 0xffffffffu; tasks[3 + 2 * i] = 0xffffffffu; }
    __syncthreads();
    if (tid < experts) {
        uint32_t c = 0;
        for (uint32_t w = 0; w < words; ++w) { before_word[tid * stride + w] = static_cast<uint16_t>(c); c += __popc(mask[tid * stride + w]); }
        own[tid] = c;
    }
    cluster_sync();   // counts of every block; the padding of the tile table is ordered before the entries below as well
    uint32_t c = 0, n = 0;
    if (tid < experts) {
        uint32_t at = 0;
#pragma unroll
        for (uint32_t q = 0; q < kTablesCluster; ++q) {
            const uint32_t v = dsmem_u32(own + tid, q);
            if (q < rank) at += v;
            c += v;
        }
        base[tid] = at;
        n = (c + tile - 1) / tile;
    }
    uint32_t incl_n = n, incl_c = c;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t tn = __shfl_up_sync(0xffffffffu, incl_n, o), tc = __shfl_up_sync(0xffffffffu, incl_c, o);
        if (lane >= static_cast<uint32_t>(o)) { incl_n += tn; incl_c += tc; }
    }
    if (lane == 31) { warp_tiles[warp] = incl_n; warp_routes[warp] = incl_c; }
    __syncthreads();
    for (uint32_t i = r0 + tid; i < r1; i += blockDim.x) {
        const uint32_t t = i / selected - t0, e = ids[i] - first;
        if (e >= experts) continue;
        const uint32_t at = e * stride + (t >> 5);
        token_map[static_cast<uint64_t>(e) * tokens + base[e] + before_word[at] + __popc(mask[at] & ((1u << (t & 31u)) - 1u))] = i;
    }
    if (rank == 0) {
        uint32_t before_n = 0, total_n = 0, before_c = 0, total_c = 0;
        for (uint32_t i = 0; i < nwarps; ++i) {
            if (i < warp) { before_n += warp_tiles[i]; before_c += warp_routes[i]; }
            total_n += warp_tiles[i]; total_c += warp_routes[i];
        }
        if (tid == 0) {
            tasks[0] = min(total_n, bound);
            tasks[1] = total_c;
            if (total_n > bound || (!local_only && total_c != routes) || total_c > routes) raise_error(error, TSP_ERR_INDEX);
            if (offsets) {
                offsets[experts] = total_c;
                for (uint32_t i = 1; i <= 4; ++i) offsets[experts + i] = 0;
            }
        }
        if (tid < experts) {
            counts[tid] = c;
            if (offsets) offsets[tid] = before_c + incl_c - c;
            const uint32_t at0 = before_n + incl_n - n;
            for (uint32_t i = 0; i < n; ++i) {
                const uint32_t at = at0 + i;
                if (at < bound) { tasks[2 + 2 * at] = tid; tasks[3 + 2 * at] = i * tile; }
            }
        }
    }
    cluster_sync();   // no block leaves while another reads its counts
}

static uint32_t cluster_words(uint32_t tokens) { return ((tokens + kTablesCluster - 1) / kTablesCluster + 31) / 32; }
static size_t cluster_smem(uint32_t tokens, uint32_t experts) { return static_cast<size_t>(experts) * (8u + (cluster_words(tokens) | 1u) * 6u); }
// The running counts are 16 bits: before a block's last word lie at most 32 * (words - 1) rows, so 2048 words at most (few experts leave shared memory for more)
constexpr uint32_t kClusterWords = 2048;
static_assert(32u * (kClusterWords - 1u) <= 0xffffu, "running counts of the cluster's tables");
static bool cluster_fits(uint32_t tokens, uint32_t experts) {
    return tokens > 256 && experts <= static_cast<uint32_t>(kPrologueThreads) && cluster_words(tokens) <= kClusterWords && cluster_smem(tokens, experts) <= 200 * 1024;
}
static int launch_tables_cluster(const uint32_t* ids, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t tile, uint32_t first, int local_only,
                                 uint32_t* token_map, uint32_t* counts, uint32_t* tasks, uint32_t* offsets, uint32_t* error, cudaStream_t st) {
    const size_t smem = cluster_smem(tokens, experts);
    static thread_local SmemAttrCache configured;
    TSP_CUDA(ensure_dynamic_smem(tables_cluster_kernel, configured, smem));
    LaunchCount& count = launch_count();
    ++count.launches;
    if (count.dry) return TSP_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kTablesCluster); cfg.blockDim = dim3(kPrologueThreads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = kTablesCluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    TSP_CUDA(cudaLaunchKernelEx(&cfg, tables_cluster_kernel, ids, tokens, experts, selected, tile, first, local_only, cluster_words(tokens), token_map, counts, tasks,
                                offsets, error));
    return TSP_OK;
}

// The one-block form covers up to 1024 rows and experts whose masks fit 96 KB of shared memory.
static bool tables_fit(uint32_t tokens, uint32_t experts) {
    return tokens >= 1 && tokens <= 1024 && experts <= static_cast<uint32_t>(kPrologueThreads) && static_cast<uint64_t>(experts) * ((tokens + 31) / 32) * 4 <= 96 * 1024;
}
static int launch_tables(const uint32_t* ids, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t tile, uint32_t first, int local_only,
                         uint32_t* token_map, uint32_t* counts, uint32_t* tasks, uint32_t* error, cudaStream_t st, const Q8Rows* dense = nullptr) {
    const uint32_t words = (tokens + 31) / 32;
    const size_t tables = static_cast<size_t>(experts) * (words | 1u) * 6;
    if (dense) {
        const size_t smem = tables > q8_rows_smem(kTablesDenseWarps) ? tables : q8_rows_smem(kTablesDenseWarps);
        static thread_local SmemAttrCache configured;
        TSP_CUDA(ensure_dynamic_smem(tables_kernel<true>, configured, smem));
        TSP_CUDA(launch_pdl(tables_kernel<true>, dim3(1 + dense->blocks), dim3(kTablesDenseWarps * 32), smem, st, ids, tokens, experts, selected, tile, first, local_only,
                            words, token_map, counts, tasks, *dense, error));
        return TSP_OK;
    }
    static thread_local SmemAttrCache configured;
    TSP_CUDA(ensure_dynamic_smem(tables_kernel<false>, configured, tables));
    TSP_CUDA(launch_pdl(tables_kernel<false>, dim3(1), dim3(kPrologueThreads), tables, st, ids, tokens, experts, selected, tile, first, local_only, words, token_map, counts,
                        tasks, Q8Rows{}, error));
    return TSP_OK;
}

// The dense Q8_0 expert of a decode batch in the prologue's launches (gate-up beside the routing, down beside the tables): its geometry, or false
// where the launches do not serve it. The limits: 128 token rows (its matrices are read once per eight rows, in launches of its own once per sixteen:
// Q8_0 layer of 64 / 128 / 192 / 256 rows 287 / 368 / 403 / 438 us, with launches of its own 307 / 376 / 407 / 437) and 512 experts (the tables' block has
// 512 threads then).
constexpr uint32_t kDenseTokens = 128;
static bool plan_dense(DecodeDense& d, uint32_t tokens, uint32_t experts, bool x16) {
    const bool ok = tokens <= kDenseTokens && experts <= kTablesDenseWarps * 32 && d.hidden % 256 == 0 && d.channels % 256 == 0 && aligned16(d.x) && d.x_stride % 16 == 0;
    if (!ok) return false;
    d.x16 = x16;
    d.up = Q8Rows{d.gate_w, d.up_w, d.hidden, d.channels, d.channels / 32 * 34, d.x, d.x_stride, d.h, d.hidden * 4ull, tokens, 1, 0, d.error};
    d.down = Q8Rows{d.down_w, nullptr, d.channels, d.hidden, d.hidden / 32 * 34, d.h, d.hidden * 4ull, d.out, d.channels * 4ull, tokens, 1, 0, d.error};
    q8_rows_plan(d.up, true, kRouteDenseWarps);
    q8_rows_plan(d.down, false, kTablesDenseWarps);
    return true;
}

template <int DENSE>
static int launch_decode_route(dim3 grid, size_t smem, cudaStream_t st, const float* logits, uint64_t logits_stride, uint32_t tokens, uint32_t experts, uint32_t selected,
                               uint32_t mode, int normalize, uint32_t route_blocks, uint32_t conv, uint32_t* ids, float* weights, const void* x16, uint64_t x16_stride,
                               float* x32, uint64_t x32_stride, uint32_t channels, const Q8Rows& dense, uint32_t* error) {
    if (DENSE && smem < q8_rows_smem(kRouteDenseWarps)) smem = q8_rows_smem(kRouteDenseWarps);
    static thread_local SmemAttrCache configured;   // per kernel instantiation, keyed by device
    TSP_CUDA(ensure_dynamic_smem(decode_route_kernel<DENSE>, configured, smem));
    TSP_CUDA(launch_pdl(decode_route_kernel<DENSE>, grid, dim3(DENSE ? kRouteDenseWarps * 32 : kPrologueRouteWarps * 32), smem, st, logits, logits_stride, tokens, experts,
                        selected, mode, normalize, route_blocks, conv, ids, weights, static_cast<const __half*>(x16), x16_stride, x32, x32_stride, channels, dense, error));
    return TSP_OK;
}

// A prefill batch's routing and the binary16 copy of its rows in K order in ONE launch (neither reads the other; one after the other they took
// 25 us of a 4096-row layer, 13 and 5 of 1003 and 160 rows; 11, 8 and 4 now): the first blocks route, a warp per row, the others copy. Register form of the routing only (up to 512 experts,
// renormalised weights); returns 1 for anything else.
constexpr uint32_t kPrefillRouteWarps = 8;
bool prefill_route_fits(uint32_t experts, int normalize) { return experts <= 512 && normalize; }

template <bool IN16>
__global__ void __launch_bounds__(256)
prefill_route_kernel(const float* logits, uint64_t logits_stride, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t mode, uint32_t route_blocks,
                     uint32_t* __restrict__ ids, float* __restrict__ weights, const void* x, uint64_t x_stride, uint32_t cols, __half* __restrict__ xk,
                     uint64_t xk_stride, uint32_t* error) {
    pdl_launch_dependents();
    pdl_wait();
    if (blockIdx.x >= route_blocks) {
        rows_f16k_block<IN16>(x, x_stride, tokens, cols, xk, xk_stride, error, blockIdx.x - route_blocks);
        return;
    }
    const uint32_t t = blockIdx.x * kPrefillRouteWarps + (threadIdx.x >> 5);
    if (t >= tokens) return;
    route_row_regs(reinterpret_cast<const float*>(reinterpret_cast<const char*>(logits) + t * logits_stride), t, experts, selected, mode, ids, weights, error,
                   threadIdx.x & 31u);
}

int launch_prefill_route(const float* logits, uint64_t logits_stride, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t mode, int normalize,
                         uint32_t* ids, float* weights, const void* x, uint64_t x_stride, uint32_t x_dtype, uint32_t cols, void* xk, uint64_t xk_stride,
                         uint32_t* error, cudaStream_t st) {
    if (!prefill_route_fits(experts, normalize)) return 1;
    const uint32_t route_blocks = (tokens + kPrefillRouteWarps - 1) / kPrefillRouteWarps, row_blocks = (tokens + 3) / 4;
    const dim3 grid(route_blocks + row_blocks);
    if (x_dtype == 1)
        TSP_CUDA(launch_pdl(prefill_route_kernel<true>, grid, dim3(256), 0, st, logits, logits_stride, tokens, experts, selected, mode, route_blocks, ids, weights, x,
                            x_stride, cols, static_cast<__half*>(xk), xk_stride, error));
    else
        TSP_CUDA(launch_pdl(prefill_route_kernel<false>, grid, dim3(256), 0, st, logits, logits_stride, tokens, experts, selected, mode, route_blocks, ids, weights, x,
                            x_stride, cols, static_cast<__half*>(xk), xk_stride, error));
    return TSP_OK;
}

// Returns 1 when the batch does not fit the short prologue (the caller then issues the separate launches). dense: a Q8_0 shared expert for these
// launches to work on; dense->done says whether they do.
int launch_decode_prologue(const float* logits, uint64_t logits_stride, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t mode,
                           int normalize, uint32_t tile, uint32_t* ids, float* weights, uint32_t* token_map, uint32_t* counts, uint32_t* tasks,
                           const void* x16, uint64_t x16_stride, float* x32, uint64_t x32_stride, uint32_t channels, DecodeDense* dense, uint32_t* error, cudaStream_t st) {
    if (tokens > kPrologueTokens || experts > kPrologueExperts || !tables_fit(tokens, experts)) return 1;
    if (x16 && (channels % 4 || x16_stride % 8 || x32_stride % 16 || reinterpret_cast<uintptr_t>(x16) % 8 || reinterpret_cast<uintptr_t>(x32) % 16)) return 1;
    const size_t smem = (experts <= 512 && normalize) ? 0 : static_cast<size_t>(kPrologueRouteWarps) * experts * sizeof(float);
    const uint32_t route_blocks = (tokens + kPrologueRouteWarps - 1) / kPrologueRouteWarps;
    // conversion blocks: enough to cover the rows in two passes
    const uint32_t conv = x16 ? min(128u, (tokens * (channels / 4) + 2 * kPrologueRouteWarps * 32 - 1) / (2 * kPrologueRouteWarps * 32)) : 0u;
    const int form = dense && plan_dense(*dense, tokens, experts, x16 != nullptr) ? (x16 ? 2 : 1) : 0;
    const Q8Rows up = form ? dense->up : Q8Rows{};
    const dim3 grid(route_blocks + conv + up.blocks);
#define TSP_ROUTE(D) launch_decode_route<D>(grid, smem, st, logits, logits_stride, tokens, experts, selected, mode, normalize, route_blocks, conv, ids, weights, x16, \
                                            x16_stride, x32, x32_stride, channels, up, error)
    if (int rc = form == 2 ? TSP_ROUTE(2) : form == 1 ? TSP_ROUTE(1) : TSP_ROUTE(0)) return rc;
#undef TSP_ROUTE
    if (int rc = launch_tables(ids, tokens, experts, selected, tile, 0, 0, token_map, counts, tasks, error, st, form ? &dense->down : nullptr)) return rc;
    TSP_CUDA(cudaGetLastError());
    if (dense) dense->done = form != 0;
    return TSP_OK;
}

// ---------------------------------------------------------------------------------------------
// combine: one block per token. Optional shared-router dot (FP32 tree sum), then the mixture in
// route-rank order starting from the gated shared term (routing.cpp:49-58).
// ---------------------------------------------------------------------------------------------
constexpr int kCombineThreads = 256;

// R16: the route rows are binary16 (the prefill path keeps them so); X16: the input rows of the shared-router dot are binary16.
template <bool R16, bool X16>
__global__ void __launch_bounds__(kCombineThreads)
combine_kernel(const void* routed, uint64_t routed_stride, const float* weights,
               const float* shared, uint64_t shared_stride, const float* shared_router,
               const void* x, uint64_t x_stride, float* shared_logit, uint32_t channels,
               uint32_t selected, float* __restrict__ out, uint64_t out_stride, __half* __restrict__ out16,
               uint64_t out16_stride, int vec4, uint32_t* error) {
    pdl_launch_dependents();
    pdl_wait();

    __shared__ float partial[kCombineThreads / 32];
    __shared__ float w_s[64];
    __shared__ float gate_s;
    const uint32_t token = blockIdx.x, tid = threadIdx.x;
    if (tid < selected) w_s[tid] = weights[static_cast<uint64_t>(token) * selected + tid];
    float gate = 1.f;
    if (shared_router) {
        const char* xr = reinterpret_cast<const char*>(x) + token * x_stride;
        float acc = 0.f;
        for (uint32_t c = tid; c < channels; c += kCombineThreads)
            acc = fmaf(shared_router[c], X16 ? __half2float(reinterpret_cast<const __half*>(xr)[c]) : reinterpret_cast<const float*>(xr)[c], acc);
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if ((tid & 31) == 0) partial[tid >> 5] = acc;
        __syncthreads();
        if (tid == 0) {
            float s = 0.f;
            for (int i = 0; i < kCombineThreads / 32; ++i) s += partial[i];
            if (!finite_f32(s)) raise_error(error, TSP_ERR_NONFINITE);
            if (shared_logit && blockIdx.y == 0) shared_logit[token] = s;
            gate_s = stable_sigmoid(s);
        }
        __syncthreads();
        gate = gate_s;
    } else {
        if (shared_logit) gate = stable_sigmoid(shared_logit[token]);
        __syncthreads();
    }
    // shared == nullptr: no shared term (the rows are partial sums that another launch finishes)
    const float* sh = shared ? reinterpret_cast<const float*>(reinterpret_cast<const char*>(shared) + token * shared_stride) : nullptr;
    float* o = reinterpret_cast<float*>(reinterpret_cast<char*>(out) + token * out_stride);
    bool bad = false;
    // gridDim.y slices of the row per token, so that a small batch still fills the machine while a large one does not repeat
    // the gate's dot product more often than needed; four channels per thread (rows are 16-byte aligned)
    const uint32_t per_slice = ((channels + gridDim.y - 1) / gridDim.y + 3u) & ~3u;
    const uint32_t c_end = min(channels, (blockIdx.y + 1) * per_slice);
    const char* y0 = reinterpret_cast<const char*>(routed) + static_cast<uint64_t>(token) * selected * routed_stride;
    if (R16 && vec4 == 2 && (channels & 7u) == 0 && gridDim.y == 1) {   // vec4 == 2: every row of every buffer starts on a 16-byte boundary
        // binary16 route rows (prefill): eight channels per thread step, one 16-byte load per route row, five rows in flight
        for (uint32_t c = tid * 8; c < channels; c += kCombineThreads * 8) {
            float v[8];
            if (sh) {
                const float4 a = *reinterpret_cast<const float4*>(sh + c), b = *reinterpret_cast<const float4*>(sh + c + 4);
                v[0] = gate * a.x; v[1] = gate * a.y; v[2] = gate * a.z; v[3] = gate * a.w; v[4] = gate * b.x; v[5] = gate * b.y; v[6] = gate * b.z; v[7] = gate * b.w;
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = 0.f;
            }
            for (uint32_t r0 = 0; r0 < selected; r0 += 5) {
                uint4 y[5];
#pragma unroll
                for (uint32_t i = 0; i < 5; ++i) y[i] = *reinterpret_cast<const uint4*>(y0 + min(r0 + i, selected - 1) * routed_stride + c * 2ull);
#pragma unroll
                for (uint32_t i = 0; i < 5; ++i) {
                    const float wr = r0 + i < selected ? w_s[r0 + i] : 0.f;
                    if (wr != 0.f) {
                        const uint32_t w4[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w4[q]));
                            v[2 * q] = fmaf(wr, f.x, v[2 * q]); v[2 * q + 1] = fmaf(wr, f.y, v[2 * q + 1]);
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) bad |= !finite_f32(v[i]);
            if (out) { *reinterpret_cast<float4*>(o + c) = make_float4(v[0], v[1], v[2], v[3]); *reinterpret_cast<float4*>(o + c + 4) = make_float4(v[4], v[5], v[6], v[7]); }
            if (out16) {
                uint32_t h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) { const __half2 t2 = __floats2half2_rn(v[2 * q], v[2 * q + 1]); h[q] = *reinterpret_cast<const uint32_t*>(&t2); }
                *reinterpret_cast<uint4*>(reinterpret_cast<char*>(out16) + token * out16_stride + c * 2ull) = make_uint4(h[0], h[1], h[2], h[3]);
            }
        }
        if (bad) raise_error(error, TSP_ERR_NONFINITE);
        return;
    }
    for (uint32_t c = blockIdx.y * per_slice + tid * 4; c < c_end; c += kCombineThreads * 4) {
        if (vec4 && c + 4 <= c_end) {
            const float4 s4 = sh ? *reinterpret_cast<const float4*>(sh + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            float v[4] = {gate * s4.x, gate * s4.y, gate * s4.z, gate * s4.w};
            // A zero weight marks a route that is not present in `routed` (expert parallelism): its row is still inside the
            // buffer, so it is loaded like the others (four rows in flight) and only the sum skips it.
            for (uint32_t r0 = 0; r0 < selected; r0 += 4) {
                float4 y[4];
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const uint32_t r = min(r0 + i, selected - 1);
                    if (R16) {
                        const uint2 h = *reinterpret_cast<const uint2*>(y0 + r * routed_stride + c * 2ull);
                        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&h.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&h.y));
                        y[i] = make_float4(a.x, a.y, b.x, b.y);
                    } else {
                        y[i] = *reinterpret_cast<const float4*>(y0 + r * routed_stride + c * 4ull);
                    }
                }
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const float wr = r0 + i < selected ? w_s[r0 + i] : 0.f;
                    if (wr != 0.f) { v[0] = fmaf(wr, y[i].x, v[0]); v[1] = fmaf(wr, y[i].y, v[1]); v[2] = fmaf(wr, y[i].z, v[2]); v[3] = fmaf(wr, y[i].w, v[3]); }
                }
            }
            bad |= !finite_f32(v[0]) | !finite_f32(v[1]) | !finite_f32(v[2]) | !finite_f32(v[3]);
            if (out) *reinterpret_cast<float4*>(o + c) = make_float4(v[0], v[1], v[2], v[3]);
            if (out16) {
                const __half2 h0 = __floats2half2_rn(v[0], v[1]), h1 = __floats2half2_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(reinterpret_cast<char*>(out16) + token * out16_stride + c * 2ull) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
            }
        } else {
            for (uint32_t cc = c; cc < min(c + 4, c_end); ++cc) {   // a row tail shorter than four channels, or rows that are not 16-byte aligned
                float v = sh ? gate * sh[cc] : 0.f;
                for (uint32_t r = 0; r < selected; ++r)
                    if (w_s[r] != 0.f) {
                        const char* yr = y0 + r * routed_stride;
                        v = fmaf(w_s[r], R16 ? __half2float(reinterpret_cast<const __half*>(yr)[cc]) : reinterpret_cast<const float*>(yr)[cc], v);
                    }
                bad |= !finite_f32(v);
                if (out) o[cc] = v;
                if (out16) reinterpret_cast<__half*>(reinterpret_cast<char*>(out16) + token * out16_stride)[cc] = __float2half_rn(v);
            }
        }
    }
    if (bad) raise_error(error, TSP_ERR_NONFINITE);
}

// ---------------------------------------------------------------------------------------------
// F32 matrix-vector product for the router projections: one warp per (matrix row, token), FP32 FMA + tree sum (f32_dot_row). `extra`
// (optional): one more matrix row with an output array of its own, the last row of every token.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
gemv_f32_kernel(const float* w, uint32_t rows, uint32_t cols, const float* extra, const float* x, uint64_t x_stride, uint32_t tokens,
                float* __restrict__ out, uint64_t out_stride, float* __restrict__ extra_out, uint32_t* error) {
    pdl_launch_dependents();
    pdl_wait();

    const uint32_t warp = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31, all = rows + (extra ? 1u : 0u);   // threads exceed 32 bits from 2^27 outputs on
    if (warp >= all * tokens) return;
    const uint32_t token = warp / all, row = warp % all;
    const float acc = f32_dot_row(row < rows ? w + static_cast<uint64_t>(row) * cols : extra,
                                  reinterpret_cast<const float*>(reinterpret_cast<const char*>(x) + token * x_stride), cols, lane);
    if (lane == 0) {
        if (!finite_f32(acc)) raise_error(error, TSP_ERR_NONFINITE);
        if (row < rows) reinterpret_cast<float*>(reinterpret_cast<char*>(out) + token * out_stride)[row] = acc;
        else extra_out[token] = acc;
    }
}

int launch_router_mma(const float*, uint32_t, uint32_t, const float*, const float*, uint64_t, uint32_t, float*, uint64_t, float*, uint32_t*, cudaStream_t);
// Fewest token rows for the tensor-core product, from 512 matrix rows: its one wave of blocks takes 18 us at 1024 columns and 28 us at 2048
// whatever the batch; one warp per output takes 15 us at 63 rows of 1024 columns, 20 us at 64 and 28 us at 95 rows of 2048. The warp form scales
// with matrix rows x token rows (64 matrix rows: 8 us at 95 token rows of 2048 columns), the other does not (28 us at 96), so a matrix of fewer
// rows would change over later: about 48 k outputs.
constexpr uint32_t kRouterMmaTokens = 96;

int launch_gemv_f32(const float* w, uint32_t rows, uint32_t cols, const float* extra, const float* x, uint64_t x_stride, uint32_t tokens, float* out,
                    uint64_t out_stride, float* extra_out, uint32_t* error, cudaStream_t st) {
    if (tokens >= kRouterMmaTokens) return launch_router_mma(w, rows, cols, extra, x, x_stride, tokens, out, out_stride, extra_out, error, st);
    const uint64_t warps = (static_cast<uint64_t>(rows) + (extra ? 1u : 0u)) * tokens;
    TSP_CUDA(launch_pdl(gemv_f32_kernel, dim3(static_cast<unsigned>((warps + 7) / 8)), dim3(256), 0, st, w, rows, cols, extra, x, x_stride, tokens, out, out_stride, extra_out,
                        error));
    return TSP_OK;
}

__global__ void rows_f16_to_f32_kernel(const __half* in, uint64_t in_stride, float* __restrict__ out,
                                       uint64_t out_stride, uint32_t rows, uint32_t cols) {
    pdl_launch_dependents();
    pdl_wait();

    const uint32_t row = blockIdx.y;
    const __half* src = reinterpret_cast<const __half*>(reinterpret_cast<const char*>(in) + row * in_stride);
    float* dst = reinterpret_cast<float*>(reinterpret_cast<char*>(out) + row * out_stride);
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x) dst[c] = __half2float(src[c]);
}

// ---------------------------------------------------------------------------------------------
// dequantise test hook: FP32 fmaf(d*sc, q, -(dmin*mn)) is the exactly rounded reference value
// because d*sc, (d*sc)*q and dmin*mn are exact in FP32 (at most 21 significant bits).
// ---------------------------------------------------------------------------------------------
__global__ void dequant_q4k_kernel(const uint8_t* expert, uint32_t layout, uint64_t total_blocks,
                                   float* __restrict__ out, uint32_t* error) {
    const uint64_t blk = blockIdx.x;
    const uint32_t i = threadIdx.x;  // 0..255
    const uint32_t g = i >> 5;
    uint32_t dbits, mbits, sc, mn, q;
    if (layout == TSP_LAYOUT_GGUF) {
        const uint8_t* b = expert + blk * 144;
        dbits = b[0] | (b[1] << 8);
        mbits = b[2] | (b[3] << 8);
        if (g < 4) { sc = b[4 + g] & 63u; mn = b[8 + g] & 63u; }
        else { sc = (b[12 + g - 4] & 15u) | ((b[4 + g - 4] >> 6) << 4); mn = (b[12 + g - 4] >> 4) | ((b[8 + g - 4] >> 6) << 4); }
        q = (b[16 + (i >> 6) * 32 + (i & 31)] >> (4 * ((i >> 5) & 1))) & 15u;
    } else {
        const uint8_t* qs = expert + blk * 128;
        const uint8_t* sm = expert + total_blocks * 128 + blk * 16;
        const uint8_t* dm = expert + total_blocks * 144 + blk * 4;
        dbits = dm[0] | (dm[1] << 8);
        mbits = dm[2] | (dm[3] << 8);
        sc = sm[g]; mn = sm[8 + g];
        if ((sc | mn) & 0xc0u) raise_error(error, TSP_ERR_INDEX);
        q = (qs[(i >> 6) * 32 + (i & 31)] >> (4 * ((i >> 5) & 1))) & 15u;
    }
    const float d = half_bits_to_float(dbits), dmin = half_bits_to_float(mbits);
    const float v = fmaf(d * static_cast<float>(sc), static_cast<float>(q), -(dmin * static_cast<float>(mn)));
    if (!finite_f32(v) || !finite_f32(d) || !finite_f32(dmin)) raise_error(error, TSP_ERR_NONFINITE);
    out[blk * 256 + i] = v;
}

__global__ void dequant_q8_kernel(const uint8_t* expert, uint32_t layout, uint64_t total_blocks,
                                  float* __restrict__ out, uint32_t* error) {
    const uint64_t blk = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (blk >= total_blocks) return;
    const uint32_t i = threadIdx.x & 31;
    uint32_t dbits;
    int q;
    if (layout == TSP_LAYOUT_GGUF) {
        const uint8_t* b = expert + blk * 34;
        dbits = b[0] | (b[1] << 8);
        q = static_cast<int8_t>(b[2 + i]);
    } else {
        const uint8_t* dm = expert + total_blocks * 32 + blk * 2;
        dbits = dm[0] | (dm[1] << 8);
        q = static_cast<int8_t>(expert[blk * 32 + i]);
    }
    const float d = half_bits_to_float(dbits);
    const float v = d * static_cast<float>(q);
    if (!finite_f32(v)) raise_error(error, TSP_ERR_NONFINITE);
    out[blk * 32 + i] = v;
}

// ---------------------------------------------------------------------------------------------
// host launchers (called by the C ABI layer in tsp_api.cu after validation)
// ---------------------------------------------------------------------------------------------
int launch_route(const float* logits, uint64_t stride, uint32_t tokens, uint32_t experts, uint32_t selected,
                 uint32_t mode, int normalize, uint32_t* ids, float* weights, uint32_t* error, cudaStream_t st, float* margins) {
    const uint32_t warps = experts > 3072 ? 2 : kRouteWarps;
    const uint32_t blocks = (tokens + warps - 1) / warps;
    TSP_CUDA(launch_pdl(route_kernel, dim3(blocks), dim3(warps * 32), warps * experts * sizeof(float), st, logits, stride, tokens, experts, selected, mode, normalize, ids, weights, error, margins));
    TSP_CUDA(cudaGetLastError());
    return TSP_OK;
}

int launch_route_offsets(const uint32_t*, uint32_t, uint32_t*, cudaStream_t);

// offsets (optional): the first permuted position of every expert and the grouped launches' counters, as launch_route_offsets writes them
int launch_permute(const uint32_t* ids, uint32_t tokens, uint32_t experts, uint32_t selected, uint32_t tile, uint32_t first, int local_only,
                   uint32_t* token_map, uint32_t* counts, uint32_t* tasks, uint32_t* error, cudaStream_t st, uint32_t* offsets) {
    const uint32_t bound = static_cast<uint32_t>((static_cast<uint64_t>(tokens) * selected) / tile + experts);
    // the cluster reads the ids until its last writes; the launches below have read them before they write tile table and offsets
    const uint64_t id_bytes = static_cast<uint64_t>(tokens) * selected * 4;
    const bool ids_apart = !overlap(ids, id_bytes, tasks, 8 + bound * 8ull) && !(offsets && overlap(ids, id_bytes, offsets, (experts + 5) * 4ull));
    // Tables of few routes alone: the one block is level up to about 1100 routes, or 640 rows of one expert each (300 rows, two of 8 experts: 3.5 us, cluster
    // 4.3; 300 rows, four of 64: 4.4 and 4.3; 512 rows, two of 8: 4.0 and 4.4; 1003 rows of one expert: 6.8 and 6.2). With offsets the cluster saves a launch.
    const bool cluster = offsets || tokens >= 640 || static_cast<uint64_t>(tokens) * selected >= 1100;
    if (cluster && ids_apart && cluster_fits(tokens, experts))
        return launch_tables_cluster(ids, tokens, experts, selected, tile, first, local_only, token_map, counts, tasks, offsets, error, st);
    if (tables_fit(tokens, experts)) {
        if (int rc = launch_tables(ids, tokens, experts, selected, tile, first, local_only, token_map, counts, tasks, error, st)) return rc;
        return offsets ? launch_route_offsets(counts, experts, offsets, st) : TSP_OK;
    }
    TSP_CUDA(launch_pdl(grouped_routes_kernel, dim3((experts + kPermuteExperts - 1) / kPermuteExperts), dim3(kPermuteThreads), 0, st, ids, tokens, experts, selected, first, local_only, token_map, counts, error));
    TSP_CUDA(cudaGetLastError());
    TSP_CUDA(launch_pdl(grouped_tasks_kernel, dim3(1), dim3(256), (experts + 1) * sizeof(uint32_t), st, counts, tokens, experts, selected, tile, bound, local_only, tasks, error));
    TSP_CUDA(cudaGetLastError());
    return offsets ? launch_route_offsets(counts, experts, offsets, st) : TSP_OK;
}

// launches of launch_permute with offsets, the ids in memory of their own
uint32_t permute_launches(uint32_t tokens, uint32_t experts) { return cluster_fits(tokens, experts) ? 1u : tables_fit(tokens, experts) ? 2u : 3u; }

int launch_combine(const void* routed, uint64_t routed_stride, uint32_t routed_f16, const float* weights, const float* shared,
                   uint64_t shared_stride, const float* shared_router, const void* x, uint64_t x_stride, uint32_t x_f16,
                   float* shared_logit, uint32_t tokens, uint32_t channels, uint32_t selected, float* out,
                   uint64_t out_stride, void* out16, uint64_t out16_stride, uint32_t* error, cudaStream_t st) {
    // about four CTAs per SM in total: 8 slices of a 2048-wide row at 64 tokens, one slice from a few hundred tokens on
    uint32_t slices = (channels + kCombineThreads - 1) / kCombineThreads;
    const uint32_t want = (4u * 148u + tokens - 1) / tokens;
    if (slices > want) slices = want;
    // output rows in the input rows (each its own): a block reads the whole row for the shared router before it writes, so one block per row
    const uint64_t x_row = channels * (x_f16 ? 2ull : 4ull);
    if (shared_router && ((out && rows_overlap(x, x_stride, x_row, out, out_stride, channels * 4ull, tokens)) ||
                          (out16 && rows_overlap(x, x_stride, x_row, out16, out16_stride, channels * 2ull, tokens)))) slices = 1;
    auto a16 = [](const void* p, uint64_t stride) { return (reinterpret_cast<uintptr_t>(p) | stride) % 16 == 0; };
    const int vec4 = (routed_f16 ? (reinterpret_cast<uintptr_t>(routed) | routed_stride) % 8 == 0 : a16(routed, routed_stride)) && (!shared || a16(shared, shared_stride)) &&
                     (!out || a16(out, out_stride)) && (!out16 || (reinterpret_cast<uintptr_t>(out16) | out16_stride) % 8 == 0);
    const int vec8 = vec4 && routed_f16 && a16(routed, routed_stride) && (!out16 || a16(out16, out16_stride));
    const dim3 grid(tokens, slices), block(kCombineThreads);
#define TSP_COMBINE(R, X) TSP_CUDA(launch_pdl(combine_kernel<R, X>, grid, block, 0, st, routed, routed_stride, weights, shared, shared_stride, shared_router, \
                                              x, x_stride, shared_logit, channels, selected, out, out_stride, static_cast<__half*>(out16), out16_stride, vec8 ? 2 : vec4, error))
    if (routed_f16) { if (x_f16) TSP_COMBINE(true, true); else TSP_COMBINE(true, false); }
    else { if (x_f16) TSP_COMBINE(false, true); else TSP_COMBINE(false, false); }
#undef TSP_COMBINE
    TSP_CUDA(cudaGetLastError());
    return TSP_OK;
}

// One thread waits on a barrier that nothing ever arrives on, with a small poll limit: the wait gives up, the kernel reports
// TSP_ERR_TIMEOUT through the error word and returns normally. This is the path every bounded wait of the library takes when
// an arrival is lost; it is exercised here without making any real pipeline misbehave.
__global__ void bounded_wait_selftest_kernel(uint32_t polls, uint32_t* error) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
    __syncthreads();
    if (threadIdx.x == 0 && !mbar_wait(&bar, 0, polls)) raise_error(error, TSP_ERR_TIMEOUT);
}

int launch_bounded_wait_selftest(uint32_t polls, uint32_t* error, cudaStream_t st) {
    bounded_wait_selftest_kernel<<<1, 32, 0, st>>>(polls, error);
    TSP_CUDA(cudaGetLastError());
    return TSP_OK;
}

int launch_f16_to_f32(const void* in, uint64_t in_stride, float* out, uint64_t out_stride, uint32_t rows, uint32_t cols,
                      cudaStream_t st) {
    dim3 grid((cols + 1023) / 1024, rows);
    TSP_CUDA(launch_pdl(rows_f16_to_f32_kernel, grid, dim3(256), 0, st, static_cast<const __half*>(in), in_stride, out, out_stride, rows, cols));
    return TSP_OK;
}

int launch_dequant(uint32_t type, uint32_t layout, const uint8_t* expert, uint64_t total_blocks, float* out,
                   uint32_t* error, cudaStream_t st) {
    if (type == TSP_TYPE_Q4_K) dequant_q4k_kernel<<<static_cast<unsigned>(total_blocks), 256, 0, st>>>(expert, layout, total_blocks, out, error);
    else dequant_q8_kernel<<<static_cast<unsigned>((total_blocks + 7) / 8), 256, 0, st>>>(expert, layout, total_blocks, out, error);
    TSP_CUDA(cudaGetLastError());
    return TSP_OK;
}

}  // namespace tsp
