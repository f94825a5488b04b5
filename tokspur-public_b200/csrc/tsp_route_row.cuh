// Router top-k of one token row by one warp, with the row's logits in registers.
#pragma once

#include "tsp_common.cuh"

namespace tsp {

__device__ __forceinline__ double softplus_f64(double v) { return fmax(v, 0.0) + log1p(exp(-fabs(v))); }
__device__ __forceinline__ double sigmoid_f64(double v) {
    if (v >= 0) return 1.0 / (1.0 + exp(-v));
    const double p = exp(v);
    return p / (1.0 + p);
}

// The same selection for rows of at most 512 logits kept in registers (expert e = lane + 32 i in slot i), used where one block
// routes a whole decode batch: about a fifth of the instructions of the shared-memory form. Same total order (value descending,
// id ascending), same double-precision weights. Full-softmax weights without renormalisation need the serial ascending-id sum
// and stay with route_row. weights: null where only the ids are wanted.
__device__ __forceinline__ void route_row_regs(const float* src, uint32_t token, uint32_t experts, uint32_t selected,
                                               uint32_t mode, uint32_t* __restrict__ ids, float* __restrict__ weights, uint32_t* error,
                                               uint32_t lane) {
    // Order-preserving 32-bit images (-0 counted as +0: equal logits tie by id), 0 = no expert or already taken. A round is one max over
    // the lane's 16 images, one warp-wide max and one warp-wide min over the ids that reach it: two reductions instead of ten shuffles.
    uint32_t k[16];
    bool bad = false;
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) {
        const uint32_t e = lane + 32 * i;
        const float f = e < experts ? src[e] : 0.f;
        bad |= !finite_f32(f);
        const uint32_t u = f == 0.f ? 0u : __float_as_uint(f);
        k[i] = e < experts ? ((u & 0x80000000u) ? ~u : (u | 0x80000000u)) : 0u;
    }
    auto lane_max = [&]() {
        uint32_t m[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) m[i] = max(k[i], k[i + 8]);
#pragma unroll
        for (int o = 4; o; o >>= 1)
#pragma unroll
            for (int i = 0; i < o; ++i) m[i] = max(m[i], m[i + o]);
        return m[0];
    };
    auto value = [](uint32_t image) { return __uint_as_float((image & 0x80000000u) ? image ^ 0x80000000u : ~image); };
    bad = __any_sync(0xffffffffu, bad);
    uint32_t* out_ids = ids + static_cast<uint64_t>(token) * selected;
    float* out_w = weights + static_cast<uint64_t>(token) * selected;
    if (bad) {
        if (lane == 0) raise_error(error, TSP_ERR_NONFINITE);
        for (uint32_t r = lane; r < selected; r += 32) { out_ids[r] = r; if (weights) out_w[r] = 0.f; }
        return;
    }
    float row_max = 0.f;
    float my_logit = 0.f, my_logit_hi = 0.f;   // the logits of ranks lane and lane + 32
    // Nine to 32 selected: the selected-th largest of the lanes' maxima is a lower bound of the selected-th largest logit, and what reaches it, a dozen
    // of 512 where ten are wanted, is ranked by counting, a lane per candidate. One after another (below; also where many logits are equal) takes 0.14 us
    // each: launches of one row of 512 logits 1.6 / 2.0 / 2.6 / 2.9 / 3.7 us for 1 / 4 / 8 / 10 / 16 selected, ranked 2.2 / 2.3 / 2.8 / 2.8 / 3.4 us. (1024 rows
    // 5.5 / 6.3 us for 8 / 10 and 6.3 / 7.0 us ranked; in the launches of a prefill layer, whose other blocks copy rows, ranking ten is the faster by 2 us of 1003.)
    uint32_t candidates = 0xffffffffu, bound = 1u;
    if (selected > 8 && selected <= 32) {
        const uint32_t m = lane_max();
        uint32_t rank = 0;
#pragma unroll
        for (uint32_t j = 0; j < 32; ++j) { const uint32_t o = __shfl_sync(0xffffffffu, m, j); rank += o > m || (o == m && j < lane); }
        bound = max(__shfl_sync(0xffffffffu, m, __ffs(__ballot_sync(0xffffffffu, rank == selected - 1u)) - 1), 1u);   // 0 marks an empty slot
        uint32_t n = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) n += k[i] >= bound;
        candidates = __reduce_add_sync(0xffffffffu, n);
    }
    if (candidates <= 32) {   // uniform
        uint32_t key = 0, id = 0, n = 0;   // this lane's candidate
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i)
            for (uint32_t votes = __ballot_sync(0xffffffffu, k[i] >= bound); votes; votes &= votes - 1u, ++n) {
                const uint32_t from = __ffs(votes) - 1, v = __shfl_sync(0xffffffffu, k[i], from);
                if (lane == n) { key = v; id = from + 32 * i; }
            }
        uint32_t rank = 0;
        for (uint32_t j = 0; j < n; ++j) {
            const uint32_t ok = __shfl_sync(0xffffffffu, key, j), oi = __shfl_sync(0xffffffffu, id, j);
            rank += ok > key || (ok == key && oi < id);
        }
        if (lane < n && rank < selected) out_ids[rank] = id;
        if (weights) {
            for (uint32_t j = 0; j < n; ++j) {
                const uint32_t r = __shfl_sync(0xffffffffu, rank, j);
                const float v = value(__shfl_sync(0xffffffffu, key, j));
                if (r == 0) row_max = v;
                if (r == lane && r < selected) my_logit = v;
            }
        }
    } else {
        for (uint32_t r = 0; r < selected; ++r) {
            const uint32_t top = __reduce_max_sync(0xffffffffu, lane_max());
            uint32_t mine = 0xffffffffu;
    #pragma unroll
            for (int i = 15; i >= 0; --i) if (k[i] == top) mine = lane + 32 * i;   // the lane's lowest id
            const uint32_t best_id = __reduce_min_sync(0xffffffffu, mine);
            const float best = value(top);
            if (r == 0) row_max = best;
            if ((r & 31u) == lane) { if (r < 32) my_logit = best; else my_logit_hi = best; }
            if (lane == 0) out_ids[r] = best_id;
            if (mine == best_id) {
    #pragma unroll
                for (uint32_t i = 0; i < 16; ++i) if ((best_id >> 5) == i) k[i] = 0u;
            }
        }
    }
    if (!weights) return;
    const double mx = row_max;
    auto activate = [&](float logit) -> double {
        const double l = logit;
        if (mode == TSP_ROUTER_SOFTMAX) return exp(l - mx);
        return exp(-softplus_f64(-l) + softplus_f64(-mx));
    };
    const double my_act = lane < selected ? activate(my_logit) : 0.0;
    const double my_act_hi = lane + 32 < selected ? activate(my_logit_hi) : 0.0;
    double denominator = my_act + my_act_hi;   // renormalised over the selection: same butterfly order as route_row
    for (int o = 16; o; o >>= 1) denominator += __shfl_xor_sync(0xffffffffu, denominator, o);
    if (!(denominator > 0) || isinf(denominator)) {
        if (lane == 0) raise_error(error, TSP_ERR_NONFINITE);
        denominator = 1.0;
    }
    if (lane < selected) out_w[lane] = static_cast<float>(my_act / denominator);
    if (lane + 32 < selected) out_w[lane + 32] = static_cast<float>(my_act_hi / denominator);
}

}  // namespace tsp
