// Expert selection by one warp (src/compute/forward.zig:516-571, src/shaders/softmax_topk.comp:49-81), as the routing kernels share it.
#pragma once

#include "common.cuh"

namespace zc {
namespace {

struct ValIdx {
    float v;
    uint32_t i;
};
__device__ __forceinline__ ValIdx better(ValIdx a, ValIdx b) {
    return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}

// Order-preserving map of (non-NaN) floats to unsigned integers and back; -0 and +0 share a key.
__device__ __forceinline__ uint32_t float_key(float v) {
    const uint32_t b = __float_as_uint(v + 0.0f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// One warp selects for one token: lane l holds experts l, l + 32, ... in registers. Ids go to o[0..k), weights (f32 bits) to o[wofs .. wofs + k): wofs = k is the
// reference's layout, a larger wofs leaves room for slots behind the selected ones. The logits are read past
// L1 (they may have been written by other CTAs of the same launch).
// Where the selection takes its logits from, in two steps so that all of a lane's reads are in flight before any
// of them is waited for: first(i) issues the read, value(i, q) completes it.
struct LogitsPlain {  // logits in global memory, read past L1
    const float* lg;
    __device__ __forceinline__ uint2 first(uint32_t i) const { return make_uint2(__float_as_uint(__ldcg(lg + i)), 1u); }
    __device__ __forceinline__ float value(uint32_t, uint2 q) const { return __uint_as_float(q.x); }
};

template <int VPL, typename Load>
__device__ __forceinline__ void softmax_topk_warp(const Load& load, const float* __restrict__ bias, uint32_t* o,
                                                  uint32_t n, uint32_t k, uint32_t rule, uint32_t wofs, int lane,
                                                  uint32_t* my_id = nullptr, uint32_t* my_w = nullptr) {
    const float floor_v = rule == 0u ? -1.0f : -INFINITY;
    const float gone = rule == 0u ? -2.0f : -INFINITY;  // never selected (again)

    float v[VPL];
    uint2 raw[VPL];
    float lmax = -INFINITY;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        const uint32_t i = lane + 32 * j;
        raw[j] = i < n ? load.first(i) : make_uint2(0xFF800000u, 1u);
    }
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        const uint32_t i = lane + 32 * j;
        v[j] = i < n ? load.value(i, raw[j]) : -INFINITY;
    }
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        const uint32_t i = lane + 32 * j;
        if (bias && i < n) v[j] += bias[i];
        lmax = fmaxf(lmax, v[j]);
    }
    if (rule == 0u) {  // softmax over all experts first
        for (int o2 = 16; o2 > 0; o2 >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xFFFFFFFFu, lmax, o2));
        float lsum = 0.f;
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            const uint32_t i = lane + 32 * j;
            v[j] = i < n ? expf(v[j] - lmax) : 0.f;
            lsum += v[j];
        }
        const float sum = warp_sum(lsum);
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            const uint32_t i = lane + 32 * j;
            if (sum > 0.f) v[j] = v[j] / sum;
            if (i >= n) v[j] = gone;
        }
    }
    const float v0 = __shfl_sync(0xFFFFFFFFu, v[0], 0);  // expert 0, for the "nothing above the floor" case
    // Up to 32 selections stay in registers (selection ki in lane ki) and reach memory once, at the end: a
    // round trip through global memory per selection and per weight costs more than the whole selection.
    const bool in_regs = k <= 32;
    float sel_v = 0.f;
    uint32_t sel_i = 0u;
    for (uint32_t ki = 0; ki < k; ++ki) {
        ValIdx best{floor_v, 0u};
#pragma unroll
        for (int j = 0; j < VPL; ++j)
            if (v[j] > best.v) best = ValIdx{v[j], (uint32_t)(lane + 32 * j)};
        // arg-max over the warp with two integer reductions: the largest value (as an order-preserving key, -0
        // folded into +0), then the lowest index among the lanes that hold it
        const uint32_t kmax = __reduce_max_sync(0xFFFFFFFFu, float_key(best.v));
        const uint32_t imin = __reduce_min_sync(0xFFFFFFFFu, float_key(best.v) == kmax ? best.i : 0xFFFFFFFFu);
        best = ValIdx{key_float(kmax), imin};
        if (!(best.v > floor_v)) best = ValIdx{rule == 0u ? floor_v : v0, 0u};
        if (in_regs) {
            if ((uint32_t)lane == ki) {
                sel_v = best.v;
                sel_i = best.i;
            }
        } else if (lane == 0) {
            o[ki] = best.i;
            o[wofs + ki] = __float_as_uint(best.v);
        }
#pragma unroll
        for (int j = 0; j < VPL; ++j)
            if (best.i == (uint32_t)(lane + 32 * j)) v[j] = gone;
    }
    if (in_regs) {
        // the sums run over the selections in order, as the sequential loops of the reference do
        float w;
        if (rule == 0u) {
            float ws = 0.f;
            for (uint32_t i = 0; i < k; ++i) ws += __shfl_sync(0xFFFFFFFFu, sel_v, (int)i);
            w = ws > 0.f ? sel_v / ws : sel_v;
        } else {
            float mx = (uint32_t)lane < k ? sel_v : -INFINITY;
            for (int o2 = 16; o2 > 0; o2 >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o2));
            const float e = expf(sel_v - mx);
            float sum = 0.f;
            for (uint32_t i = 0; i < k; ++i) sum += __shfl_sync(0xFFFFFFFFu, e, (int)i);
            w = sum > 0.f ? e / sum : e;
        }
        if ((uint32_t)lane < k) {
            o[lane] = sel_i;
            o[wofs + lane] = __float_as_uint(w);
        }
        if (my_id) {  // lane ki's selection, for a caller that goes on with it
            *my_id = sel_i;
            *my_w = __float_as_uint(w);
        }
        return;
    }
    if (lane == 0) {
        if (rule == 0u) {
            float ws = 0.f;
            for (uint32_t i = 0; i < k; ++i) ws += __uint_as_float(o[wofs + i]);
            if (ws > 0.f)
                for (uint32_t i = 0; i < k; ++i) o[wofs + i] = __float_as_uint(__uint_as_float(o[wofs + i]) / ws);
        } else {
            float mx = -INFINITY;
            for (uint32_t i = 0; i < k; ++i) mx = fmaxf(mx, __uint_as_float(o[wofs + i]));
            float sum = 0.f;
            for (uint32_t i = 0; i < k; ++i) {
                const float w = expf(__uint_as_float(o[wofs + i]) - mx);
                o[wofs + i] = __float_as_uint(w);
                sum += w;
            }
            if (sum > 0.f)
                for (uint32_t i = 0; i < k; ++i) o[wofs + i] = __float_as_uint(__uint_as_float(o[wofs + i]) / sum);
        }
    }
}

// The same for up to 256 experts and 32 selections with the logits (bias included; -inf from n on) in registers: v[j] is expert lane +
// 32 j's. Lane i < k gets selection i's id and weight. Keys instead of values in the rounds, none to be selected again as zero.
__device__ __forceinline__ void select_experts(float (&v)[8], uint32_t n, uint32_t k, uint32_t rule, uint32_t lane, uint32_t& id, float& weight) {
    const float floor_v = rule == 0u ? -1.0f : -INFINITY;
    if (rule == 0u) {  // softmax over all experts first
        float m = fmaxf(fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3])), fmaxf(fmaxf(v[4], v[5]), fmaxf(v[6], v[7])));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = lane + 32 * j < n ? expf(v[j] - m) : 0.f;
            sum += v[j];
        }
        sum = warp_sum(sum);
        if (sum > 0.f) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = v[j] / sum;
        }
    }
    const float v0 = __shfl_sync(0xFFFFFFFFu, v[0], 0);  // expert 0, for the "nothing above the floor" case
    uint32_t key[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) key[j] = lane + 32 * j < n && v[j] > floor_v ? float_key(v[j]) : 0u;
    float sel = 0.f;
    id = 0u;
#pragma unroll 1
    for (uint32_t i = 0; i < k; ++i) {
        const uint32_t m = max(max(max(key[0], key[1]), max(key[2], key[3])), max(max(key[4], key[5]), max(key[6], key[7])));
        const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, m);
        uint32_t mine = 0xFFFFFFFFu;
#pragma unroll
        for (int j = 7; j >= 0; --j) mine = key[j] == top ? lane + 32 * j : mine;
        const uint32_t at = __reduce_min_sync(0xFFFFFFFFu, mine);
#pragma unroll
        for (int j = 0; j < 8; ++j) key[j] = at == lane + 32 * j ? 0u : key[j];
        if (lane == i) {
            id = top ? at : 0u;
            sel = top ? key_float(top) : rule == 0u ? floor_v : v0;
        }
    }
    // the sums run over the selections in order, as the sequential loops of the reference do
    float e = sel;
    if (rule != 0u) {
        float m = lane < k ? sel : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
        e = expf(sel - m);
    }
    float sum = 0.f;
#pragma unroll 1
    for (uint32_t i = 0; i < k; ++i) sum += __shfl_sync(0xFFFFFFFFu, e, (int)i);
    weight = sum > 0.f ? e / sum : e;
}

}  // namespace
}  // namespace zc
