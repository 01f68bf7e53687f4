// Recorded MoE decode layers (router + selection, gate + up + activation, down + weighted sum) as one kernel: what the three calls of a
// layer contribute, and how a run of layers is laid out.
#pragma once

#include <cuda.h>

#include "kernels.h"

namespace zc {

constexpr uint32_t kMoeMaxLayers = 160;   // of a program: 14 KB of kernel parameters

// The three calls of a layer as they were made.
struct MoeRouterCall {
    const float* x;
    const float* norm_w;
    const float* W;
    const float* bias;
    float* logits;
    uint32_t* routing;
    const uint32_t* routing_local;
    uint32_t n_experts, K, k, rule, shared;
};
struct MoeCalls {
    MoeRouterCall router;
    uint32_t gate_up_type, down_type;
    DmmvArgs gate_up, down;
};

// What the layers of a program have in common.
struct MoeShape {
    uint32_t mx;                          // MXFP4 throughout; else Q4_K gate and up, Q6_K down
    uint32_t E, k, slots, shared, rule, act, H, F;
    uint64_t gate_stride, down_stride;    // bytes between experts
    bool biases_gu, bias_d;
    bool operator==(const MoeShape& o) const {
        return mx == o.mx && E == o.E && k == o.k && slots == o.slots && shared == o.shared && rule == o.rule && act == o.act && H == o.H && F == o.F &&
               gate_stride == o.gate_stride && down_stride == o.down_stride && biases_gu == o.biases_gu && bias_d == o.bias_d;
    }
};

struct MoeLayer {
    const float *x, *router, *router_bias, *bg, *bu, *bd;
    float *logits, *act, *hidden;
    uint32_t* routing;
    uint32_t x_waits;                     // x is what an earlier layer of the program adds to
};

struct MoeProgram {
    uint32_t n_layers, grid;
    uint32_t E, k, slots, n_maps, rule, act, H, F;   // n_maps: tensor maps of a layer. (Four bytes less here and the pairs that the compiler loads at once
                                                   // shift: more is spilled, and 40 layers of 256 experts take 412 us instead of 403.)
    // Tiles are 16 rows, units 16 rows x 512 columns.
    uint32_t gu_tiles_slot, gu_tiles, gu_units;   // of a slot; of all; units of a tile (both streams)
    uint32_t gu_even, gu_takers;                  // which CTAs get how many (Stage)
    uint32_t d_tiles, d_units_slot, d_units;      // tiles; units of a tile along one slot, along all
    uint32_t ring, place_bytes;                   // units of weights under way, bytes of one
    uint32_t gu_tiles_slot_mul, gu_units_mul, d_units_mul, d_units_slot_mul, blocks_slot_mul, ring_mul;   // reciprocals
    uint32_t router_rows;                         // of a CTA, at most
    // shared memory: the ring, x and the router's rows, two tables of x, the activations' table or two (act_step apart; 0: one), zeros, parts
    uint32_t at_x, at_table, table_bytes, at_act, act_step, at_zeros, at_parts_g, at_parts_d, at_sync, smem;
    uint64_t* logits_x;       // [2][E] {value, tag}: how the CTAs exchange logits ..
    uint64_t* act_x;          // [2][slots * F] .. and activations
    uint32_t* words;          // tags used so far, CTAs that have left, CTAs whose rows of hidden are written
    const uint8_t* maps;      // of a layer: gate, up, down of the experts and of the shared expert
    uint32_t spin_limit;
    uint32_t* status;
    MoeLayer layers[kMoeMaxLayers];
};
static_assert(sizeof(MoeProgram) <= 32764, "kernel parameters");

// The layer that three calls in a row make; false: they stay launches.
bool moe_layer(const MoeCalls& c, int sm_count, MoeShape& shape, MoeLayer& layer);
// Lays the first layers of `calls` (n of them, none refused by moe_layer, all of one shape) out as a program; returns how many it took.
uint32_t moe_plan(const MoeCalls* calls, uint32_t n, int sm_count, MoeProgram& p);
uint64_t moe_exchange_bytes(const MoeProgram& p);
// Fills n_layers x n_maps tensor maps; false: one could not be described.
bool moe_maps(const MoeCalls* calls, const MoeProgram& p, CUtensorMap* maps);
cudaError_t moe_program_kernel(bool mx, int sm_count, const MoeProgram& p, void** func, uint32_t& threads);

}  // namespace zc
