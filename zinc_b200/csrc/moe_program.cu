// Recorded MoE decode layers as one persistent kernel.
// Stands in for the reference's GPU-routed MoE layer (src/compute/forward.zig:6139-6545, 6712-6930: router DMMV, softmax_topk, fused
// gate + up, activation, fused down + weighted accumulate) over as many layers as follow one another in a recording.
//
// As three launches a layer is a chain of launch, drain and fill latencies around 3 us of bytes (256 experts, top-8 and a shared one,
// 2048 wide: 19.5 us; 32 MXFP4 experts, top-4, 2880 wide, 8 us of bytes: 38). Here one CTA per SM walks through the layers, and what
// the SMs owe one another within a layer, logits and activations, goes from SM to SM as 64-bit {value, tag} words: a store and a poll,
// no barrier over the grid. Every CTA selects the experts for itself from all logits.
// The warps have roles: one requests weights as soon as a layer's experts are known, across the layers' borders; three do the routing, up
// to two layers ahead (where x is not what the layer before adds to), so that the next layer's weights are under way before it begins;
// sixteen compute.
// Measured (launches / this kernel): 40 layers of the first kind 780 / 403 us, 24 of the second 886 / 511; the same with each layer's x
// what the one before added to 769 / 699 and 906 / 763; single layers behind a kernel that makes their x 21.3 / 20.5 and 41.4 / 35.4,
// of 15 other shapes between 4 % more and 24 % less, K-quants 4 % less in the mean, with no rule found that tells them apart: so every
// layer is joined, whatever is around it.
// Bound: for the first kind by the exchange of the activations (half of a layer: 0.5 us until the last word is seen, 2 until they are
// converted) and by the latency of one unit per warp; for MXFP4 by the instructions of the dot product. What it took: polls of one
// word per tile instead of all words (12.1 -> 10 us and 27.8 -> 26.3 a layer), code that is not unrolled (26.3 -> 23.4), conversion
// shared by a pair of CTAs and gate and up tiles dealt by what down leaves (23.3 -> 21.2), selection by one warp on keys (11.9 -> 9.9).
// Worse: the dot products as functions that are called (21.4 -> 24.6), rings of their own for the two stages (35), routing by the
// compute warps (38).
// Arithmetic: that of the streaming matvecs.
#include "moe_program.h"

#ifndef ZC_MOE_BEFORE_DOWN
#define ZC_MOE_BEFORE_DOWN(layer)  // where a test lets a CTA fall behind its pair
#endif

#include <algorithm>
#include <cstring>

#include "expert_select.cuh"
#include "kquant_dot.cuh"
#include "mx_dot.cuh"
#include "stream_skel.cuh"
#include "tc_common.cuh"

namespace zc {
namespace {

constexpr int kWarps = 16, kRouters = 3, kMoeThreads = (kWarps + kRouters + 1) * 32, kComputeThreads = kWarps * 32;
constexpr uint32_t kMaxRing = 32, kUnits = 64, kMinRing = 8, kMaxRouterRows = 4, kIds = 4;
constexpr uint32_t kMoeSmem = 232448;
constexpr uint32_t kPolls = 1u << 22;   // of a wait for another SM, a microsecond each and more

// Units of 16 rows x 512 columns (Q6_K 256: with as many bytes as Q4_K's, so that a place in the ring is none too large for either).
// Formats whose rows have no 16-byte pitch: a tile is the rows c, c + 8, .. of 128, which lie at one
// place within their groups of eight (eight rows have such a pitch).
enum { UNIT_Q4K, UNIT_Q6K, UNIT_MX };
template <int KIND>
struct UnitOf {
    static constexpr bool kApart = KIND != UNIT_Q4K;
    static constexpr uint32_t kPitch = KIND == UNIT_Q4K ? 288u : KIND == UNIT_Q6K ? 240u : kMxPitch, kBytes = 16 * kPitch;  // in shared memory
    static constexpr uint32_t kStep = KIND == UNIT_Q4K ? 288u : KIND == UNIT_Q6K ? 210u : kMxUnitBytes;                      // along a row
    static __host__ __device__ constexpr uint32_t row_bytes(uint32_t K) { return KIND == UNIT_Q4K ? K / 256 * 144 : KIND == UNIT_Q6K ? K / 256 * 210 : K / 32 * 17; }
    static __host__ __device__ constexpr uint32_t units(uint32_t K) { return KIND == UNIT_Q6K ? K / 256 : (K + 511) / 512; }
    static __host__ __device__ constexpr uint32_t tiles(uint32_t M) { return kApart ? (M + 127) / 128 * 8 : (M + 15) / 16; }
    // of `slots` vectors of K elements
    static __host__ __device__ constexpr uint32_t table(uint32_t K, uint32_t slots) {
        return slots * (KIND == UNIT_Q4K ? K / 256 * kQ4kTable : KIND == UNIT_Q6K ? K / 256 * kQ6kTable : units(K) * kMxTable);
    }
    static __device__ __forceinline__ uint32_t row(uint32_t tile, uint32_t r) { return kApart ? (tile >> 3) * 128 + (tile & 7u) + 8 * r : tile * 16 + r; }
};

static_assert(kUnits >= kWarps + kMaxRing, "see Sync");
struct Sync {
    // Arrival of unit n: barrier n % kUnits, not that of its place: a compute warp that waits for unit n knows no more than that the one
    // sixteen before it was requested, and so that those kUnits before it have been read (kUnits >= kWarps + kMaxRing). Of its place
    // it would not know whether the unit before has arrived, and a parity tells two rounds apart only.
    uint64_t full[kUnits];
    uint64_t empty[kMaxRing];             // by places
    uint64_t rows;                        // arrival of x and of the router's rows
    uint64_t table;                       // the activations' table is filled: the compute warps of both CTAs of the pair
    uint64_t read;                        // one table: the pair's other CTA has read its own
    uint32_t ids[kIds][32], weights[kIds][32];  // the selections of a layer
    float row_part[kMaxRouterRows][kRouters];
    uint32_t routed;                      // layers whose experts are known and whose x is in its table
    uint32_t collected;                   // layers whose activations have been collected
    uint32_t rows_issued;
    uint32_t gave_up;
};

// ---- waits: all bounded. One that gives up reports, all others of the pair of CTAs are passed by, and nothing more is written. -----
__device__ __forceinline__ uint32_t volatile_u32(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }
__device__ __forceinline__ void store_volatile(uint32_t* p, uint32_t v) { *reinterpret_cast<volatile uint32_t*>(p) = v; }
__device__ __forceinline__ bool dead(const Sync* s) { return volatile_u32(&s->gave_up) != 0; }
// how far on in the cluster's window the pair's other CTA has what this one has at p
__device__ __forceinline__ uint32_t to_other(const void* p) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(cluster_ctarank() ^ 1u));
    return r - smem_u32(p);
}
// The other CTA gives up too: this one arrives at the barriers they share without waiting there, which the other could not make out.
__device__ __noinline__ void give_up(const MoeProgram& p, Sync* s, uint32_t site) {
    if (dead(s)) return;
    store_volatile(&s->gave_up, 1);
    st_cluster(smem_u32(&s->gave_up) + to_other(&s->gave_up), 1u);
    p.status[0] = 1;
    p.status[1] = site;
}
__device__ __forceinline__ bool wait_bar(const MoeProgram& p, Sync* s, uint64_t* bar, uint32_t parity, uint32_t site) {
    for (uint32_t n = 0; !mbar_try_wait(bar, parity);) {
        if (dead(s)) return false;
        if (++n > kWaitLimit) {
            give_up(p, s, site);
            return false;
        }
    }
    return true;
}
// .. for something that the pair's other CTA does a part of
__device__ __forceinline__ bool wait_pair(const MoeProgram& p, Sync* s, uint64_t* bar, uint32_t parity, uint32_t site) {
    for (uint32_t n = 0;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (dead(s)) return false;
        if (++n > kWaitLimit) {
            give_up(p, s, site);
            return false;
        }
    }
}
__device__ __forceinline__ void arrive_at(uint64_t* bar, uint32_t rank) {
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %0, %1;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar)),
        "r"(rank)
        : "memory");
}
__device__ __forceinline__ void bar_compute() { asm volatile("bar.sync 1, %0;" ::"n"(kComputeThreads) : "memory"); }
__device__ __forceinline__ void bar_routers() { asm volatile("bar.sync 2, %0;" ::"n"(kRouters * 32) : "memory"); }
// until a counter in shared memory has reached n (a converged warp)
__device__ __forceinline__ bool await(const MoeProgram& p, Sync* s, const uint32_t* counter, uint32_t n, uint32_t sleep, uint32_t site) {
    for (uint32_t polls = 0; !__all_sync(0xFFFFFFFFu, volatile_u32(counter) >= n); ++polls) {
        if (__any_sync(0xFFFFFFFFu, dead(s))) return false;
        if (polls > 16u * kWaitLimit) {
            give_up(p, s, site);
            return false;
        }
        if (sleep) __nanosleep(sleep);
    }
    __threadfence_block();
    return true;
}

// n / d by the high word of a product with d's reciprocal; 0: d = 1
__device__ __forceinline__ uint32_t over(uint32_t n, uint32_t mul) { return mul ? __umulhi(n, mul) : n; }

// ---- the exchange between SMs --------------------------------------------------------------------------------------
__device__ __forceinline__ void publish(uint64_t* p, float v, uint32_t tag) {
    const uint64_t w = (uint64_t)tag << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ uint64_t look(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
struct Two {
    uint64_t a, b;
    __device__ __forceinline__ bool tagged(uint32_t tag) const { return (uint32_t)(a >> 32) == tag && (uint32_t)(b >> 32) == tag; }
};
__device__ __forceinline__ Two look2(const uint64_t* p) {
    Two v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p) : "memory");
    return v;
}
// a load that stays where it stands
__device__ __forceinline__ float load_now(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float value(uint64_t w) { return __uint_as_float((uint32_t)w); }

// ---- weights ------------------------------------------------------------------------------------------------------
// What one stage of a layer is to a CTA: gate + up (kDown false) or down. Down tiles go to the CTAs in turn, from the last one on; gate
// and up tiles in turn for gu_even rounds and then to the first gu_takers CTAs only, those with a down tile less, where that is even.
template <int KIND, bool kDown>
struct Stage {
    using U = UnitOf<KIND>;
    uint32_t tiles, per, n;  // the CTA's tiles, units of a tile, of all of them
    __device__ __forceinline__ explicit Stage(const MoeProgram& p) {
        per = kDown ? p.d_units : p.gu_units;
        if (kDown) {
            const uint32_t cta = p.grid - 1 - blockIdx.x;
            tiles = cta < p.d_tiles ? (p.d_tiles - cta + p.grid - 1) / p.grid : 0u;
        } else {
            const uint32_t rest = p.gu_tiles - p.gu_even * p.grid;
            tiles = p.gu_even;
            if (blockIdx.x < p.gu_takers && blockIdx.x < rest) tiles += (rest - blockIdx.x + p.gu_takers - 1) / p.gu_takers;
        }
        n = tiles * per;
    }
    static __device__ __forceinline__ uint32_t tile(const MoeProgram& p, uint32_t q) {
        if (kDown) return p.grid - 1 - blockIdx.x + q * p.grid;
        return q < p.gu_even ? blockIdx.x + q * p.grid : p.gu_even * p.grid + blockIdx.x + (q - p.gu_even) * p.gu_takers;
    }
    // the tensor copy of unit u of layer l
    __device__ __forceinline__ void request(const MoeProgram& p, const Sync* s, uint32_t l, uint32_t u, uint32_t dst, uint64_t* bar) const {
        const uint32_t q = over(u, kDown ? p.d_units_mul : p.gu_units_mul), r = u - q * per;
        uint32_t tile = Stage::tile(p, q), which, kb, slot;
        if (kDown) {
            slot = over(r, p.d_units_slot_mul);
            kb = r - slot * p.d_units_slot;
            which = 2;
        } else {
            slot = over(tile, p.gu_tiles_slot_mul);
            tile -= slot * p.gu_tiles_slot;
            kb = r >> 1;
            which = r & 1u;
        }
        uint32_t expert = s->ids[l % kIds][slot];
        if (expert == kSharedExpert) {
            expert = 0;
            which += 3;
        }
        uint32_t x = kb * U::kStep, row = tile * 16;
        if (U::kApart) {
            x += (tile & 7u) * U::row_bytes(kDown ? p.F : p.H);
            row = (tile >> 3) * 16;
        }
        mbar_expect_tx(bar, U::kBytes);
        asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                     "l"(p.maps + ((uint64_t)l * p.n_maps + which) * 128u), "r"((x & ~15u) >> 1), "r"(row), "r"(expert), "r"(smem_u32(bar))
                     : "memory");
    }
};

// Requests the units of the CTA's tiles, layer by layer, gate + up before down: one tensor copy each, a lane per unit, as many at a
// time as there is room for. Returns how many it requested.
template <int GU, int D>
__device__ uint32_t fetch_weights(const MoeProgram& p, Sync* s, uint32_t ring, int lane) {
    const Stage<GU, false> g(p);
    const Stage<D, true> d(p);
    const uint32_t R = p.ring, n = g.n + d.n;
    uint32_t head = 0, place = 0, use = 0;  // the next unit, its place, and how often that has been used
    for (uint32_t l = 0; l < p.n_layers; ++l) {
        // the maps lie in memory that another recording may have had for its own, and are cached by their addresses
        if (lane < p.n_maps)
            asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(p.maps + ((uint64_t)l * p.n_maps + lane) * 128u) : "memory");
        __syncwarp();
        if (!await(p, s, &s->routed, l + 1, 40, 210)) return head;
        for (uint32_t i = 0, polls = 0; i < n;) {
            const uint32_t most = min(min(n - i, 32u), R), at = place + lane, mine = at >= R ? at - R : at, uses = use + (at >= R ? 1u : 0u);
            const bool ok = lane < most && (uses == 0 || mbar_test_addr(smem_u32(&s->empty[mine]), (uses - 1) & 1));
            const uint32_t no = ~__ballot_sync(0xFFFFFFFFu, ok), got = no ? __ffs(no) - 1 : 32u;  // lanes from 0 on that have room
            if (got == 0) {
                if (__any_sync(0xFFFFFFFFu, dead(s))) return head;
                if (++polls > 16u * kWaitLimit) {
                    give_up(p, s, 211);
                    return head;
                }
                __nanosleep(20);
                continue;
            }
            if (lane < got) {
                uint64_t* const bar = &s->full[(head + lane) & (kUnits - 1)];
                if (i + lane < g.n) g.request(p, s, l, i + lane, ring + mine * p.place_bytes, bar);
                else d.request(p, s, l, i + lane - g.n, ring + mine * p.place_bytes, bar);
            }
            __syncwarp();
            i += got;
            head += got;
            place += got;
            if (place >= R) {
                place -= R;
                ++use;
            }
            polls = 0;
        }
    }
    return head;
}
// After a wait has given up: copies that nobody has waited for end before the CTA does.
__device__ void await_copies(uint64_t* full, uint32_t ring, uint32_t head, int lane) {
    const uint32_t u = head - 1 - lane;
    if (lane < ring && lane < head)
        for (uint32_t n = 0; n < kWaitLimit && !mbar_try_wait(&full[u & (kUnits - 1)], (u / kUnits) & 1);) ++n;
}

// ---- dot products --------------------------------------------------------------------------------------------------
// The rows g and g + 8 of a unit with its part of x (the table of `nb` blocks, K-quants: the unit's first one is blk, whether it
// has two; MXFP4: the unit, `left` blocks from there on); complete in the lanes t = 0 of each row.
template <int KIND>
struct Dot {
    uint32_t g, t, msel, m0, m1, zeros, tab, nb;
    uint32_t xb, xstep;
    MxLane mx;
    __device__ __forceinline__ void init(uint32_t table, uint32_t blocks, uint32_t zeros_at, int lane) {
        g = lane >> 2;
        t = lane & 3;
        zeros = zeros_at;
        tab = table;
        nb = blocks;
        if constexpr (KIND == UNIT_Q4K) {
            msel = (2u * t) | ((2u * t + 1u) << 4) | 0x7700u;
            const bool live = g < 6 && (g & 1) == (t >> 1);
            xb = live ? tab + (g >> 1) * (nb * 256) + 64u * (t >> 1) + 16u * (t & 1) : zeros + 32u;
            xstep = live ? 256u : 0u;
        } else if constexpr (KIND == UNIT_Q6K) {
            m0 = g < 6 && (g & 1) == 0 ? 1u : 0u;
            m1 = g < 6 && (g & 1) ? 1u : 0u;
            xb = tab + (g < 6 ? g : g - 2) * 64u + t * 16u;
            xstep = g < 6 ? 96u : 0u;
        } else {
            mx.init(tab, tab + nb * 2048, zeros, lane);
        }
    }
    __device__ __forceinline__ void unit(uint32_t slot, uint32_t o, uint32_t blk, bool both, uint32_t left, float& v0, float& v1) const {
        using U = UnitOf<KIND>;
        if constexpr (KIND == UNIT_Q4K) {
            Q4kAcc acc;
            acc.clear();
            const uint32_t rA = slot + q4k_row(g) * U::kPitch, rB = rA + 8 * U::kPitch;
            const uint32_t sx = tab + nb * 768 + 8 * t + blk * 32, xs = tab + nb * 800 + blk * 4, x = xb + blk * xstep;
            q4k_block(rA, rB, x, sx, xs, t, msel, acc);
            if (both) q4k_block(rA + 144, rB + 144, x + xstep, sx + 32, xs + 4, t, msel, acc);
            const float ds = __uint_as_float((137u - 7u * t) << 23);
            v0 = fmaf(acc.M[0], ds, -acc.m[0]);
            v1 = fmaf(acc.M[1], ds, -acc.m[1]);
        } else if constexpr (KIND == UNIT_Q6K) {
            float acc[2] = {0.f, 0.f};
            const uint32_t r = slot + g * U::kPitch + (o & ~3u), x = xb + blk * 768;
            const uint32_t sums = (g < 6 ? tab + nb * 768 + g * 16 + 4 * t : zeros) + blk * xstep;
            const float xs = lds_f1(tab + nb * 864 + blk * 4);
            if (o & 2u) q6k_block<kHalfWord>(r, r + 8 * U::kPitch, 0u, 0u, x, m0, m1, sums, 4 * t, xs, acc);
            else q6k_block<kWord>(r, r + 8 * U::kPitch, 0u, 0u, x, m0, m1, sums, 4 * t, xs, acc);
            const float ds = __uint_as_float((141u - 7u * t) << 23);
            v0 = acc[0] * ds;
            v1 = acc[1] * ds;
        } else {
            float acc[2] = {0.f, 0.f};
            const uint32_t a = slot + g * U::kPitch + o;
            mx.dot(a, a + 8 * U::kPitch, left, blk, acc);
            v0 = acc[0];
            v1 = acc[1];
        }
        v0 += __shfl_xor_sync(0xFFFFFFFFu, v0, 1);
        v1 += __shfl_xor_sync(0xFFFFFFFFu, v1, 1);
        v0 += __shfl_xor_sync(0xFFFFFFFFu, v0, 2);
        v1 += __shfl_xor_sync(0xFFFFFFFFu, v1, 2);
    }
    static __device__ __forceinline__ uint32_t part_row(uint32_t g) { return KIND == UNIT_Q4K ? q4k_row(g) : g; }
};

// Works off the units of a stage of a layer, which begin with unit `first`; their sums go to parts[unit][16].
template <int KIND, bool down>
__device__ __forceinline__ void dots(const MoeProgram& p, Sync* s, uint32_t first, uint32_t ring, uint32_t table, uint32_t zeros, float* parts,
                                  uint32_t warp, int lane) {
    using U = UnitOf<KIND>;
    using St = Stage<KIND, down>;
    const uint32_t n = St(p).n, per = down ? p.d_units : p.gu_units, per_mul = down ? p.d_units_mul : p.gu_units_mul;
    const uint32_t K = down ? p.F : p.H, bpr = K / 256, pitch = U::row_bytes(K);
    Dot<KIND> d;
    d.init(table, (KIND == UNIT_MX ? U::units(K) : bpr) * (down ? p.slots : 1u), zeros, lane);
#pragma unroll 1
    for (uint32_t u = warp; u < n; u += kWarps) {
        const uint32_t seq = first + u, place = seq - over(seq, p.ring_mul) * p.ring;
        const uint32_t q = over(u, per_mul), r = u - q * per;
        uint32_t tile = St::tile(p, q), kb = r >> 1, blk;
        if (down) {
            const uint32_t slot = over(r, p.d_units_slot_mul);
            kb = r - slot * p.d_units_slot;
            blk = KIND == UNIT_Q4K ? slot * bpr + 2 * kb : r;
        } else {
            if (U::kApart) tile -= over(tile, p.gu_tiles_slot_mul) * p.gu_tiles_slot;
            blk = KIND == UNIT_MX ? kb : 2 * kb;
        }
        const uint32_t o = U::kApart ? ((tile & 7u) * pitch + kb * U::kStep) & 15u : 0u;
        if (!__all_sync(0xFFFFFFFFu, wait_bar(p, s, &s->full[seq & (kUnits - 1)], (seq / kUnits) & 1, down ? 213 : 212))) continue;
        float v0, v1;
        d.unit(ring + place * p.place_bytes, o, blk, 2 * kb + 1 < bpr, K / 32 - kb * 16, v0, v1);
        // the place may be refilled once its reads are done: the sums depend on all of them
        if (__any_sync(0xFFFFFFFFu, (__float_as_uint(v0) ^ __float_as_uint(v1)) == 0x9E3779B9u)) __nanosleep(1);
        if (lane == 0) mbar_arrive(&s->empty[place]);
        if ((lane & 3) == 0) {
            float* o16 = parts + u * 16 + Dot<KIND>::part_row(lane >> 2);
            o16[0] = v0;
            o16[8] = v1;
        }
    }
}

// ---- a layer's steps ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t router_rows_here(const MoeProgram& p) {
    const uint32_t r0 = blockIdx.x * p.router_rows;
    return r0 < p.E ? min(p.router_rows, p.E - r0) : 0u;
}
// x and the CTA's rows of the router, on their way
__device__ __forceinline__ void request_rows(const MoeProgram& p, Sync* s, uint32_t l, uint8_t* xbuf) {
    const uint32_t n = router_rows_here(p), bytes = p.H * 4;
    const MoeLayer& ly = p.layers[l];
    s->rows_issued = l + 1;
    mbar_expect_tx(&s->rows, bytes * (1 + n));
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(xbuf)), "l"(ly.x), "r"(bytes),
                 "r"(smem_u32(&s->rows))
                 : "memory");
    if (n)
        asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(xbuf) + bytes),
                     "l"(ly.router + (uint64_t)blockIdx.x * p.router_rows * p.H), "r"(bytes * n), "r"(smem_u32(&s->rows))
                     : "memory");
}

// The routers: the CTA's logits of every layer, x into the layer's table, and the layer's experts (CTA 0 writes them out).
template <int KIND>
__device__ void route(const MoeProgram& p, Sync* s, uint8_t* smem, uint32_t base_tag, uint32_t warp, int lane) {
    const uint32_t tid = warp * 32 + lane, n = router_rows_here(p), K4 = p.H >> 2;
    uint8_t* xbuf = smem + p.at_x;
    const float4* x4 = reinterpret_cast<const float4*>(xbuf);
    if (tid == 0) request_rows(p, s, 0, xbuf);
    for (uint32_t l = 0; l < p.n_layers; ++l) {
        const MoeLayer& ly = p.layers[l];
        const uint32_t tag = base_tag + l + 1;
        // All SMs know the experts of the layer two before, and this one has done with its table of x, when its activations are here.
        // (A wait that gives up is passed by and the warps go on, here as in compute(): they meet at barriers that know no limit.)
        if (l >= 2) await(p, s, &s->collected, l - 1, 40, 217);
        wait_bar(p, s, &s->rows, l & 1, 214);
        __syncwarp();
        for (uint32_t r = 0; r < n; ++r) {
            const float4* w4 = x4 + (r + 1) * K4;
            float sum = 0.f, sum2 = 0.f;
            uint32_t i = tid;
#pragma unroll 2
            for (; i + kRouters * 32 < K4; i += 2 * kRouters * 32) {
                const float4 v = x4[i], w = w4[i], v2 = x4[i + kRouters * 32], w2 = w4[i + kRouters * 32];
                sum += v.x * w.x + v.y * w.y + v.z * w.z + v.w * w.w;
                sum2 += v2.x * w2.x + v2.y * w2.y + v2.z * w2.z + v2.w * w2.w;
            }
            if (i < K4) {
                const float4 v = x4[i], w = w4[i];
                sum += v.x * w.x + v.y * w.y + v.z * w.z + v.w * w.w;
            }
            sum = warp_sum(sum + sum2);
            if (lane == 0) s->row_part[r][warp] = sum;
        }
        bar_routers();
        if (tid < n && !dead(s)) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < kRouters; ++w) sum += s->row_part[tid][w];
            const uint32_t row = blockIdx.x * p.router_rows + tid;
            ly.logits[row] = sum;
            publish(p.logits_x + (l & 1) * p.E + row, sum, tag);
        }
        __syncwarp();
        if (warp == 0) {  // ---- the layer's experts ----
            const uint64_t* src = p.logits_x + (l & 1) * p.E;
            uint64_t w[8];
            for (uint32_t tries = 0;; ++tries) {  // all logits, from the SMs that have them
                bool all = true;
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) w[j] = lane + 32 * j < p.E ? look(src + lane + 32 * j) : (uint64_t)tag << 32;
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) all = all && (uint32_t)(w[j] >> 32) == tag;
                if (__all_sync(0xFFFFFFFFu, all) || __any_sync(0xFFFFFFFFu, dead(s))) break;
                if (tries > p.spin_limit) {
                    give_up(p, s, 500);
                    break;
                }
                __nanosleep(30);
            }
            float v[8];
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                const uint32_t i = lane + 32 * j;
                v[j] = i < p.E ? value(w[j]) + (ly.router_bias ? __ldg(ly.router_bias + i) : 0.0f) : -INFINITY;
            }
            uint32_t id;
            float weight;
            select_experts(v, p.E, p.k, p.rule, lane, id, weight);
            if (lane < p.slots) {
                if (lane >= p.k) {
                    id = kSharedExpert;
                    weight = 1.0f;
                }
                s->ids[l % kIds][lane] = id;
                s->weights[l % kIds][lane] = __float_as_uint(weight);
                if (blockIdx.x == 0 && !dead(s)) {
                    ly.routing[lane] = id;
                    ly.routing[p.slots + lane] = __float_as_uint(weight);
                }
            }
        } else {  // ---- x, for the dot products ----
            uint8_t* table = smem + p.at_table + (l & 1) * p.table_bytes;
            if constexpr (KIND == UNIT_MX) {
#pragma unroll 1
                for (uint32_t c = warp - 1; c < 2 * UnitOf<KIND>::units(p.H); c += kRouters - 1) {
                    const uint32_t e0 = c * 256 + (lane >> 2) * 32 + 4 * (lane & 3);
                    MxX r;
                    r.lo = r.hi = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (e0 < p.H) {
                        r.lo = x4[e0 >> 2];
                        r.hi = x4[(e0 + 16) >> 2];
                    }
                    mx_prep(reinterpret_cast<uint4*>(table), reinterpret_cast<float*>(table + UnitOf<KIND>::units(p.H) * 2048), r, c, lane);
                }
            } else {
#pragma unroll 1
                for (uint32_t b = warp - 1; b < p.H / 256; b += kRouters - 1) {
                    const X8 r = {x4[b * 64 + 2 * lane], x4[b * 64 + 2 * lane + 1]};
                    prep_q4k(table, r, p.H, b, lane);
                }
            }
        }
        __threadfence_block();
        bar_routers();
        if (tid == 0) {
            if (!dead(s)) {
                store_volatile(&s->routed, l + 1);
                if (l + 1 < p.n_layers && !p.layers[l + 1].x_waits) request_rows(p, s, l + 1, xbuf);
            }
        }
    }
}

// The gate and up row of the CTA that a thread finishes, and its biases, requested ahead of the dot products.
struct GateUpRow {
    uint32_t q, r, at;   // tile and row in the parts, place among the activations
    float b0, b1;
};
template <int KIND>
__device__ __forceinline__ GateUpRow gate_up_row(const MoeProgram& p, const Sync* s, uint32_t l, uint32_t i) {
    GateUpRow o{0u, 0u, 0xFFFFFFFFu, 0.f, 0.f};
    const uint32_t q = i >> 4;
    if (q >= Stage<KIND, false>(p).tiles) return o;
    const uint32_t T = Stage<KIND, false>::tile(p, q);
    const uint32_t slot = over(T, p.gu_tiles_slot_mul), row = UnitOf<KIND>::row(T - slot * p.gu_tiles_slot, i & 15u);
    if (row >= p.F) return o;
    o.q = q;
    o.r = i & 15u;
    o.at = slot * p.F + row;
    const MoeLayer& ly = p.layers[l];
    if (ly.bg) {
        const uint32_t e = s->ids[l % kIds][slot];
        if (e < p.E) {
            o.b0 = load_now(ly.bg + (uint64_t)e * p.F + row);
            o.b1 = load_now(ly.bu + (uint64_t)e * p.F + row);
        }
    }
    return o;
}
// Adds its parts, applies the activation and hands the result to all SMs.
__device__ __forceinline__ void activate(const MoeProgram& p, Sync* s, uint32_t l, const float* parts, uint32_t tag, const GateUpRow& o) {
    if (o.at == 0xFFFFFFFFu) return;
    const float* g = parts + o.q * p.gu_units * 16 + o.r;
    float v0 = 0.f, v1 = 0.f;
#pragma unroll 2
    for (uint32_t k = 0; k < p.gu_units; k += 2) {
        v0 += g[k * 16];
        v1 += g[k * 16 + 16];
    }
    const float a = gate_up_act(p.act, v0 + o.b0, v1 + o.b1);
    if (dead(s)) return;
    publish(p.act_x + (uint64_t)(l & 1) * p.slots * p.F + o.at, a, tag);
    p.layers[l].act[o.at] = a;
}

// All activations of layer l, scaled by their slots' weights, into the table of the down projection: every other block of 256 by each
// CTA of a pair, written to both. (All by every CTA: 18 blocks took 1.9 us, 48 took 4.2.)
// The other CTA must have read what is written over there, and nothing awaited here says so of the layer before: the words are other
// CTAs' for most blocks, and its part in s->table of that layer came ahead of its down products. With two tables by the layers' parity
// s->table of the layer between does (every warp arrives there behind its down products of the layer that is written over); with one,
// s->read (compute()).
template <int GU, int KIND>
__device__ __forceinline__ void collect(const MoeProgram& p, Sync* s, uint32_t l, uint8_t* table, uint32_t tag, uint32_t warp, int lane) {
    const uint64_t* src = p.act_x + (uint64_t)(l & 1) * p.slots * p.F;
    const uint32_t per = KIND == UNIT_MX ? 2 * UnitOf<KIND>::units(p.F) : p.F / 256, n = per * p.slots;
    const uint32_t other = to_other(table);
    const uint32_t c0 = 2 * warp + cluster_ctarank();
    auto place = [&](uint32_t c, uint32_t& slot, bool& live) {  // the first of this lane's elements (MXFP4: eight of them 16 apart)
        slot = over(c, p.blocks_slot_mul);
        if constexpr (KIND == UNIT_MX) {
            const uint32_t e0 = (c - slot * per) * 256 + (lane >> 2) * 32 + 4 * (lane & 3);
            live = e0 < p.F;
            return slot * p.F + e0;
        } else {
            live = true;
            return c * 256 + 8 * lane;
        }
    };
    auto load = [&](Two (&w)[4], uint32_t at) {
        const uint64_t *lo = src + at, *hi = lo + (KIND == UNIT_MX ? 16 : 4);
        w[0] = look2(lo);
        w[1] = look2(lo + 2);
        w[2] = look2(hi);
        w[3] = look2(hi + 2);
    };
    // One word of each tile of 16 rows until they are there, 16 a block, and only then all: polls of everything by all SMs took so
    // much of L2 that nothing else got through (256 experts 12.1 us a layer).
#pragma unroll 1
    for (uint32_t c = c0; c < n; c += 2 * kWarps) {
        const uint32_t slot = over(c, p.blocks_slot_mul), e = (c - slot * per) * 256 + (UnitOf<GU>::kApart ? ((lane >> 3) & 1) * 128 + (lane & 7) : (lane & 15) * 16);
        const bool watch = lane < 16 && e < p.F;
        for (uint32_t tries = 0; !__all_sync(0xFFFFFFFFu, !watch || (uint32_t)(look(src + slot * p.F + e) >> 32) == tag); ++tries) {
            if (__any_sync(0xFFFFFFFFu, dead(s))) break;
            if (tries > p.spin_limit) {
                give_up(p, s, 215);
                break;
            }
            __nanosleep(30);
        }
    }
    Two w[4];
    uint32_t slot = 0, at = 0;
    bool live = false;
    if (c0 < n) {
        at = place(c0, slot, live);
        if (live) load(w, at);
    }
#pragma unroll 1
    for (uint32_t c = c0; c < n; c += 2 * kWarps) {
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (live) {
            for (uint32_t tries = 0; !(w[0].tagged(tag) && w[1].tagged(tag) && w[2].tagged(tag) && w[3].tagged(tag)); ++tries) {
                if (dead(s)) break;
                if (tries > p.spin_limit) {
                    give_up(p, s, 215);
                    break;
                }
                load(w, at);
            }
            const float f = __uint_as_float(s->weights[l % kIds][slot]);
            lo = make_float4(value(w[0].a) * f, value(w[0].b) * f, value(w[1].a) * f, value(w[1].b) * f);
            hi = make_float4(value(w[2].a) * f, value(w[2].b) * f, value(w[3].a) * f, value(w[3].b) * f);
        }
        if (c + 2 * kWarps < n) {
            at = place(c + 2 * kWarps, slot, live);
            if (live) load(w, at);
        }
        __syncwarp();
        if constexpr (KIND == UNIT_MX) {
            mx_prep<true>(reinterpret_cast<uint4*>(table), reinterpret_cast<float*>(table + UnitOf<KIND>::units(p.F) * p.slots * 2048), MxX{lo, hi}, c, lane,
                          other);
        } else {
            prep_q6k<true>(table, X8{lo, hi}, n, c, lane, other);
        }
    }
    __syncwarp();
    if (lane < 2) arrive_at(&s->table, (uint32_t)lane);
    __syncwarp();
    wait_pair(p, s, &s->table, l & 1, 219);
}

// The row of hidden that four threads finish, and what its value was and is to get besides the sums.
struct DownRow {
    uint32_t q, r, row;
    float old, bias;
};
template <int KIND>
__device__ __forceinline__ DownRow down_row(const MoeProgram& p, const Sync* s, uint32_t l, uint32_t i) {
    DownRow o{0u, 0u, 0xFFFFFFFFu, 0.f, 0.f};
    const uint32_t q = i >> 6, r = (i >> 2) & 15u, part = i & 3u;
    if (q >= Stage<KIND, true>(p).tiles) return o;
    const uint32_t row = UnitOf<KIND>::row(Stage<KIND, true>::tile(p, q), r);
    if (row >= p.H) return o;
    o.q = q;
    o.r = r;
    o.row = row;
    const MoeLayer& ly = p.layers[l];
    if (part == 0) o.old = ld_cg_f32(ly.hidden + row);
    if (ly.bd)
        for (uint32_t k = part; k < p.slots; k += 4) {
            const uint32_t e = s->ids[l % kIds][k];
            if (e < p.E) o.bias = fmaf(__uint_as_float(s->weights[l % kIds][k]), load_now(ly.bd + (uint64_t)e * p.H + row), o.bias);
        }
    return o;
}
__device__ __forceinline__ void add_row(const MoeProgram& p, Sync* s, uint32_t l, const float* parts, uint32_t i, const DownRow& o) {
    const bool live = o.row != 0xFFFFFFFFu;
    float v = o.bias;
    if (live) {
        const float* d = parts + o.q * p.d_units * 16 + o.r;
#pragma unroll 4
        for (uint32_t k = i & 3u; k < p.d_units; k += 4) v += d[k * 16];
    }
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
    if (live && (i & 3u) == 0 && !dead(s)) p.layers[l].hidden[o.row] = o.old + v;
}

template <int GU, int D>
__device__ void compute(const MoeProgram& p, Sync* s, uint8_t* smem, uint32_t base_tag, uint32_t warp, int lane) {
    float *parts_g = reinterpret_cast<float*>(smem + p.at_parts_g), *parts_d = reinterpret_cast<float*>(smem + p.at_parts_d);
    const uint32_t ring = smem_u32(smem), zeros = ring + p.at_zeros, tid = warp * 32 + lane;
    const uint32_t n_g = Stage<GU, false>(p).n, n_d = Stage<D, true>(p).n;
    uint32_t waits = 0, first = 0;
#pragma unroll 1
    for (uint32_t l = 0; l < p.n_layers; ++l, first += n_g + n_d) {
        const uint32_t tag = base_tag + l + 1;
        uint8_t* act_table = smem + p.at_act + (l & 1) * p.act_step;
        await(p, s, &s->routed, l + 1, 20, 218);
        const GateUpRow gu = gate_up_row<GU>(p, s, l, tid);
        dots<GU, false>(p, s, first, ring, ring + p.at_table + (l & 1) * p.table_bytes, zeros, parts_g, warp, lane);
        // One table: the other CTA has read its own before this one writes there (collect()). For all warps by the barrier, in one warp:
        // 24 layers of 2880 508 -> 511 us; each warp waiting ahead of its first store 528, a warp of its own for it (fewer registers) 541.
        if (p.act_step == 0 && l > 0 && warp == kWarps - 1) {
            wait_pair(p, s, &s->read, (l - 1) & 1, 220);
            __syncwarp();
        }
        bar_compute();
        activate(p, s, l, parts_g, tag, gu);
        collect<GU, D>(p, s, l, act_table, tag, warp, lane);
        if (tid == 0) store_volatile(&s->collected, l + 1);  // by all warps
        const DownRow dr = down_row<D>(p, s, l, tid);
        ZC_MOE_BEFORE_DOWN(l);
        dots<D, true>(p, s, first + n_g, ring, smem_u32(act_table), zeros, parts_d, warp, lane);
        bar_compute();
        if (p.act_step == 0 && tid == kComputeThreads - 1 && l + 1 < p.n_layers) arrive_at(&s->read, cluster_ctarank() ^ 1u);
        __syncwarp();
        add_row(p, s, l, parts_d, tid, dr);
        if (l + 1 < p.n_layers && p.layers[l + 1].x_waits) {  // the next layer's x is what was just written, on all SMs
            ++waits;
            __threadfence();
            asm volatile("fence.proxy.async;" ::: "memory");
            bar_compute();
            if (tid == 0 && !dead(s)) {
                atomicAdd(p.words + 2, 1u);
                bool ok = true;
                for (uint32_t n = 0; ok && ld_acquire_u32(p.words + 2) < waits * p.grid;) {
                    if (dead(s) || ++n > p.spin_limit) {
                        give_up(p, s, 216);
                        ok = false;
                    }
                }
                asm volatile("fence.proxy.async;" ::: "memory");
                if (ok) request_rows(p, s, l + 1, smem + p.at_x);
            }
        }
    }
}

template <int GU, int D>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kMoeThreads, 1) moe_program_kernel_fn(const __grid_constant__ MoeProgram p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    Sync* s = reinterpret_cast<Sync*>(smem + p.at_sync);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < (int)kMxZeros / 16) reinterpret_cast<uint4*>(smem + p.at_zeros)[tid] = make_uint4(0u, 0u, 0u, 0u);
    if (tid < (int)kUnits) mbar_init(&s->full[tid], 1);
    if (tid < (int)kMaxRing) mbar_init(&s->empty[tid], 1);
    if (tid == 0) {
        mbar_init(&s->rows, 1);
        mbar_init(&s->table, 2 * kWarps);
        mbar_init(&s->read, 1);
        s->routed = s->collected = s->rows_issued = s->gave_up = 0;
    }
    mbar_fence_init();
    const uint32_t base_tag = volatile_u32(p.words);  // changed by the last CTA to leave only
    __syncthreads();
    cluster_sync_all();  // the other CTA's barriers exist before anything arrives there
    uint32_t requested = 0;
    if (warp < kWarps) compute<GU, D>(p, s, smem, base_tag, (uint32_t)warp, lane);
    else if (warp < kWarps + kRouters) route<GU>(p, s, smem, base_tag, (uint32_t)warp - kWarps, lane);
    else requested = fetch_weights<GU, D>(p, s, smem_u32(smem), lane);
    if (__syncthreads_or(dead(s))) {  // one answer for all threads
        if (warp == kWarps + kRouters) await_copies(s->full, p.ring, requested, lane);
        __syncthreads();
    }
    cluster_sync_all();  // the other CTA writes and arrives here no more
    if (tid == 0) {
        if (s->rows_issued)  // a copy that nobody has waited for (after a wait has given up)
            for (uint32_t n = 0; n < kWaitLimit && !mbar_try_wait(&s->rows, (s->rows_issued - 1) & 1);) ++n;
        __threadfence();
        if (atomicAdd(p.words + 1, 1u) == p.grid - 1) {  // the last CTA to leave
            p.words[0] = base_tag + p.n_layers;
            p.words[1] = p.words[2] = 0;
        }
    }
}

// ---- planning ------------------------------------------------------------------------------------------------------
struct Range {
    uintptr_t lo, hi;
    bool meets(const Range& o) const { return lo < o.hi && o.lo < hi; }
    bool same(const Range& o) const { return lo == o.lo && hi == o.hi; }
};
Range range(const void* p, uint64_t bytes) {
    const uintptr_t q = reinterpret_cast<uintptr_t>(p);
    return {q, q + (p ? bytes : 0)};
}
constexpr int kWrites = 4;  // logits, routing, activations, hidden
void writes(const MoeLayer& y, const MoeShape& s, Range (&w)[kWrites]) {
    w[0] = range(y.logits, 4ull * s.E);
    w[1] = range(y.routing, 8ull * s.slots);
    w[2] = range(y.act, 4ull * s.slots * s.F);
    w[3] = range(y.hidden, 4ull * s.H);
}
Range x_of(const MoeLayer& y, const MoeShape& s) { return range(y.x, 4ull * s.H); }
uint32_t row_bytes(uint32_t type, uint32_t K) { return K / block_size(type) * bytes_per_block(type); }
// Does `a` write what `b` has as weights or biases (requested ahead of everything)?
bool writes_weights(const MoeLayer& a, const MoeCalls& b, const MoeLayer& lb, const MoeShape& s) {
    Range w[kWrites];
    writes(a, s, w);
    const uint64_t gu = (uint64_t)(s.E - 1) * s.gate_stride + (uint64_t)s.F * row_bytes(b.gate_up_type, s.H), gu1 = (uint64_t)s.F * row_bytes(b.gate_up_type, s.H);
    const uint64_t d = (uint64_t)(s.E - 1) * s.down_stride + (uint64_t)s.H * row_bytes(b.down_type, s.F), d1 = (uint64_t)s.H * row_bytes(b.down_type, s.F);
    const Range reads[] = {range(lb.router, 4ull * s.E * s.H), range(lb.router_bias, 4ull * s.E), range(b.gate_up.A, gu), range(b.gate_up.A2, gu),
                           range(b.gate_up.A_sh, gu1), range(b.gate_up.A2_sh, gu1), range(b.down.A, d), range(b.down.A_sh, d1),
                           range(lb.bg, 4ull * s.E * s.F), range(lb.bu, 4ull * s.E * s.F), range(lb.bd, 4ull * s.E * s.H)};
    for (const Range& r : reads)
        for (const Range& o : w)
            if (o.meets(r)) return true;
    return false;
}
// Outputs of two layers: each the other's very buffer or apart from all of the other's.
bool outputs_clash(const MoeLayer& a, const MoeLayer& b, const MoeShape& s, bool same_layer) {
    Range wa[kWrites], wb[kWrites];
    writes(a, s, wa);
    writes(b, s, wb);
    for (int i = 0; i < kWrites; ++i)
        for (int j = 0; j < kWrites; ++j)
            if (wa[i].meets(wb[j]) && !(i == j && (same_layer || wa[i].same(wb[j])))) return true;
    return false;
}

template <int GU, int D>
bool lay_out(const MoeShape& s, int sm_count, MoeProgram& p) {
    using G = UnitOf<GU>;
    using W = UnitOf<D>;
    const uint32_t sms = sm_count > 0 ? (uint32_t)sm_count : 148u;
    p.E = s.E;
    p.k = s.k;
    p.slots = s.slots;
    p.rule = s.rule;
    p.act = s.act;
    p.H = s.H;
    p.F = s.F;
    p.gu_tiles_slot = G::tiles(s.F);
    p.gu_tiles = p.gu_tiles_slot * s.slots;
    p.gu_units = 2 * G::units(s.H);
    p.d_tiles = W::tiles(s.H);
    p.d_units_slot = W::units(s.F);
    p.d_units = p.d_units_slot * s.slots;
    // Every CTA has gate and up rows: its activations show that it has read what the next layer but one writes over in the exchange.
    p.grid = std::min(sms, p.gu_tiles) & ~1u;   // in pairs
    if (p.grid < sms / 2) return false;
    p.router_rows = (s.E + p.grid - 1) / p.grid;
    if (p.router_rows > kMaxRouterRows) return false;
    p.n_maps = s.shared ? 6 : 3;
    const uint32_t nd = (p.d_tiles + p.grid - 1) / p.grid * p.d_units;
    // gate and up tiles: in turn; or fewer for the CTAs with a down tile more, where the busiest CTA then has less to do
    p.gu_even = p.gu_tiles / p.grid;
    p.gu_takers = p.grid;
    uint32_t most_tiles = (p.gu_tiles + p.grid - 1) / p.grid, least = most_tiles * p.gu_units + nd;
    const uint32_t low = p.grid - p.d_tiles % p.grid;  // CTAs with the fewer down tiles
    for (uint32_t even = p.gu_tiles / p.grid; even >= 1 && low < p.grid; --even) {
        const uint32_t rest = p.gu_tiles - even * p.grid, tiles = even + (rest + low - 1) / low;
        const uint32_t busiest = std::max(even * p.gu_units + nd, tiles * p.gu_units + p.d_tiles / p.grid * p.d_units);
        if (busiest < least) {
            least = busiest;
            p.gu_even = even;
            p.gu_takers = low;
            most_tiles = tiles;
        }
    }
    const uint32_t ng = most_tiles * p.gu_units;
    auto up = [](uint32_t n) { return (n + 127u) & ~127u; };
    p.table_bytes = up(G::table(s.H, 1));
    const uint32_t x_bytes = up(s.H * 4 * (1 + p.router_rows));
    const uint32_t act_bytes = up(W::table(s.F, s.slots));
    const uint32_t fixed = 128 + x_bytes + 2 * p.table_bytes + act_bytes + kMxZeros + up(ng * 64) + up(nd * 64) + up(sizeof(Sync));
    if (ng / p.gu_units * 16 > kComputeThreads || nd / p.d_units * 64 > kComputeThreads) return false;
    p.place_bytes = std::max(G::kBytes, W::kBytes);
    if (fixed + kMinRing * p.place_bytes > kMoeSmem) return false;
    auto ring = [&](uint32_t taken) { return taken > kMoeSmem ? 0u : std::min(kMaxRing, (kMoeSmem - taken) / p.place_bytes); };
    p.ring = ring(fixed);
    // a second table where the ring stays as long: 40 layers of 256 experts take 403 us with it, 414 with one table; the MXFP4 layers of
    // 2880, whose ring it would take from 25 places to 15, 622 and 509
    p.act_step = ring(fixed + act_bytes) == p.ring ? act_bytes : 0;
    bool exact = true;
    auto mul = [&](uint32_t d, uint64_t limit) {
        const uint32_t m = reciprocal(d, limit);
        exact = exact && (m != 0 || d == 1);
        return m;
    };
    const uint32_t blocks_slot = s.mx ? 2 * W::units(s.F) : s.F / 256;
    p.gu_tiles_slot_mul = mul(p.gu_tiles_slot, p.gu_tiles);
    p.gu_units_mul = mul(p.gu_units, ng);
    p.d_units_mul = mul(p.d_units, nd);
    p.d_units_slot_mul = mul(p.d_units_slot, nd);
    p.blocks_slot_mul = mul(blocks_slot, blocks_slot * s.slots);
    p.ring_mul = mul(p.ring, (uint64_t)kMoeMaxLayers * (ng + nd));
    if (!exact) return false;
    uint32_t at = up(p.ring * p.place_bytes);
    auto take = [&](uint32_t bytes) {
        const uint32_t here = at;
        at += up(bytes);
        return here;
    };
    p.at_x = take(x_bytes);
    p.at_table = take(2 * p.table_bytes);
    p.at_act = take(act_bytes + p.act_step);
    p.at_zeros = take(kMxZeros);
    p.at_parts_g = take(ng * 64);
    p.at_parts_d = take(nd * 64);
    p.at_sync = take(sizeof(Sync));
    p.smem = at + 128;
    return p.smem <= kMoeSmem;
}
bool lay_out(const MoeShape& s, int sm_count, MoeProgram& p) {
    return s.mx ? lay_out<UNIT_MX, UNIT_MX>(s, sm_count, p) : lay_out<UNIT_Q4K, UNIT_Q6K>(s, sm_count, p);
}

}  // namespace

bool moe_layer(const MoeCalls& c, int sm_count, MoeShape& s, MoeLayer& y) {
    const MoeRouterCall& r = c.router;
    const DmmvArgs &g = c.gate_up, &d = c.down;
    if (r.norm_w || r.routing_local || r.n_experts > 256 || r.k > 31 || r.k > r.n_experts) return false;
    s = MoeShape{};
    if (c.gate_up_type == T_MXFP4 && c.down_type == T_MXFP4) s.mx = 1;
    else if (c.gate_up_type != T_Q4_K || c.down_type != T_Q6_K) return false;
    s.E = r.n_experts;
    s.k = r.k;
    s.shared = r.shared;
    s.slots = r.k + r.shared;
    s.rule = r.rule;
    s.act = g.act;
    s.H = r.K;
    s.F = g.M;
    s.gate_stride = g.expert_stride;
    s.down_stride = d.expert_stride;
    s.biases_gu = g.bias != nullptr;
    s.bias_d = d.bias != nullptr;
    if (!g.act || g.y2 || g.x != r.x || g.K != s.H || g.routing != r.routing || g.n_used != s.slots || g.x_expert_stride != 0) return false;
    if (d.x != g.y || d.K != s.F || d.M != s.H || d.routing != r.routing || d.n_used != s.slots || d.x_expert_stride != s.F) return false;
    // ids are below the number of experts then, and every slot has a matrix
    if (g.n_experts_max < s.E || d.n_experts_max < s.E) return false;
    if ((g.A_sh != nullptr) != (s.shared != 0) || (d.A_sh != nullptr) != (s.shared != 0)) return false;
    if (g.push.world || g.consume.n || d.push.world || d.consume.n || (g.bias && !g.bias2)) return false;
    const uint32_t cols = s.mx ? 64 : 256;  // eight rows of MXFP4 have a 16-byte pitch where a row has an even number of blocks
    if (s.H % cols || s.F % cols || s.H % 8 || s.F % 8) return false;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.A2) | reinterpret_cast<uintptr_t>(g.A_sh) |
                            reinterpret_cast<uintptr_t>(g.A2_sh) | reinterpret_cast<uintptr_t>(d.A) | reinterpret_cast<uintptr_t>(d.A_sh) |
                            reinterpret_cast<uintptr_t>(r.x) | reinterpret_cast<uintptr_t>(r.W) | (uintptr_t)s.gate_stride | (uintptr_t)s.down_stride;
    if (bases & 15u) return false;
    if (!s.mx && ((uint64_t)s.F * s.slots > 12288 || s.H > 12288)) return false;  // as far as the fixed-point forms of x reach
    y = MoeLayer{};
    y.x = r.x;
    y.router = r.W;
    y.router_bias = r.bias;
    y.logits = r.logits;
    y.routing = r.routing;
    y.act = g.y;
    y.hidden = d.y;
    y.bg = g.bias;
    y.bu = g.bias2;
    y.bd = d.bias;
    // a layer that writes what it reads (but for x, which all SMs have when hidden is written)
    Range w[kWrites];
    writes(y, s, w);
    for (int i = 0; i < kWrites - 1; ++i)
        if (w[i].meets(x_of(y, s))) return false;
    if (writes_weights(y, c, y, s) || outputs_clash(y, y, s, true)) return false;
    MoeProgram p;
    return lay_out(s, sm_count, p);
}

uint32_t moe_plan(const MoeCalls* calls, uint32_t n, int sm_count, MoeProgram& p) {
    MoeShape shape, s;
    p.n_layers = 0;
    p.spin_limit = kPolls;
    for (uint32_t j = 0; j < n && j < kMoeMaxLayers; ++j) {
        MoeLayer y;
        if (!moe_layer(calls[j], sm_count, s, y) || (j && !(s == shape))) break;
        shape = s;
        bool clash = false;
        for (uint32_t i = 0; i < j && !clash; ++i) {
            const MoeLayer& o = p.layers[i];
            Range w[kWrites], v[kWrites];
            writes(o, s, w);
            writes(y, s, v);
            clash = writes_weights(o, calls[j], y, s) || writes_weights(y, calls[i], o, s) || outputs_clash(o, y, s, false);
            for (int k = 0; k < kWrites - 1; ++k) clash = clash || w[k].meets(x_of(y, s)) || v[k].meets(x_of(o, s));
            if (w[kWrites - 1].meets(x_of(y, s))) y.x_waits = 1;
        }
        if (clash) break;
        p.layers[j] = y;
        p.n_layers = j + 1;
    }
    if (p.n_layers && !lay_out(shape, sm_count, p)) p.n_layers = 0;
    return p.n_layers;
}

uint64_t moe_exchange_bytes(const MoeProgram& p) { return 16ull * p.E + 16ull * p.slots * p.F + 256; }

bool moe_maps(const MoeCalls* calls, const MoeProgram& p, CUtensorMap* maps) {
    EncodeFn encode = encode_fn();
    if (!encode) return false;
    for (uint32_t l = 0; l < p.n_layers; ++l) {
        const MoeCalls& c = calls[l];
        for (uint32_t i = 0; i < p.n_maps; ++i) {
            const bool down = i % 3 == 2, shared = i >= 3;
            const DmmvArgs& a = down ? c.down : c.gate_up;
            const uint8_t* A = i % 3 == 1 ? (shared ? a.A2_sh : a.A2) : (shared ? a.A_sh : a.A);
            const uint32_t type = down ? c.down_type : c.gate_up_type;
            const uint64_t rows = type == T_Q4_K ? 1 : 8, pitch = (uint64_t)row_bytes(type, a.K) * rows;
            const uint32_t box0 = type == T_Q4_K ? UnitOf<UNIT_Q4K>::kPitch : type == T_Q6_K ? UnitOf<UNIT_Q6K>::kPitch : UnitOf<UNIT_MX>::kPitch;
            const cuuint64_t dims[3] = {pitch / 2, a.M / rows, shared ? 1 : p.E};
            const cuuint64_t strides[2] = {pitch, shared ? pitch * (a.M / rows) : a.expert_stride};
            const cuuint32_t box[3] = {box0 / 2, 16, 1}, steps[3] = {1, 1, 1};
            if (encode(maps + (size_t)l * p.n_maps + i, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<uint8_t*>(A), dims, strides, box, steps,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
                CUDA_SUCCESS)
                return false;
        }
    }
    return true;
}

cudaError_t moe_program_kernel(bool mx, int sm_count, const MoeProgram& p, void** func, uint32_t& threads) {
    static std::atomic<uint64_t> done[2];
    auto k = mx ? moe_program_kernel_fn<UNIT_MX, UNIT_MX> : moe_program_kernel_fn<UNIT_Q4K, UNIT_Q6K>;
    if (cudaError_t e = ensure_dynamic_smem(k, kMoeSmem, done[mx ? 1 : 0]); e != cudaSuccess) return e;
    int pairs = 0, dev = 0, sms = 0, coop = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.grid);
    cfg.blockDim = dim3(kMoeThreads);
    cfg.dynamicSmemBytes = p.smem;
    if (cudaError_t e = cudaOccupancyMaxActiveClusters(&pairs, k, &cfg); e != cudaSuccess) return e;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if ((uint32_t)pairs * 2 < p.grid || sms < sm_count || !coop) return cudaErrorNotSupported;
    *func = reinterpret_cast<void*>(k);
    threads = kMoeThreads;
    return cudaSuccess;
}

}  // namespace zc
