// A recorded run of matvecs (Q4_K and Q6_K, one token) as one persistent kernel.
// Stands in for the reference's command buffer of one token's dispatches (src/compute/forward.zig:4530-4564, 5511, 7377-7420,
// 7714), which its queue runs with barriers in between.
//
// As launches of their own the matvecs of a dense decode token (145 of them, 5 to 14 us each) spend about 3 us apiece on
// what is not streaming: CTAs wait for room, convert x, drain. Here one CTA per SM walks through all of them, and its warps
// have roles: one requests weights, across the borders of the calls, as weights depend on no kernel; fourteen compute; one
// converts its share of the calls' x (every block of x is converted once on the GPU, not once per SM) and one brings
// converted x into shared memory, both ahead; three add up and write finished rows. A call whose x or y meets an earlier
// one's waits for that one's tiles to be complete on all SMs; no other call waits for anything.
// The units (16 rows x 512 columns) of a CTA's tiles are dealt to its compute warps one by one; the parts of a tile meet in
// shared memory and are added in the order of the units: no barrier between warps, and sums that do not depend on timing.
// Bound: HBM for some 20 tokens in a row (a dense 8B token, 4.88 GB in 145 calls, 807 us: 6.05 TB/s, 0.92 of the measured copy
// rate), then the card's power limit (900-960 us at 1.66 GHz); as launches 1557. That is with calls that do not read one another's
// results; those that do are better off as launches (What joining gains, below).
// Arithmetic: that of the streaming matvecs (x as 21-bit fixed point per 256 elements, exact integer dot products per block).
#include "program.h"

#include <algorithm>
#include <cstring>

#include "kquant_dot.cuh"
#include "stream_skel.cuh"
#include "tc_common.cuh"

namespace zc {
namespace {

// warps that compute (dense 8B token, 8 / 10 / 12 / 14 / 16: 892 / 823 / 815 / 801 / 844 us, the last short of registers); that write rows
constexpr int kWarps = 14, kWriters = 3, kBlockThreads = (kWarps + 3 + kWriters) * 32;
constexpr uint32_t kRing = 161280;           // bytes of weights under way: 35 units of Q4_K, 23 of Q6_K (21 where rows are not aligned)
constexpr uint32_t kUnits = 64;              // barriers and descriptions; at most kUnits - kWarps units are under way
constexpr uint32_t kParts = 8;               // tiles of a CTA whose parts may be under way
constexpr uint32_t kPartBytes = kWarps * 16 * 4;
constexpr uint32_t kZeros = 256;
constexpr uint32_t kSmem = 232448;
// Polls of a wait, with sleeps of 50 to 300 ns in between: a second and more. The caller's limit for peers and hand-offs is none for
// these waits, most of which are for earlier calls to be complete, as long as that takes.
constexpr uint32_t kPollLimit = 1u << 24;
constexpr uint32_t kNoOp = 0xFFFFu;          // op of a description: there are no more units
struct Sync {
    uint4 unit[kUnits];                      // {address, op | part << 16, block | last << 16 | alignment << 20, tile of the CTA}
    uint64_t full[kUnits];
    uint64_t table;                          // arrival of an x table
    uint32_t start[kUnits];                  // bytes handed out before a unit
    uint32_t taken[kWarps];                  // units a compute warp has read
    uint32_t at[kWarps];                     // the op a compute warp has reached
    uint64_t parts[kParts];                  // the parts of a tile: kWarps arrivals, the first part's makes up for missing ones
    uint32_t added[kParts];                  // tiles that have been added up from that place
    uint32_t maps_ready;                     // tensor maps that can be used
    uint32_t ready;                          // ops whose x table is there
    uint32_t issued;                         // units requested, when the requesting warp is done
    uint32_t gave_up;
};
constexpr uint32_t kTables = (kSmem - 128 - kRing - kZeros - kParts * kPartBytes - (uint32_t)sizeof(Sync)) & ~127u;

// ---- x tables --------------------------------------------------------------------------------------------
__host__ __device__ constexpr uint32_t table_bytes(uint32_t kind, uint32_t K) { return (K / 256) * (kind == PROG_Q4K ? kQ4kTable : kQ6kTable); }
// A unit in the ring: 16 rows of two blocks each, Q6_K as the 16-byte aligned bytes around them. Its rows lie an odd multiple of
// 16 bytes apart, so that a 32-bit read of eight rows meets 32 banks.
__host__ __device__ constexpr uint32_t unit_pitch(uint32_t kind) { return kind == PROG_Q4K ? 288u : kind == PROG_Q6K ? 432u : 464u; }

// x may have been written by another SM within this kernel: read through L2
__device__ __forceinline__ X8 load_x(const float* x, uint32_t blk, int lane) {
    const float4* p = reinterpret_cast<const float4*>(x + (size_t)blk * 256 + 8 * lane);
    return {__ldcg(p), __ldcg(p + 1)};
}

// ---- waits ------------------------------------------------------------------------------------------------
// Every wait is bounded: one that gives up reports, the compute warps stop, and all other waits of the CTA are passed by; the
// results are then wrong and the status says so.
__device__ __forceinline__ uint32_t volatile_u32(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }
__device__ __forceinline__ void store_volatile(uint32_t* p, uint32_t v) { *reinterpret_cast<volatile uint32_t*>(p) = v; }
__device__ __forceinline__ void gave_up(const Program& p, Sync* s, uint32_t site) {
    if (volatile_u32(&s->gave_up)) return;  // the first one says where
    store_volatile(&s->gave_up, 1);
    p.status[0] = 1;
    p.status[1] = site;
}
__device__ __forceinline__ bool wait_bar(const Program& p, Sync* s, uint64_t* bar, uint32_t parity, uint32_t site) {
    for (uint32_t n = 0; !mbar_try_wait(bar, parity);) {  // each sleeps for a while (test and nanosleep instead: 820 -> 834 us)
        if (++n > kWaitLimit || volatile_u32(&s->gave_up)) {
            gave_up(p, s, site);
            return false;
        }
    }
    return true;
}
// polls `ok` until it holds, each lane for itself: no warp-wide operations in it
template <typename Ok>
__device__ __forceinline__ void poll(const Program& p, Sync* s, uint32_t site, uint32_t sleep, Ok ok) {
    for (uint32_t n = 0; !ok(); ++n) {
        if (volatile_u32(&s->gave_up)) break;
        if (n > p.spin_limit) {
            gave_up(p, s, site);
            break;
        }
        if (sleep) __nanosleep(sleep);
    }
}
// The same for a whole warp, whose lanes leave together: those that saw the flag or ran out alone would leave the others in a
// warp-wide operation that never completes.
template <typename Ok>
__device__ __forceinline__ bool poll_warp(const Program& p, Sync* s, uint32_t site, uint32_t sleep, Ok ok) {
    for (uint32_t n = 0; !__all_sync(0xFFFFFFFFu, ok()); ++n) {
        if (__any_sync(0xFFFFFFFFu, volatile_u32(&s->gave_up))) return false;
        if (n > p.spin_limit) {
            gave_up(p, s, site);
            return false;
        }
        if (sleep) __nanosleep(sleep);
    }
    return true;
}
// until `n` ops are complete on all SMs
__device__ __forceinline__ void await_ops(const Program& p, Sync* sync, uint32_t first, uint32_t n, int lane) {
    if (n == 0) return;
    for (uint32_t d = lane; d < n; d += 32) {
        const uint32_t i = p.deps[first + d], want = p.ops[i].tiles;
        poll(p, sync, 191, 100, [&] { return ld_acquire_u32(p.done + i) >= want; });
    }
    __syncwarp();
    __threadfence();
}

__device__ __forceinline__ uint32_t first_of(const Program& p, uint32_t first) {
    return blockIdx.x >= first ? blockIdx.x - first : blockIdx.x + p.grid - first;
}
__device__ __forceinline__ uint32_t tiles_here(const Program& p, uint32_t op) {
    const uint32_t t = first_of(p, p.ops[op].first), n = p.ops[op].tiles;
    return t < n ? (n - t + p.grid - 1) / p.grid : 0u;
}

// ---- the warps ---------------------------------------------------------------------------------------------
// all units below have been read
__device__ __forceinline__ uint32_t units_taken(const Sync* sync, int lane) {
    return __reduce_min_sync(0xFFFFFFFFu, lane < kWarps ? volatile_u32(&sync->taken[lane]) * kWarps + lane : 0xFFFFFFFFu);
}
// The tensor maps, before this CTA's first use: they lie in memory that another recording may have had for its own, and are cached
// by their addresses. (Dense 8B token: 950 us without, 953 so; with each map prefetched behind its fence 959, four at a time 1011;
// fenced by the requesting warp, an op's at a time, 25 us more, by all threads at the start 7.)
__device__ void acquire_maps(const Program& p, Sync* sync, int lane) {
    for (uint32_t i = 0; i < p.n_maps; i += 32) {
        if (i + lane < p.n_maps)
            asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(p.maps + (i + lane) * 128u) : "memory");
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            store_volatile(&sync->maps_ready, i + 32);
        }
    }
}
// Requests the units of the CTA's tiles, in order, into a ring: one tensor copy each, a lane per unit, as many at a time as
// there is room for. (Five warps with 16-byte copies, 9 or 14 a lane and unit, took so many issue slots that a dense 8B token
// was 1650 us; nine, beside eight that compute, 1190; this one 1030 before the other roles' changes.)
__device__ void fetch_weights(const Program& p, Sync* sync, uint32_t ring, int lane) {
    uint32_t head = 0, bytes0 = 0, off = 0, seq0 = 0;  // next unit; bytes handed out; place in the ring; tiles of earlier ops
    for (uint32_t j = 0; j < p.n_ops; ++j) {
        const ProgramOp& op = p.ops[j];
        const uint32_t nt = tiles_here(p, j), units = op.units, n = nt * units, kind = op.kind, size = 16 * unit_pitch(kind);
        const uint32_t tile0 = first_of(p, op.first), pitch = (op.K >> 8) * 210u, end0 = op.tile_end[0], end1 = op.tile_end[1];
        const bool two = op.streams == 2;
        const uint8_t* maps = p.maps + op.map * 128u;
        const uint32_t map_end = j + 1 < p.n_ops ? p.ops[j + 1].map : p.n_maps;
        if (!poll_warp(p, sync, 189, 60, [&] { return volatile_u32(&sync->maps_ready) >= map_end; })) {
            if (lane == 0) sync->issued = head;
            return;
        }
        for (uint32_t i = 0; i < n;) {
            uint32_t k = 0;
            for (uint32_t polls = 0;; ++polls) {
                const uint32_t tail = units_taken(sync, lane);
                uint32_t used = tail < head ? bytes0 - volatile_u32(&sync->start[tail & (kUnits - 1)]) : 0u, o = off;
                if (o + size > kRing) {
                    used += kRing - o;
                    o = 0;
                }
                if (used + size <= kRing) {
                    const uint32_t room = min(kRing - used, kRing - o);
                    k = kind == PROG_Q4K ? room / (16 * 288u) : kind == PROG_Q6K ? room / (16 * 432u) : room / (16 * 464u);
                    k = min(min(k, n - i), min(kUnits - kWarps - (head - tail), 32u));
                }
                if (k) {
                    bytes0 += o == off ? 0u : kRing - off;
                    off = o;
                    break;
                }
                if (polls > p.spin_limit || __any_sync(0xFFFFFFFFu, volatile_u32(&sync->gave_up))) {
                    gave_up(p, sync, 195);
                    if (lane == 0) sync->issued = head;
                    return;
                }
                if (polls) __nanosleep(250);
            }
            if (lane < k) {
                const uint32_t q = (i + lane) / units, idx = i + lane - q * units, e = (head + lane) & (kUnits - 1);
                uint32_t tl = tile0 + q * p.grid, m = 0;
                const uint32_t kb = two ? idx >> 1 : idx;
                if (two) {
                    m = idx & 1u;
                } else {
                    m = (tl >= end0 ? 1u : 0u) + (tl >= end1 ? 1u : 0u);
                    tl -= m == 0 ? 0u : m == 1 ? end0 : end1;
                }
                uint32_t x = kb * 288u, row = tl * 16u;  // byte within a row (of rows c, c + 8, ..: within eight of them), row
                if (kind != PROG_Q4K) x = kb * 420u;
                if (kind == PROG_Q6K_APART) {
                    x += (tl & 7u) * pitch;
                    row = (tl >> 3) * 16u;
                }
                const uint32_t dst = ring + off + lane * size;
                sync->unit[e] = make_uint4(dst, j | (idx % kWarps) << 16, kb | (idx + kWarps >= units ? 1u << 16 : 0u) | (x & 15u) << 20, seq0 + q);
                sync->start[e] = bytes0 + lane * size;
                mbar_expect_tx(&sync->full[e], size);
                asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                             "l"(maps + m * 128u), "r"((x & ~15u) >> 1), "r"(row), "r"(smem_u32(&sync->full[e]))
                             : "memory");
            }
            __syncwarp();
            i += k;
            head += k;
            bytes0 += k * size;
            off += k * size;
        }
        seq0 += nt;
    }
    if (lane == 0) sync->issued = head;
    poll_warp(p, sync, 195, 50, [&] { return head + kWarps - units_taken(sync, lane) <= kUnits; });  // the barriers have been seen
    if (lane < kWarps && !volatile_u32(&sync->gave_up)) {  // no more units
        const uint32_t e = (head + lane) & (kUnits - 1);
        sync->unit[e] = make_uint4(0u, kNoOp, 0u, 0u);
        mbar_arrive(&sync->full[e]);
    }
}

// After a wait has given up: the units that were requested and that nobody has waited for. Their copies end before the CTA does,
// whose shared memory another one may have next.
__device__ void await_copies(Sync* sync, int lane) {
    const uint32_t head = sync->issued;
    for (uint32_t u = units_taken(sync, lane) + lane; u < head; u += 32)
        for (uint32_t n = 0; n < kWaitLimit && !mbar_try_wait(&sync->full[u & (kUnits - 1)], (u / kUnits) & 1);) ++n;
}

// Converts this CTA's share of the calls' x, a block of 256 at a time, as soon as what they wait for is complete.
__device__ void convert_x(const Program& p, Sync* sync, int lane) {
    for (uint32_t j = 0; j < p.n_ops; ++j) {
        const ProgramOp& op = p.ops[j];
        const uint32_t nb = op.K >> 8;
        uint32_t b = first_of(p, op.x_first);
        if (b >= nb) continue;
        await_ops(p, sync, op.dep0, op.deps_x, lane);
        uint8_t* tab = p.tables + (uint64_t)op.x_table * 16u;
        uint32_t n = 0;
        for (; b < nb; b += p.grid, ++n) {
            const X8 r = load_x(op.x, b, lane);
            if (op.kind == PROG_Q4K) prep_q4k(tab, r, op.K, b, lane);
            else prep_q6k(tab, r, op.K >> 8, b, lane);
        }
        __threadfence();
        asm volatile("fence.proxy.async;" ::: "memory");  // read by bulk copies
        __syncwarp();
        if (lane == 0) atomicAdd(p.converted + j, n);
    }
}

// Brings the converted x of the calls into shared memory, ahead of the compute warps.
__device__ void fetch_x(const Program& p, Sync* sync, uint32_t tables, int lane) {
    uint32_t phase = 0;
    for (uint32_t j = 0; j < p.n_ops; ++j) {
        const ProgramOp& op = p.ops[j];
        if (tiles_here(p, j)) {
            const uint32_t need = op.wait_warps, nb = op.K >> 8;
            poll_warp(p, sync, 190, 300, [&] { return lane >= kWarps || volatile_u32(&sync->at[lane]) >= need; });
            if (lane == 0) {
                poll(p, sync, 196, 0, [&] { return ld_acquire_u32(p.converted + j) >= nb; });
                asm volatile("fence.proxy.async;" ::: "memory");
                const uint32_t bytes = (table_bytes(op.kind, op.K) + 15u) & ~15u;
                mbar_expect_tx(&sync->table, bytes);
                asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(tables + op.table * 16u),
                             "l"(p.tables + (uint64_t)op.x_table * 16u), "r"(bytes), "r"(smem_u32(&sync->table))
                             : "memory");
                for (uint32_t n = 0; !mbar_try_wait(&sync->table, phase);) {  // whatever else has given up: the copy ends
                    if (++n > kWaitLimit) {
                        gave_up(p, sync, 197);
                        break;
                    }
                }
            }
            phase ^= 1;
            __syncwarp();
        }
        if (lane == 0) {
            __threadfence_block();
            store_volatile(&sync->ready, j + 1);
        }
        __syncwarp();
    }
}

// Adds the parts of the tiles of every kWriters-th call, in the order of the units, and writes the rows. (A fence and a count
// at the end of every call, and waits for what y needs, behind the old rows: one warp for all calls and four tiles under way
// 1030 us for a dense 8B token, three warps and eight tiles 906.)
__device__ void write_rows(const Program& p, Sync* sync, const float* parts, uint32_t me, int lane) {
    uint32_t seq = 0;
    for (uint32_t j = 0; j < p.n_ops; ++j) {
        const ProgramOp& op = p.ops[j];
        const uint32_t nt = tiles_here(p, j);
        if (nt == 0) continue;
        if (j % kWriters != me) {
            seq += nt;
            continue;
        }
        const uint32_t n_parts = min((uint32_t)kWarps, (uint32_t)op.units), epi = op.epi;
        const bool two = op.streams == 2, adds = epi == PROG_SIGMOID_ACC || (epi == PROG_PLAIN && op.acc);
        float gate = 1.f;
        uint32_t tile = first_of(p, op.first);
        for (uint32_t q = 0; q < nt; ++q, tile += p.grid, ++seq) {
            uint32_t m = 0, tl = tile;
            if (!two) {
                m = (tl >= op.tile_end[0] ? 1u : 0u) + (tl >= op.tile_end[1] ? 1u : 0u);
                tl -= m == 0 ? 0u : op.tile_end[m - 1];
            }
            const uint32_t r = op.kind == PROG_Q6K_APART ? (tl >> 3) * 128 + (tl & 7u) + lane * 8 : tl * 16 + lane;
            const bool live = lane < 16 && r < op.M[m];
            float* y = op.y[m] + r;
            const uint32_t s = seq & (kParts - 1);
            // The parity tells a round from the one before only, and the tile before in this place may be another row writer's.
            poll_warp(p, sync, 198, 60, [&] { return volatile_u32(&sync->added[s]) == seq / kParts; });
            wait_bar(p, sync, &sync->parts[s], (seq / kParts) & 1, 199);
            __syncwarp();
            if (q == 0) {  // parts are there: what x waits for is complete
                await_ops(p, sync, op.dep0 + op.deps_x, op.deps_y, lane);
                __threadfence();
                if (epi == PROG_SIGMOID_ACC) gate = 1.0f / (1.0f + expf(-__ldcg(op.gate)));
            }
            const float old = live && adds ? __ldcg(y) : 0.f;
            // lanes 0..15 add the even parts of the rows, lanes 16..31 the odd ones (gate + up: the two streams)
            const volatile float* part = parts + s * (kPartBytes / 4) + (lane & 15);
            float v = 0.f;
            for (uint32_t k = lane >> 4; k < n_parts; k += 2) v += part[k * 16];
            const float o = __shfl_xor_sync(0xFFFFFFFFu, v, 16);
            if (lane == 0) store_volatile(&sync->added[s], seq / kParts + 1);
            if (live) *y = epi == PROG_GATE_UP ? (v / (1.0f + expf(-v))) * o : epi == PROG_SIGMOID_ACC ? old + gate * (v + o) : old + (v + o);
        }
        if (op.awaited) {
            __threadfence();
            __syncwarp();
            if (lane == 0) atomicAdd(p.done + j, nt);
        }
    }
}

__device__ __forceinline__ void compute(const Program& p, Sync* sync, uint32_t tables, uint32_t zeros, float* parts, uint32_t warp, int lane) {
    const uint32_t g = lane >> 2, t = lane & 3;
    const uint32_t msel = (2u * t) | ((2u * t + 1u) << 4) | 0x7700u;
    const uint32_t m0 = g < 6 && (g & 1) == 0 ? 1u : 0u, m1 = g < 6 && (g & 1) ? 1u : 0u;
    Q4kAcc acc;
    acc.clear();
    uint32_t cur = 0xFFFFFFFFu, kind = 0, tab = 0, bpr = 0, xb = 0, xstep = 0;
    for (uint32_t u = warp, n = 1;; u += kWarps, ++n) {
        const uint32_t e = u & (kUnits - 1);
        if (!__all_sync(0xFFFFFFFFu, wait_bar(p, sync, &sync->full[e], (u / kUnits) & 1, 193))) break;
        const uint4 d = sync->unit[e];
        const uint32_t op_i = d.y & 0xFFFFu;
        if (op_i != cur) {
            if (lane == 0) store_volatile(&sync->at[warp], op_i == kNoOp ? p.n_ops : op_i);
            if (op_i == kNoOp) break;
            cur = op_i;
            const ProgramOp& op = p.ops[cur];
            kind = op.kind;
            bpr = op.K >> 8;
            tab = tables + op.table * 16u;
            if (kind == PROG_Q4K) {
                const bool b_live = g < 6 && (g & 1) == (t >> 1);
                xb = b_live ? tab + (g >> 1) * op.K + 64u * (t >> 1) + 16u * (t & 1) : zeros + 32u;
                xstep = b_live ? 256u : 0u;
            } else {
                xb = tab + (g < 6 ? g : g - 2) * 64u + t * 16u;
                xstep = g < 6 ? 96u : 0u;   // dead columns: zeros
            }
            if (!poll_warp(p, sync, 192, 60, [&] { return volatile_u32(&sync->ready) > cur; })) break;
            __threadfence_block();
            __syncwarp();
        }
        const uint32_t slot = d.x, kb = d.z & 0xFFFFu;
        if (kind == PROG_Q4K) {
            const uint32_t rA = slot + q4k_row(g) * 288, rB = rA + 8 * 288, blk = 2 * kb;
            const uint32_t sx = tab + bpr * 768 + 8 * t + blk * 32, xs = tab + bpr * 800 + blk * 4, x = xb + blk * xstep;
            q4k_block(rA, rB, x, sx, xs, t, msel, acc);
            if (blk + 1 < bpr) q4k_block(rA + 144, rB + 144, x + xstep, sx + 32, xs + 4, t, msel, acc);
        } else {
            // one of the two blocks starts on a word, the other one in the middle of one: bl, bh
            const uint32_t pitch = unit_pitch(kind), o = d.z >> 20, r = slot + g * pitch + (o & ~3u), half = (o >> 1) & 1u, blk = 2 * kb;
            const uint32_t nb = (g < 6 ? tab + bpr * 768 + g * 16 + 4 * t : zeros) + blk * xstep, xs = tab + bpr * 864 + blk * 4, x = xb + blk * 768;
            const bool both = blk + 1 < bpr;
            if (half == 0 || both) {
                const uint32_t a = r + half * 212;
                q6k_block<kWord>(a, a + 8 * pitch, 0u, 0u, x + half * 768, m0, m1, nb + half * xstep, 4 * t, lds_f1(xs + half * 4), acc.M);
            }
            if (half == 1 || both) {
                const uint32_t a = r + (half ^ 1u) * 208, b = half ^ 1u;
                q6k_block<kHalfWord>(a, a + 8 * pitch, 0u, 0u, x + b * 768, m0, m1, nb + b * xstep, 4 * t, lds_f1(xs + b * 4), acc.M);
            }
        }
        // The place may be refilled once its reads are done: the sums depend on all of them.
        const uint32_t all = __float_as_uint(acc.M[0]) ^ __float_as_uint(acc.M[1]) ^ __float_as_uint(acc.m[0]) ^ __float_as_uint(acc.m[1]);
        if (__any_sync(0xFFFFFFFFu, all == 0x9E3779B9u)) __nanosleep(1);
        if (lane == 0) store_volatile(&sync->taken[warp], n);
        if (!(d.z & 0x10000u)) continue;

        // ---- the warp's part of the tile is complete ----
        float v0, v1;
        if (kind == PROG_Q4K) {
            const float ds = __uint_as_float((137u - 7u * t) << 23);
            v0 = fmaf(acc.M[0], ds, -acc.m[0]);
            v1 = fmaf(acc.M[1], ds, -acc.m[1]);
        } else {
            const float ds = __uint_as_float((141u - 7u * t) << 23);
            v0 = acc.M[0] * ds;
            v1 = acc.M[1] * ds;
        }
        acc.clear();
        v0 += __shfl_xor_sync(0xFFFFFFFFu, v0, 1);
        v1 += __shfl_xor_sync(0xFFFFFFFFu, v1, 1);
        v0 += __shfl_xor_sync(0xFFFFFFFFu, v0, 2);
        v1 += __shfl_xor_sync(0xFFFFFFFFu, v1, 2);
        const uint32_t seq = d.w;
        // the place for its parts is free (else no arrival there: it would be one too many)
        if (!poll_warp(p, sync, 194, 100, [&] { return volatile_u32(&sync->added[seq & (kParts - 1)]) == seq / kParts; })) break;
        if (t == 0) {
            float* q = parts + (seq & (kParts - 1)) * (kPartBytes / 4) + (d.y >> 16) * 16 + (kind == PROG_Q4K ? q4k_row(g) : g);
            q[0] = v0;
            q[8] = v1;
        }
        __syncwarp();
        if (lane == 0) {
            const uint32_t units = p.ops[cur].units, arrivals = (d.y >> 16) == 0 && units < kWarps ? kWarps + 1 - units : 1u;
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&sync->parts[seq & (kParts - 1)])), "r"(arrivals) : "memory");
        }
    }
}

__global__ void __launch_bounds__(kBlockThreads, 1) program_kernel_fn(const __grid_constant__ Program p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    uint8_t* tables = base + kRing;
    uint8_t* zeros = tables + kTables;
    float* parts = reinterpret_cast<float*>(zeros + kZeros);
    Sync* sync = reinterpret_cast<Sync*>(zeros + kZeros + kParts * kPartBytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < (int)kZeros / 16) reinterpret_cast<uint4*>(zeros)[tid] = make_uint4(0u, 0u, 0u, 0u);
    if (tid < (int)kUnits) {
        mbar_init(&sync->full[tid], 1);
        sync->start[tid] = 0;
    }
    if (tid < kWarps) sync->taken[tid] = sync->at[tid] = 0;
    if (tid < (int)kParts) {
        mbar_init(&sync->parts[tid], kWarps);
        sync->added[tid] = 0;
    }
    __syncthreads();
    if (tid == 0) {
        mbar_init(&sync->table, 1);
        sync->ready = sync->maps_ready = sync->issued = sync->gave_up = 0;
        mbar_fence_init();
    }
    __syncthreads();
    if (warp < kWarps) compute(p, sync, smem_u32(tables), smem_u32(zeros), parts, warp, lane);
    else if (warp == kWarps) fetch_weights(p, sync, smem_u32(base), lane);
    else if (warp == kWarps + 1) convert_x(p, sync, lane);
    else if (warp == kWarps + 2) fetch_x(p, sync, smem_u32(tables), lane);
    else {
        if (warp == kWarps + 2 + kWriters) acquire_maps(p, sync, lane);  // its first rows are two calls away
        write_rows(p, sync, parts, warp - kWarps - 3, lane);
    }
    __syncthreads();
    if (volatile_u32(&sync->gave_up)) {
        if (warp == kWarps) await_copies(sync, lane);
        __syncthreads();
    }
    if (tid == 0) {  // the last CTA to leave clears the counters for the next launch
        __threadfence();
        if (atomicAdd(p.left, 1u) == p.grid - 1) {
            for (uint32_t i = 0; i < p.n_ops; ++i) p.done[i] = p.converted[i] = 0;
            *p.left = 0;
        }
    }
}

// ---- planning ------------------------------------------------------------------------------------------------
struct Range {
    uintptr_t lo, hi;
    bool meets(const Range& o) const { return lo < o.hi && o.lo < hi; }
};
Range range(const void* p, uint64_t bytes) {
    const uintptr_t q = reinterpret_cast<uintptr_t>(p);
    return {q, q + (p ? bytes : 0)};
}
int matrices(const ProgramOp& o) { return o.streams == 2 ? 1 : o.M[1] == 0 ? 1 : o.M[2] == 0 ? 2 : 3; }
Range out(const ProgramOp& o, int i) { return range(o.y[i], (uint64_t)o.M[i] * 4); }
Range x_of(const ProgramOp& o) { return range(o.x, (uint64_t)o.K * 4); }

// Does `b`, which comes later, read x behind `a`?
bool x_follows(const ProgramOp& a, const ProgramOp& b) {
    for (int i = 0; i < matrices(a); ++i)
        if (out(a, i).meets(x_of(b))) return true;
    return false;
}
// Does it have to write y (or read the gate) behind it?
bool y_follows(const ProgramOp& a, const ProgramOp& b) {
    for (int i = 0; i < matrices(a); ++i) {
        if (out(a, i).meets(range(b.gate, 4))) return true;
        for (int j = 0; j < matrices(b); ++j)
            if (out(a, i).meets(out(b, j))) return true;
    }
    for (int j = 0; j < matrices(b); ++j)
        if (out(b, j).meets(x_of(a)) || out(b, j).meets(range(a.gate, 4))) return true;
    return false;
}
// weights are requested ahead of everything: none may be written within the program
bool writes_weights(const ProgramOp& a, const ProgramOp& b) {
    const uint64_t pitch = (uint64_t)(b.K >> 8) * (b.kind == PROG_Q4K ? 144u : 210u);
    const int n = b.streams == 2 ? 2 : matrices(b);
    for (int i = 0; i < matrices(a); ++i)
        for (int j = 0; j < n; ++j)
            if (out(a, i).meets(range(b.A[j], (uint64_t)b.M[b.streams == 2 ? 0 : j] * pitch))) return true;
    return false;
}

void finish_op(ProgramOp& op) {
    const uint32_t bpr = op.K >> 8;
    op.tiles = 0;
    for (int i = 0; i < matrices(op); ++i) {
        op.tiles += op.kind == PROG_Q6K_APART ? (op.M[i] + 127) / 128 * 8 : (op.M[i] + 15) / 16;
        if (i < 2) op.tile_end[i] = op.tiles;
    }
    for (int i = matrices(op) - 1; i < 2; ++i) op.tile_end[i] = 0xFFFFFFFFu;
    op.units = (uint16_t)((bpr + 1) / 2 * op.streams);
}

uint32_t round128(uint32_t n) { return (n + 127u) & ~127u; }

// Where the x tables lie in shared memory. A table can be replaced when all compute warps have passed its op.
struct Tables {
    uint32_t lo[kProgMaxOps + 1], hi[kProgMaxOps + 1];
    // ops [0, after) must be passed before op j's table can lie at `at`; no further back than `first`
    uint32_t after(uint32_t j, uint32_t at, uint32_t bytes, uint32_t first = 0) const {
        for (uint32_t i = j; i-- > first;)
            if (lo[i] < at + bytes && at < hi[i]) return i + 1;
        return 0;
    }
};
// Chooses op j's place so that its table and the next one's replace tables as old as can be: three ops of 13 KB and one of 46 KB
// in turn then always leave room for the next op's while one is in use (placed one behind the other they waited for the op in
// use twice in four ops: a dense 8B token 906 us, 834 so).
void place_table(Tables& t, uint32_t j, uint32_t bytes, uint32_t next) {
    auto lag = [&](uint32_t i, uint32_t at, uint32_t size) {  // ops in between, up to three
        const uint32_t after = t.after(i, at, size, i < 4 ? 0 : i - 4);
        return i - after < 3 ? i - after : 3u;
    };
    auto candidates = [&](uint32_t i, uint32_t size, auto&& f) {
        f(0u);
        f(kTables - size);
        for (uint32_t k = i, n = 0; k-- > 0 && n < 8; ++n) {
            if (t.hi[k] + size <= kTables) f(t.hi[k]);
            if (t.lo[k] >= size) f(t.lo[k] - size);
        }
    };
    uint32_t best = 0, best_at = 0;
    candidates(j, bytes, [&](uint32_t at) {
        t.lo[j] = at;
        t.hi[j] = at + bytes;
        const uint32_t mine = lag(j, at, bytes);
        uint32_t then = next ? 0u : 3u;
        if (next) candidates(j + 1, next, [&](uint32_t b) { then = std::max(then, lag(j + 1, b, next)); });
        const uint32_t score = 1 + std::min(mine, then) * 4 + mine + then;
        if (score > best) {
            best = score;
            best_at = at;
        }
    });
    t.lo[j] = best_at;
    t.hi[j] = best_at + bytes;
}

// What joining gains or costs: estimates in us, fitted to 382 runs of 2 to 8 calls of 2.4 to 510 MB with another kernel between the
// runs, joined and as launches. None of the runs that pay by them was slower joined; of those that do not, 27 would have been 5 to 24 %
// faster, nearly all of 2 to 4 calls. Measured, joined and as launches:
//   start and end of a joined kernel cost more than those of launches: two calls of Q4_K 4096 x 1024 10.2 and 8.1, four 12.9 and 14.3,
//     eight 18.4 and 26.6; two of Q6_K 12288 x 4096 26.2 and 29.2
//   three warps of an SM write rows: eight calls of Q4_K 65536 x 512, 28 tiles on an SM each, 111.2 and 52.3, of 65536 x 2048 129.0 and 119.6
//   a call that reads what the call before wrote waits for all SMs, has that converted and fetched: eight of Q4_K 4096 x 4096 in a
//     chain 72.7 and 41.1, eight beside one another 24.2 and 41.0; an 8B token whose calls read one another's results 1894 and 1527,
//     one whose calls only add to one vector 900 and 1557
//   one that adds to what the call before wrote waits with its rows only: eight of Q4_K 4096 x 1024 35.2 and 26.7, of 1024 x 4096 29.4
//     and 35.3, of Q6_K 4096 x 4096 47.3 and 55.6; with a call between the two Q4_K 4096 x 4096 31.3 and 41.0
constexpr float kStartUs = 6.7f, kStartTileUs = 0.21f, kReadUs = 6.7f, kAddUs = 1.8f, kAddTileUs = 1.2f, kFullUs = 2.6f;
constexpr float kSafety = 0.97f;      // of the launches' time
constexpr float kHopelessUs = 100.f;  // so far behind its best part a run is looked at no further
float mega_bytes(const ProgramOp& op) {
    const float pitch = (float)(op.K >> 8) * (op.kind == PROG_Q4K ? 144.f : 210.f);
    return ((float)op.M[0] * op.streams + (float)op.M[1] + (float)op.M[2]) * pitch * 1e-6f;
}
float launch_us(const ProgramOp& op) {
    const float mb = mega_bytes(op), start = 2.7f + 0.21f * (float)op.K / 1024.f;
    return op.kind == PROG_Q4K ? start + std::min(mb, 28.f) / 6.5f + std::max(0.f, mb - 28.f) / 6.1f
                               : start + std::min(mb, 40.f) / 4.4f + std::max(0.f, mb - 40.f) / 5.3f;
}

// Adds ops to a program's estimate one by one.
struct Worth {
    float end[kProgMaxOps];  // when an op's rows are written
    float t = 0.f, launches = 0.f;
    void add(const Program& p, uint32_t j) {
        const ProgramOp& op = p.ops[j];
        const uint32_t sm_tiles = (op.tiles + p.grid - 1) / p.grid;
        const float tiles = (float)sm_tiles, stream = std::max(0.63f + mega_bytes(op) / 6.0f, 0.4f * tiles);
        if (j == 0) t = kStartUs + kStartTileUs * tiles;
        t += stream;
        for (uint32_t d = 0; d < op.deps_x; ++d) t = std::max(t, end[p.deps[op.dep0 + d]] + kReadUs + stream);
        for (uint32_t d = op.deps_x; d < (uint32_t)op.deps_x + op.deps_y; ++d) {
            const uint32_t i = p.deps[op.dep0 + d];
            // the tiles on hold and the next ones have no places left
            if (i + 1 == j && sm_tiles + (p.ops[i].tiles + p.grid - 1) / p.grid > kParts) t += kFullUs;
            t = std::max(t, end[i] + kAddUs + kAddTileUs * tiles);
        }
        end[j] = t;
        launches += launch_us(op);
    }
    float gain() const { return kSafety * launches - t; }
};

}  // namespace

bool program_op(uint32_t type, int mode, const DmmvArgs& a, ProgramOp& op) {
    if (a.merge.partial || a.push.world || a.consume.n || a.late) return false;
    const uint64_t bytes = (uint64_t)a.M * (a.K / block_size(type)) * bytes_per_block(type) * (mode == MODE_GATE_UP_SWIGLU ? 2 : 1);
    if (bytes < kStreamMinBytes) return false;
    op = ProgramOp{};
    if (warp_dmmv_eligible(type, mode, a)) op.kind = PROG_Q4K;
    else if (!q6k_dmmv_eligible(type, mode, a)) return false;
    else if ((a.K >> 8) % 8u == 0) op.kind = PROG_Q6K;
    else if (a.M % 8u == 0) op.kind = PROG_Q6K_APART;
    else return false;
    if (table_bytes(op.kind, a.K) > kTables) return false;
    op.epi = mode == MODE_GATE_UP_SWIGLU ? PROG_GATE_UP : mode == MODE_SIGMOID_ACC ? PROG_SIGMOID_ACC : PROG_PLAIN;
    op.streams = mode == MODE_GATE_UP_SWIGLU ? 2 : 1;
    op.A[0] = a.A;
    op.A[1] = a.A2;
    op.y[0] = a.y;
    op.x = a.x;
    op.gate = mode == MODE_SIGMOID_ACC ? a.gate : nullptr;
    op.M[0] = a.M;
    op.K = a.K;
    op.acc = a.acc_mode != 0;
    finish_op(op);
    return true;
}

bool program_op_multi(uint32_t type, uint32_t n, const uint8_t* const* A, float* const* y, const uint32_t* M, const DmmvArgs& common,
                      ProgramOp& op) {
    if (common.push.world || common.consume.n || common.late || !warp_dmmv_multi_eligible(type, n, A, M, common.K, common)) return false;
    if (table_bytes(PROG_Q4K, common.K) > kTables) return false;
    op = ProgramOp{};
    op.kind = PROG_Q4K;
    op.epi = PROG_PLAIN;
    op.streams = 1;
    for (uint32_t i = 0; i < n; ++i) {
        op.A[i] = A[i];
        op.y[i] = y[i];
        op.M[i] = M[i];
    }
    op.x = common.x;
    op.K = common.K;
    op.acc = common.acc_mode != 0;
    finish_op(op);
    return true;
}

uint32_t program_plan(const ProgramOp* list, uint32_t n, int sm_count, Program& p, float* gain) {
    p.n_ops = 0;
    p.spin_limit = kPollLimit;
    p.grid = sm_count > 0 ? (uint32_t)sm_count : 148u;
    uint32_t n_deps = 0, best = 0;
    bool before[kProgMaxOps][kProgMaxOps];  // [j][i]: i is complete before j writes
    Worth worth;
    float most = 0.f;
    for (uint32_t j = 0; j < n && j < kProgMaxOps; ++j) {
        ProgramOp op = list[j];
        bool clash = false;
        for (uint32_t i = 0; i <= j && !clash; ++i) {
            const ProgramOp& o = i == j ? op : p.ops[i];
            clash = writes_weights(o, op) || (i < j && writes_weights(op, o));
        }
        // outputs that meet what the call itself reads, or each other: its tiles are not ordered among themselves
        for (int i = 0; i < matrices(op); ++i) {
            clash = clash || out(op, i).meets(x_of(op)) || out(op, i).meets(range(op.gate, 4));
            for (int k = i + 1; k < matrices(op); ++k) clash = clash || out(op, i).meets(out(op, k));
        }
        if (clash) break;
        op.dep0 = (uint16_t)n_deps;
        memset(before[j], 0, sizeof(before[j]));
        uint32_t added[2] = {0, 0};
        for (int pass = 0; pass < 2; ++pass) {  // x's, then y's: y is written when x has been read
            for (uint32_t i = j; i-- > 0 && n_deps < kProgMaxDeps;) {
                if (before[j][i] || !(pass ? y_follows(p.ops[i], op) : x_follows(p.ops[i], op))) continue;
                p.deps[n_deps++] = (uint16_t)i;
                ++added[pass];
                p.ops[i].awaited = 1;
                before[j][i] = true;
                for (uint32_t k = 0; k < i; ++k) before[j][k] = before[j][k] || before[i][k];
            }
        }
        if (n_deps == kProgMaxDeps) break;
        op.deps_x = (uint16_t)added[0];
        op.deps_y = (uint16_t)added[1];
        p.ops[j] = op;
        p.n_ops = j + 1;
        if (!gain) continue;
        worth.add(p, j);
        if (j > 0 && worth.gain() > most) {
            most = worth.gain();
            best = j + 1;
        }
        if (worth.gain() < most - kHopelessUs) break;
    }
    if (gain) {
        *gain = most;
        p.n_ops = best;
    }
    Tables place;
    uint32_t first = 0, x_first = 0, x_table = 0, maps = 0;
    for (uint32_t j = 0; j < p.n_ops; ++j) {
        ProgramOp& op = p.ops[j];
        op.map = (uint16_t)maps;
        maps += op.streams == 2 ? 2 : (uint32_t)matrices(op);
        op.first = (uint16_t)first;
        first = (uint32_t)((first + op.tiles) % p.grid);
        const uint32_t need = round128(table_bytes(op.kind, op.K));
        place_table(place, j, need, j + 1 < p.n_ops ? round128(table_bytes(p.ops[j + 1].kind, p.ops[j + 1].K)) : 0u);
        op.x_first = (uint16_t)x_first;
        x_first = (x_first + (op.K >> 8)) % p.grid;
        op.x_table = x_table;
        x_table += need / 16;
        op.wait_warps = (uint16_t)place.after(j, place.lo[j], need);
        op.table = (uint16_t)(place.lo[j] / 16);
    }
    p.table_bytes = x_table * 16;
    p.n_maps = maps;
    return p.n_ops >= 2 ? p.n_ops : 0;
}

uint32_t program_maps(const Program& p, CUtensorMap* maps) {
    EncodeFn encode = encode_fn();
    if (!encode) return 0;
    for (uint32_t j = 0; j < p.n_ops; ++j) {
        const ProgramOp& op = p.ops[j];
        const int n = op.streams == 2 ? 2 : matrices(op);
        const uint64_t pitch = (uint64_t)(op.K >> 8) * (op.kind == PROG_Q4K ? 144u : 210u), rows = op.kind == PROG_Q6K_APART ? 8 : 1;
        for (int i = 0; i < n; ++i) {
            const cuuint64_t dims[2] = {pitch * rows / 2, op.M[op.streams == 2 ? 0 : i] / rows}, strides[1] = {pitch * rows};
            const cuuint32_t box[2] = {unit_pitch(op.kind) / 2, 16}, steps[2] = {1, 1};
            if (encode(maps + op.map + i, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<uint8_t*>(op.A[i]), dims, strides, box, steps,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return j;
        }
    }
    return p.n_ops;
}

cudaError_t program_kernel(int sm_count, void** func, uint32_t& threads, uint32_t& smem) {
    static std::atomic<uint64_t> done{0};
    if (cudaError_t e = ensure_dynamic_smem(program_kernel_fn, kSmem, done); e != cudaSuccess) return e;
    int per_sm = 0, dev = 0, sms = 0, coop = 0;
    if (cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, program_kernel_fn, kBlockThreads, kSmem); e != cudaSuccess) return e;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (per_sm < 1 || sms < sm_count || !coop) return cudaErrorNotSupported;
    *func = reinterpret_cast<void*>(program_kernel_fn);
    threads = kBlockThreads;
    smem = kSmem;
    return cudaSuccess;
}

}  // namespace zc
