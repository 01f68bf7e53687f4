// MoE prefill: tokens grouped by routed expert, one tensor-core dequant-GEMM tile per (expert, 128 weight
// rows, up to BN of that expert's tokens), so that an expert's weights are read and dequantised once per
// token tile instead of once per (token, slot) pair.
//
//   1. moe_group_kernel     counts the (token, slot) pairs of every expert, lays the experts' pair lists
//                           side by side (no padding) and writes tile records of at most BN pairs, an expert's pairs
//                           shared out equally
//   2. moe_gather_x_kernel  packs the activation row of every pair, in list order, as bf16 [n_pairs][K]
//   3. Q4_K and Q6_K: moe_gemm_pair.cu; MXFP4: gemm_mx.cu (whose activations are split there); Q6_K rows not a multiple of
//      eight: moe_gemm_tc_kernel. It also serves plain GEMMs on weights without a 16-byte row pitch (MXFP4, Q6_K), K split
//      over several items where tiles are few.
// moe_gemm_tc_kernel: persistent CTAs walk the (tile, row tile) work items: tcgen05.mma with the 128 weight rows on the
// TMEM lanes and the tile's pairs on the columns (as many as it has); the activation box (BN rows from the tile's first
// pair) comes by TMA and may run into the next expert's rows, whose columns are never stored. Raw weight blocks are fetched
// by the dequant threads themselves with 16-byte cp.async pieces of the aligned superset of each row's block into a ring as
// deep as shared memory allows; each copy reports to the slot's mbarrier itself. Types: Q4_K, Q6_K (K % 256 == 0) and
// MXFP4 (K % 64 == 0; dequantised exactly to bf16).
// Warp roles (23 warps): 0 tensor-memory owner + MMA issuer, 1 TMA loader of the activations, 2 idle,
// 3-18 dequant (set j = 4 warps = group j of every 256-column block = weight stage j), 19-22 epilogue.
// Two accumulators in tensor memory let the epilogue of one item overlap the MMAs of the next.
// Bound: the dequant warps' integer pipe (MXFP4: 73 % busy) and the turn-around of one stage per set.
// Every mbarrier wait is bounded; a wait that gives up records {1, site}, raises the CTA's flag, and
// every role drains to the common exit where tensor memory is released.
//
// Replaces recordMoeBatchedDispatch's per-pair kernel for prefill batches
// (src/compute/dmmv.zig:746-792; src/shaders/dmmv_q4k_moe_batched.comp:70-164) with the grouping the
// reference's Metal path does (src/shaders/metal/moe_route_pack.metal:13-36).
#include <math.h>

#include "kernels.h"
#include "tc_common.cuh"

namespace zc {
namespace {

constexpr int kMoeDeqWarp0 = 3, kMoeEpiWarp0 = 19;
constexpr int kMoeThreads = 23 * 32;
// One activation slot (BN x 64 bf16) per weight stage: its TMA load reports to the stage's own barrier, so the
// issuing thread waits once and commits once per stage (each wait and each commit costs it a few hundred
// cycles in this kernel; with a separate activation ring and two waits per stage a layer took 7-20 % longer).
constexpr uint32_t kMoeSmemMax = 227u * 1024u;

// The raw-block ring takes what the weight stages and activation slots leave of the 227 KB: its depth is
// what hides the memory latency (one CTA per SM, so blocks in flight per SM = slots - 1).
template <int TYPE, int BN>
struct MoeTile {
    static constexpr uint32_t kRawBytes = kBM * Raw<TYPE>::kBox;
    static constexpr uint32_t kXBytes = BN * kBK * 2;
    static constexpr uint32_t kAccCols = BN <= 32 ? 32 : BN <= 64 ? 64 : BN <= 128 ? 128 : 256;  // tensor memory: powers of two
    // (two stages per dequant set with 32-token tiles took the raw ring its depth: 360 -> 375 us on 256 experts, T = 512)
    static constexpr int kStages = kAStages;
    static constexpr uint32_t kRawOffset = kStages * kABytes;
    static constexpr int kXSlots = kStages;
    static constexpr uint32_t kAvail = kMoeSmemMax - (512 + 1024) - 1024 - kRawOffset - kXSlots * kXBytes;
    static constexpr int kRawSlots = kAvail / kRawBytes > 8 ? 8 : (int)(kAvail / kRawBytes);
    static constexpr uint32_t kXOffset = (kRawOffset + kRawSlots * kRawBytes + 1023u) & ~1023u;
    static constexpr uint32_t kBarOffset = kXOffset + kXSlots * kXBytes;
    static constexpr uint32_t kSmemBytes = kBarOffset + 512 + 1024;
};

struct MoeBars {
    uint64_t full_a[kAStages];
    uint64_t empty_a[kAStages];
    uint64_t accum_full[2];
    uint64_t accum_empty[2];
    uint64_t full_w[8];   // raw ring: 512 copy-completion arrivals per fill
    uint64_t empty_w[8];  // 16 warp releases per use
    uint32_t tmem_base;
    volatile uint32_t failed;
};

struct MoeGemmArgs {
    const uint8_t* A;
    const uint8_t* a_end;         // one past the last byte of the expert stack
    uint64_t expert_stride;       // bytes
    float* Y;
    const uint32_t* header;       // [0] = number of tiles, [1] = number of listed pairs
    const uint4* tiles;           // {expert, first list slot, pairs in the tile, 0}
    const uint32_t* list;         // pair ids (token * n_used + slot) grouped by expert
    uint32_t M, K, n_used, y_token_stride, row_tiles;
    uint32_t* status;
    uint32_t dense_n;             // > 0: plain GEMM over dense_n tokens (one "expert", identity pair list, no tables) ..
    uint32_t dense_tile;          // .. in tiles of this many
    uint32_t splits, slice;       // work items along K per tile, 256-column blocks in each; two: they add into a zeroed Y
    float* parts;                 // more: [work item][dense_tile][128 rows], added afterwards
};

// Work item w: every slice of K of a row tile, then the next row tile, then the next tile of pairs.
struct Item {
    uint32_t tile, m0;
    int b0, b1;  // blocks of 256 columns
};
__device__ __forceinline__ Item item_of(const MoeGemmArgs& g, uint32_t w, int nblk) {
    Item it;
    uint32_t t = w;
    it.b0 = 0;
    it.b1 = nblk;
    if (g.splits > 1) {
        t = w / g.splits;
        it.b0 = (int)((w - t * g.splits) * g.slice);
        it.b1 = min(nblk, it.b0 + (int)g.slice);
    }
    it.tile = t / g.row_tiles;
    it.m0 = (t - it.tile * g.row_tiles) * kBM;
    return it;
}

// Tile t: from the table, or (dense) the t-th run of tokens of the only matrix.
__device__ __forceinline__ uint4 moe_tile(const MoeGemmArgs& g, uint32_t t) {
    if (g.dense_n) return make_uint4(0u, t * g.dense_tile, min(g.dense_tile, g.dense_n - t * g.dense_tile), 0u);
    return __ldg(&g.tiles[t]);
}

// Position of the dequant warps in the flat sequence of (work item, 256-column block).
struct BlockCursor {
    uint32_t w;             // work item
    int b, b1;              // block of the item; one past its last
    const uint8_t* expert;  // first byte of the item's expert
    uint32_t m0;            // first row of the item's row tile
    uint64_t row_off;       // byte offset of this thread's row inside the expert
};

template <int TYPE, int BN>
__global__ void __launch_bounds__(kMoeThreads, 1)
moe_gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const MoeGemmArgs args) {
    // everything this kernel reads but the weights comes from the kernels before it
    chain_wait();
    MoeGemmArgs g = args;
    after_wait(g.header);
    after_wait(g.tiles);
    after_wait(g.list);
    using T = MoeTile<TYPE, BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* smem_w = smem + T::kRawOffset;
    uint8_t* smem_x = smem + T::kXOffset;
    MoeBars* bars = reinterpret_cast<MoeBars*>(smem + T::kBarOffset);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t n_items = (g.dense_n ? (g.dense_n + g.dense_tile - 1) / g.dense_tile : g.header[0]) * g.row_tiles * g.splits;
    const int n_stages = g.K >> 6;           // 64 columns each
    const int nblk = (n_stages + 3) >> 2;    // 256-column blocks, the last one possibly short (MXFP4)
    constexpr uint32_t kBlock = Raw<TYPE>::kBlock, kBox = Raw<TYPE>::kBox;
    constexpr int kPieces = TYPE == T_MXFP4 ? 10 : (int)kBox / 16;
    const uint64_t row_bytes = TYPE == T_MXFP4 ? (uint64_t)(g.K >> 5) * 17u : (uint64_t)nblk * kBlock;

    if (tid == 0) {
        for (int s = 0; s < T::kStages; ++s) {
            mbar_init(&bars->full_a[s], 5);  // one arrival per warp of the owning set + the activation box
            mbar_init(&bars->empty_a[s], 1);
        }
        for (int s = 0; s < T::kRawSlots; ++s) {
            mbar_init(&bars->full_w[s], 512);
            mbar_init(&bars->empty_w[s], 16);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars->accum_full[s], 1);
            mbar_init(&bars->accum_empty[s], 4);  // one arrival per epilogue warp
        }
        bars->failed = 0;
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&bars->tmem_base)),
                     "r"((uint32_t)(2 * T::kAccCols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(bars->tmem_base);

    if (warp == 0) {
        {  // ---- MMA issuer ----
            uint32_t gs = 0, i = 0;
            bool ok = true;
            for (uint32_t w = blockIdx.x; w < n_items && ok; w += gridDim.x, ++i) {
                const uint32_t ab = i & 1;
                // as many columns as the tile has pairs (N in steps of 16)
                const Item it = item_of(g, w, nblk);
                const int s0 = 4 * it.b0, s1 = min(n_stages, 4 * it.b1);
                const uint32_t cols = warp_uniform((moe_tile(g, it.tile).z + 15u) & ~15u);
                const uint32_t idesc = instr_desc<16>() + ((cols - 16u) >> 3 << 17);
                ok = warp_poll(smem_u32(&bars->accum_empty[ab]), ((i >> 1) & 1) ^ 1, bars, g.status, 121);
                if (!ok) break;
                tc_fence_after();
                for (int s = s0; s < s1; ++s, ++gs) {
                    const int st = gs % T::kStages;
                    const uint32_t ph = (gs / T::kStages) & 1;
                    ok = warp_poll(smem_u32(&bars->full_a[st]), ph, bars, g.status, 122);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t da = smem_desc(smem_u32(smem + st * kABytes));
                    const uint64_t dx = smem_desc(smem_u32(smem_x + st * T::kXBytes));
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < kBK / 16; ++k)
                            umma_bf16(tmem + ab * T::kAccCols, da + 2 * k, dx + 2 * k, idesc, s > s0 || k ? 1u : 0u);
                        umma_commit(&bars->empty_a[st]);
                    }
                }
                if (ok && elect_one()) umma_commit(&bars->accum_full[ab]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // ---- TMA loader of the packed activations ----
            uint32_t gs = 0;
            bool ok = true;
            for (uint32_t w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
                const Item it = item_of(g, w, nblk);
                const uint4 tile = moe_tile(g, it.tile);
                for (int s = 4 * it.b0; s < min(n_stages, 4 * it.b1); ++s, ++gs) {
                    const int st = gs % T::kStages;
                    ok = poll_or_fail(&bars->empty_a[st], ((gs / T::kStages) & 1) ^ 1, bars, g.status, 124);
                    if (!ok) break;
                    mbar_expect_tx(&bars->full_a[st], T::kXBytes);
                    tma_load_2d(smem_x + st * T::kXBytes, &tmap_x, s * kBK, (int)tile.y, &bars->full_a[st]);
                }
            }
        }
    } else if (warp >= kMoeDeqWarp0 && warp < kMoeEpiWarp0) {
        // ---- dequant producers: thread = (row, set j); set j always fills the stages j mod 4. A block that
        // starts at running stage gs hands its group q to set (gs + q) & 3 ----
        const int p = tid - kMoeDeqWarp0 * 32;
        const int row = p & 127, j = p >> 7;
        auto locate = [&](uint32_t w, BlockCursor& c) {
            c.w = w;
            if (w < n_items) {
                const Item it = item_of(g, w, nblk);
                const uint4 tile = moe_tile(g, it.tile);
                c.m0 = it.m0;
                c.b = it.b0;
                c.b1 = it.b1;
                const uint32_t grow = min(c.m0 + (uint32_t)row, g.M - 1);  // rows past M are computed and dropped
                c.expert = g.A + (uint64_t)tile.x * g.expert_stride;
                c.row_off = (uint64_t)grow * row_bytes;
            }
        };
        // The 16-byte pieces of the aligned supersets of all rows' blocks, dealt to the 512 threads row by row: a warp's
        // copy instruction covers three rows' runs of bytes, a handful of cache lines, where one row per lane met 32.
        constexpr int kFetches = (kBM * kPieces + 511) / 512;
        uint32_t f_row[kFetches], f_dst[kFetches];  // byte offset of the thread's pieces' rows in a tile; place in the slot
#pragma unroll
        for (int i = 0; i < kFetches; ++i) {
            const uint32_t idx = (uint32_t)p + 512u * i, r = idx / kPieces, piece = idx - r * kPieces;
            f_row[i] = r * (uint32_t)row_bytes;
            f_dst[i] = (kBM * kPieces) % 512 == 0 || r < (uint32_t)kBM ? (r << 20) | (piece << 16) | (r * kBox + piece * 16) : 0xFFFFFFFFu;
        }
        auto fetch = [&](const BlockCursor& c, uint32_t slot_idx) {
            const uint32_t slot = smem_u32(smem_w) + slot_idx * T::kRawBytes;
            const uint8_t* first = c.expert + (uint64_t)c.m0 * row_bytes + (uint32_t)c.b * kBlock;  // the tile's first row
            const uint32_t low = (uint32_t)reinterpret_cast<uintptr_t>(first) & 15u;
            if (c.m0 + kBM <= g.M && first + (uint64_t)(kBM - 1) * row_bytes + kPieces * 16 <= g.a_end) {
#pragma unroll
                for (int i = 0; i < kFetches; ++i) {
                    if (f_dst[i] != 0xFFFFFFFFu) {
                        const uint8_t* s = first - low + (((low + f_row[i]) & ~15u) + ((f_dst[i] >> 12) & 0xF0u));
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot + (f_dst[i] & 0xFFFFu)), "l"(s) : "memory");
                    }
                }
            } else {  // rows past M repeat the last one (computed, dropped); bytes past the stack are zeros, not read
#pragma unroll 1
                for (int i = 0; i < kFetches; ++i) {
                    const uint32_t idx = (uint32_t)p + 512u * i, r = idx / kPieces, piece = idx - r * kPieces;
                    if (r >= (uint32_t)kBM) break;
                    const uint64_t o = (uint64_t)min(c.m0 + r, g.M - 1) * row_bytes + (uint64_t)c.b * kBlock;
                    const uint8_t* s = c.expert + (o & ~(uint64_t)15) + piece * 16;
                    const uint32_t n = s + 16 <= g.a_end ? 16u : (s < g.a_end ? (uint32_t)(g.a_end - s) : 0u);
                    cp_async16_zfill(smem_w + slot_idx * T::kRawBytes + r * kBox + piece * 16, n ? s : g.A, n);
                }
            }
        };
        auto advance = [&](BlockCursor& c) {
            if (c.b + 1 < c.b1)
                ++c.b;
            else
                locate(c.w + gridDim.x, c);
        };
        // The raw ring: a slot is filled by all 512 threads (each its pieces) and every copy reports to the
        // slot's mbarrier by itself when it lands (cp.async.mbarrier.arrive.noinc), so no thread has to
        // reach a program point for the others and the four sets drift apart as the MMA order wants.
        // A warp releases a slot once it has read its part; the refill waits for all 16 releases.
        constexpr int kSlots = T::kRawSlots;
        BlockCursor cur, ahead;
        locate(blockIdx.x, cur);
        ahead = cur;
        uint32_t gs = 0, slot_c = 0, use_c = 0, slot_f = 0, use_f = 0;
        bool dead = false;
        auto issue_fetch = [&]() {
            if (ahead.w >= n_items) return;
            if (!dead) dead = !poll_or_fail(&bars->empty_w[slot_f], (use_f & 1) ^ 1, bars, g.status, 127);
            if (!dead) fetch(ahead, slot_f);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bars->full_w[slot_f]))
                         : "memory");
            advance(ahead);
            if (++slot_f == (uint32_t)kSlots) {
                slot_f = 0;
                ++use_f;
            }
        };
        for (int d = 0; d < kSlots - 1; ++d) issue_fetch();
        while (cur.w < n_items) {
            const int ns = min(4, n_stages - 4 * cur.b);
            const int q = (j - (int)gs) & 3;  // this set's group of the block, if the block has that many
            const bool mine = q < ns;
            if (mine && !dead) dead = !poll_or_fail(&bars->full_w[slot_c], use_c & 1, bars, g.status, 128);
            if (mine && !dead)
                dead = !poll_or_fail(&bars->empty_a[(gs + q) % T::kStages], (((gs + q) / T::kStages) & 1) ^ 1, bars, g.status, 125);
            if (mine && !dead) {
                uint8_t* a_stage = smem + ((gs + q) % T::kStages) * kABytes;
                const uint8_t* slot = smem_w + slot_c * T::kRawBytes + row * kBox;
                if constexpr (TYPE == T_Q6_K) {
                    const uint32_t off = (uint32_t)((cur.row_off + (uint64_t)cur.b * kBlock) & 15u);
                    dequant_group_q6k(slot, off, q, a_stage, row);
                } else {
                    const uint32_t off = (uint32_t)((cur.row_off + (uint64_t)cur.b * kBlock) & 15u) + 34u * q;
                    dequant_group_mxfp4(slot, off, a_stage, row);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->full_a[(gs + q) % T::kStages]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->empty_w[slot_c]);  // this warp is done with the slot
            advance(cur);
            if (++slot_c == (uint32_t)kSlots) {
                slot_c = 0;
                ++use_c;
            }
            gs += ns;
            issue_fetch();
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp >= kMoeEpiWarp0) {
        // ---- epilogue: lane = weight row, column = pair of the tile ----
        const uint32_t q = warp & 3;
        uint32_t i = 0;
        for (uint32_t w = blockIdx.x; w < n_items; w += gridDim.x, ++i) {
            const uint32_t ab = i & 1;
            const Item it = item_of(g, w, nblk);
            const uint4 tile = moe_tile(g, it.tile);
            const uint32_t m = it.m0 + q * 32 + lane;
            if (!poll_or_fail(&bars->accum_full[ab], (i >> 1) & 1, bars, g.status, 126)) break;
            __syncwarp();
            tc_fence_after();
#pragma unroll 1
            for (uint32_t c = 0; c * 32 < tile.z; ++c) {
                uint32_t v[32];
                const uint32_t taddr = tmem + ((q * 32u) << 16) + ab * T::kAccCols + c * 32;
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                    "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                      "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                      "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
                      "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
                      "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(taddr)
                    : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                // pair of column c*32 + lane; its output row starts at Y + token * y_token_stride + slot * M
                const uint32_t idx = c * 32 + lane;
                const uint32_t pair = idx >= tile.z ? 0u : (g.dense_n ? tile.y + idx : __ldg(&g.list[tile.y + idx]));
                const uint32_t tok = pair / g.n_used, slot = pair - tok * g.n_used;
#pragma unroll
                for (int jj = 0; jj < 32; ++jj) {
                    const uint32_t t_j = __shfl_sync(0xFFFFFFFFu, tok, jj);
                    const uint32_t s_j = __shfl_sync(0xFFFFFFFFu, slot, jj);
                    if (c * 32 + jj < tile.z && m < g.M) {
                        float* y = g.Y + (uint64_t)t_j * g.y_token_stride + (uint64_t)s_j * g.M + m;
                        if (g.parts)
                            g.parts[((uint64_t)w * g.dense_tile + c * 32 + jj) * kBM + q * 32 + lane] = __uint_as_float(v[jj]);
                        else if (g.splits > 1)
                            atomicAdd(y, __uint_as_float(v[jj]));
                        else
                            *y = __uint_as_float(v[jj]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->accum_empty[ab]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(2 * T::kAccCols))
                     : "memory");
    }
}

// ---- grouping ------------------------------------------------------------------------------------------
// One CTA. Shared: cnt[n_experts], seg[n_experts] (first list slot; without held pairs the running cursor), tstart[n_experts],
// totals.
// Bound: latencies in a row, one thread or eight pairs make no difference. So up to 4096 pairs are read once, all loads under
// way together, and keep their expert and their place in it (the count's atomic returns it) in registers; every thread scans
// its own experts; shares are divided in 32 bits where they fit (the code is fetched for this one CTA: less of it is time too). A prefill layer of 256 experts, 4096
// pairs, groups twice: 215.4 us before, 212.0 now; 51 pairs of 16 experts 54.4 and 54.7.
constexpr int kGroupHeld = 4;  // pairs a thread keeps
constexpr uint32_t kGroupTotals = 256;

// pair number k of an expert's c, which `parts` tiles share: its tile and its place there
template <typename T>
__device__ __forceinline__ uint32_t group_place(uint32_t k, uint32_t c, uint32_t parts, uint32_t tstart) {
    const uint32_t i = (uint32_t)(((T)(k + 1) * parts - 1) / c);
    return (tstart + i) << 8 | (k - (uint32_t)((T)i * c / parts));
}

__global__ void __launch_bounds__(1024, 1)
moe_group_kernel(const uint32_t* routing, uint32_t n_pairs, uint32_t n_experts, uint32_t bn, uint32_t* header, uint4* tiles,
                 uint32_t* list, uint2* where, uint32_t* status) {
    extern __shared__ uint32_t sh[];
    uint32_t* cnt = sh;
    uint32_t* seg = sh + n_experts;
    uint32_t* tstart = sh + 2 * n_experts;
    uint32_t* totals = sh + 3 * n_experts;  // the warps' pairs and tiles
    const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t e = tid; e < n_experts; e += nt) cnt[e] = 0;
    __syncthreads();
    chain_wait();
    after_wait(routing);
    const bool held = n_pairs <= kGroupHeld * nt;
    uint32_t mine[kGroupHeld], place[kGroupHeld];
    uint32_t wrong = 0xFFFFFFFFu;  // not an expert (and not the "no expert here" mark): left out and reported
    if (held) {
#pragma unroll
        for (int i = 0; i < kGroupHeld; ++i) mine[i] = tid + i * nt < n_pairs ? routing[tid + i * nt] : 0xFFFFFFFFu;
#pragma unroll
        for (int i = 0; i < kGroupHeld; ++i) {
            if (mine[i] < n_experts) place[i] = atomicAdd(&cnt[mine[i]], 1u);
            else wrong = min(wrong, mine[i]);
        }
    } else {
        for (uint32_t p = tid; p < n_pairs; p += nt) {
            const uint32_t e = routing[p];
            if (e < n_experts) atomicAdd(&cnt[e], 1u);
            else wrong = min(wrong, e);
        }
    }
    if (status && wrong != 0xFFFFFFFFu) {
        status[0] = 2u;
        status[1] = wrong;
    }
    __syncthreads();
    {  // exclusive scan of the pair and tile counts: a chunk of experts per thread
        const uint32_t per = (n_experts + nt - 1) / nt;
        const uint32_t e0 = min(tid * per, n_experts), e1 = min(e0 + per, n_experts);
        uint32_t sp = 0, st = 0;
        for (uint32_t e = e0; e < e1; ++e) {
            sp += cnt[e];
            st += (cnt[e] + bn - 1) / bn;
        }
        uint32_t ip = sp, it = st;
        auto scan = [&](uint32_t& x, uint32_t& y) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, x, o), b = __shfl_up_sync(0xFFFFFFFFu, y, o);
                if ((int)lane >= o) {
                    x += a;
                    y += b;
                }
            }
        };
        scan(ip, it);
        if (lane == 31) {
            totals[warp] = ip;
            totals[32 + warp] = it;
        }
        __syncthreads();
        uint2 t = make_uint2(totals[lane], totals[32 + lane]);  // nt is 1024
        scan(t.x, t.y);
        const uint32_t before = warp ? warp - 1 : 0;
        uint32_t wp = __shfl_sync(0xFFFFFFFFu, t.x, before), wt = __shfl_sync(0xFFFFFFFFu, t.y, before);
        if (warp == 0) wp = wt = 0;
        if (tid == 31) {
            header[0] = t.y;
            header[1] = t.x;
        }
        uint32_t bp = wp + ip - sp, bt = wt + it - st;
        for (uint32_t e = e0; e < e1; ++e) {
            const uint32_t c = cnt[e], parts = (c + bn - 1) / bn;
            seg[e] = bp;
            tstart[e] = bt;
            for (uint32_t i = 0; i < parts; ++i) {  // equal shares: the MMAs take as many columns as a tile has pairs
                const uint32_t lo = (uint32_t)((uint64_t)i * c / parts), hi = (uint32_t)((uint64_t)(i + 1) * c / parts);
                tiles[bt + i] = make_uint4(e, bp + lo, hi - lo, 0u);
            }
            bp += c;
            bt += parts;
        }
    }
    __syncthreads();
    if (held) {
#pragma unroll
        for (int i = 0; i < kGroupHeld; ++i) {
            const uint32_t p = tid + i * nt, e = mine[i];
            if (p >= n_pairs) break;
            if (e < n_experts) list[seg[e] + place[i]] = p;
            if (where) {  // the products of a pair and the parts fit 32 bits
                uint2 to = make_uint2(0xFFFFFFFFu, 0u);
                if (e < n_experts) to = make_uint2(seg[e] + place[i], group_place<uint32_t>(place[i], cnt[e], (cnt[e] + bn - 1) / bn, tstart[e]));
                where[p] = to;
            }
        }
    } else {
        for (uint32_t p = tid; p < n_pairs; p += nt) {
            const uint32_t e = routing[p];
            uint2 to = make_uint2(0xFFFFFFFFu, 0u);
            if (e < n_experts) {
                to.x = atomicAdd(&seg[e], 1u);
                list[to.x] = p;
                if (where) to.y = group_place<uint64_t>(to.x - tiles[tstart[e]].y, cnt[e], (cnt[e] + bn - 1) / bn, tstart[e]);
            }
            if (where) where[p] = to;
        }
    }
}

// One warp per listed pair: its token's activation row as bf16.
__global__ void __launch_bounds__(256)
moe_gather_x_kernel(const float* X, const uint32_t* header, const uint32_t* list, __nv_bfloat16* Xp, uint32_t K,
                    uint32_t n_used, uint32_t x_token_stride) {
    chain_wait();
    after_wait(X);
    after_wait(header);
    after_wait(list);
    const uint32_t slot = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (slot >= header[1]) return;
    const uint32_t pair = list[slot];
    const float* src = X + (uint64_t)(pair / n_used) * x_token_stride;
    uint4* dst = reinterpret_cast<uint4*>(Xp + (uint64_t)slot * K);
    for (uint32_t c = lane; c < K / 8; c += 32) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(src) + 2 * c);
        const float4 b = __ldg(reinterpret_cast<const float4*>(src) + 2 * c + 1);
        uint4 o;
        o.x = bf2_bits(__floats2bfloat162_rn(a.x, a.y));
        o.y = bf2_bits(__floats2bfloat162_rn(a.z, a.w));
        o.z = bf2_bits(__floats2bfloat162_rn(b.x, b.y));
        o.w = bf2_bits(__floats2bfloat162_rn(b.z, b.w));
        dst[c] = o;
    }
}

constexpr uint32_t kMoeMaxExperts = 4096;

struct WsLayout {
    uint64_t header, tiles, list, where, xp, total;
    uint32_t max_tiles;
};
WsLayout ws_layout(uint64_t n_pairs, uint32_t K, uint32_t n_experts, uint32_t bn, bool mx) {
    WsLayout l;
    l.max_tiles = (uint32_t)(n_pairs / bn + n_experts);
    l.header = 0;
    l.tiles = 256;
    l.list = l.tiles + (uint64_t)l.max_tiles * 16;
    l.where = (l.list + n_pairs * 4 + 255) & ~(uint64_t)255;
    l.xp = mx ? (l.where + n_pairs * 8 + 255) & ~(uint64_t)255 : l.where;
    l.total = l.xp + (mx ? mx_bytes(n_pairs, K, l.max_tiles, bn) : n_pairs * K * 2);
    return l;
}

template <int TYPE, int BN>
cudaError_t launch_gemm(const CUtensorMap& map, const MoeGemmArgs& g, uint32_t max_items, cudaStream_t s) {
    auto kern = moe_gemm_tc_kernel<TYPE, BN>;
    static std::atomic<uint64_t> attr_done{0};  // per device ordinal
    if (cudaError_t ea = ensure_dynamic_smem(kern, (int)MoeTile<TYPE, BN>::kSmemBytes, attr_done); ea != cudaSuccess) return ea;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t grid = max_items < (uint32_t)sms ? max_items : (uint32_t)sms;
    return launch_chained(kern, dim3(grid), dim3(kMoeThreads), MoeTile<TYPE, BN>::kSmemBytes, s, map, g);
}

// Most pairs per tile. An expert's weights are unpacked once per tile, which is what bounds the kernel, so an expert
// should need one tile: the average count and two of its standard deviations (about its root each) have to fit.
// 32 and 64 leave shared memory for a deeper ring of raw blocks; Q6_K's blocks are the largest, and beside 160 pairs only
// two fit (12288 x 1280, 77 tokens in one tile: 16.3 us beside 160, 14.6 beside 128).
uint32_t bn_most(uint32_t type) { return type == T_MXFP4 ? 160u : 128u; }
uint32_t pick_bn(uint32_t type, uint64_t n_pairs, uint32_t n_experts) {
    const double avg = (double)n_pairs / n_experts, most = avg + 2.0 * sqrt(avg);
    return most <= 32.0 ? 32u : most <= 64.0 ? 64u : bn_most(type);
}

template <int BN>
cudaError_t launch_gemm_type(uint32_t type, const CUtensorMap& map, const MoeGemmArgs& g, uint32_t max_items, cudaStream_t s) {
    if constexpr (BN == 160) {
        return launch_gemm<T_MXFP4, BN>(map, g, max_items, s);
    } else if constexpr (BN == 128) {
        return launch_gemm<T_Q6_K, BN>(map, g, max_items, s);
    } else {
        return type == T_MXFP4 ? launch_gemm<T_MXFP4, BN>(map, g, max_items, s) : launch_gemm<T_Q6_K, BN>(map, g, max_items, s);
    }
}
cudaError_t launch_gemm_bn(uint32_t type, uint32_t bn, const CUtensorMap& map, const MoeGemmArgs& g, uint32_t max_items, cudaStream_t s) {
    switch (bn) {
        case 32: return launch_gemm_type<32>(type, map, g, max_items, s);
        case 64: return launch_gemm_type<64>(type, map, g, max_items, s);
        case 128: return launch_gemm_type<128>(type, map, g, max_items, s);
        default: return launch_gemm_type<160>(type, map, g, max_items, s);
    }
}

}  // namespace

uint64_t moe_grouped_workspace_bytes(uint64_t n_pairs, uint32_t K, uint32_t n_experts) {
    uint64_t most = 0;  // whatever the type and the tiles
    for (const uint32_t bn : {32u, 64u, 160u}) most = max(most, ws_layout(n_pairs, K, n_experts, bn, true).total);
    return most;
}

bool moe_grouped_eligible(uint32_t type, const uint8_t* A, uint32_t K, uint64_t expert_stride, uint32_t n_experts,
                          uint64_t n_pairs, const float* X, uint32_t x_token_stride, uint64_t ws_size) {
    if (type != T_Q4_K && type != T_Q6_K && type != T_MXFP4) return false;
    if ((type == T_MXFP4 ? (K & 63u) : (K & 255u)) || K < 64 || n_experts > kMoeMaxExperts || n_pairs > 0x7FFFFFFFull)
        return false;
    if (type == T_Q4_K && !moe_pair_eligible(type, kBM, K)) return false;  // the tile kernel here has no Q4_K
    if ((reinterpret_cast<uintptr_t>(A) & 15u) || (expert_stride & 15u)) return false;
    if ((reinterpret_cast<uintptr_t>(X) & 15u) || (x_token_stride & 3u)) return false;
    return ws_size >= ws_layout(n_pairs, K, n_experts, 32, false).total;  // the smallest tile needs the longest table
}

cudaError_t launch_moe_grouped(uint32_t type, const uint8_t* A, uint64_t a_bytes, const float* X, float* Y,
                               const uint32_t* routing, uint32_t M, uint32_t K, uint64_t expert_stride,
                               uint32_t n_experts, uint32_t n_used, uint32_t n_tokens, uint32_t x_token_stride,
                               uint32_t y_token_stride, void* ws, uint64_t ws_size, uint32_t* status, cudaStream_t s,
                               uint64_t* launches, const uint8_t* A2, uint64_t a2_bytes, float* Y2) {
    EncodeFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const uint64_t n_pairs = (uint64_t)n_tokens * n_used;
    const uint32_t bn = pick_bn(type, n_pairs, n_experts);
    // MXFP4 with room for bf16 activations only: the tile kernel on weights unpacked to bf16
    const bool mx = type == T_MXFP4 && ws_size >= ws_layout(n_pairs, K, n_experts, bn, true).total;
    const WsLayout l = ws_layout(n_pairs, K, n_experts, bn, mx);
    uint8_t* base = static_cast<uint8_t*>(ws);
    uint32_t* header = reinterpret_cast<uint32_t*>(base + l.header);
    uint4* tiles = reinterpret_cast<uint4*>(base + l.tiles);
    uint32_t* list = reinterpret_cast<uint32_t*>(base + l.list);
    uint2* where = mx ? reinterpret_cast<uint2*>(base + l.where) : nullptr;
    __nv_bfloat16* xp = reinterpret_cast<__nv_bfloat16*>(base + l.xp);

    cudaError_t e = cudaSuccess;
    if (n_experts * 12 + kGroupTotals > 48u * 1024u) {
        static std::atomic<uint64_t> group_attr{0};
        e = ensure_dynamic_smem(moe_group_kernel, kMoeMaxExperts * 12 + kGroupTotals, group_attr);
        if (e != cudaSuccess) return e;
    }
    e = launch_chained(moe_group_kernel, dim3(1), dim3(1024), n_experts * 12 + kGroupTotals, s, routing, (uint32_t)n_pairs,
                                   n_experts, bn, header, tiles, list, where, status);
    if (e != cudaSuccess) return e;
    if (mx) {  // the weights as they are, the activations as two FP8 terms
        uint8_t* terms = base + l.xp;
        e = launch_mx_terms(X, false, n_tokens, K, x_token_stride, n_used, where, 0, n_pairs, l.max_tiles, bn, terms, s);
        MxGemm p{A, a_bytes, expert_stride, Y, header, tiles, list, M, K, n_experts, n_used, y_token_stride, 0u, 0u, status};
        if (e == cudaSuccess) e = launch_mx_gemm(p, n_pairs, l.max_tiles, bn, terms, s);
        if (e == cudaSuccess && A2) {
            p.A = A2;
            p.a_bytes = a2_bytes;
            p.Y = Y2;
            e = launch_mx_gemm(p, n_pairs, l.max_tiles, bn, terms, s);
        }
        if (e == cudaSuccess && launches) *launches += A2 ? 4 : 3;
        return e;
    }
    e = launch_chained(moe_gather_x_kernel, dim3((uint32_t)((n_pairs + 7) / 8)), dim3(256), 0, s, X, header, list, xp, K,
                       n_used, x_token_stride);
    if (e != cudaSuccess) return e;

    if (moe_pair_eligible(type, M, K)) {
        MoePair p{A, expert_stride, Y, header, tiles, list, M, K, n_experts, n_used, y_token_stride, status};
        e = launch_moe_pair(type, p, xp, n_pairs, l.max_tiles, bn, s);
        if (e == cudaSuccess && A2) {
            p.A = A2;
            p.Y = Y2;
            e = launch_moe_pair(type, p, xp, n_pairs, l.max_tiles, bn, s);
        }
        if (e == cudaSuccess && launches) *launches += A2 ? 4 : 3;
        return e;
    }
    CUtensorMap map;
    const cuuint64_t dims[2] = {K, n_pairs};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {kBK, bn};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, xp, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    MoeGemmArgs g{A, A + a_bytes, expert_stride, Y, header, tiles, list, M, K, n_used, y_token_stride,
                  (M + kBM - 1) / kBM, status, 0u, 0u, 1u, 0u, nullptr};
    const uint64_t max_items64 = (uint64_t)l.max_tiles * g.row_tiles;
    const uint32_t max_items = max_items64 > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)max_items64;
    // one grouping and one packed activation buffer serve both matrices of a pair (gate and up)
    for (int pass = 0; pass < (A2 ? 2 : 1); ++pass) {
        if (pass == 1) {
            g.A = A2;
            g.a_end = A2 + a2_bytes;
            g.Y = Y2;
        }
        e = launch_gemm_bn(type, bn, map, g, max_items, s);
        if (e != cudaSuccess) return e;
    }
    if (launches) *launches += A2 ? 4 : 3;
    return e;
}

// Plain prefill GEMM D[n][m] = sum_k W[m][k] X[n][k] through the same tile kernel (one matrix, token tiles in
// order, no grouping tables): serves the weight layouts a tensor map cannot describe, i.e. MXFP4 (K % 64 == 0)
// and Q6_K with a row pitch that is not a multiple of 16 bytes. X is bf16 [N][stride_b].
bool mul_mm_cp_async_eligible(uint32_t type, const uint8_t* A, const void* B, uint32_t N, uint32_t K,
                              uint32_t stride_b) {
    if (type != T_MXFP4 && type != T_Q6_K) return false;
    if ((type == T_MXFP4 ? (K & 63u) : (K & 255u)) || K < 64 || N < 16) return false;
    return !(reinterpret_cast<uintptr_t>(A) & 15u) && !(reinterpret_cast<uintptr_t>(B) & 15u) && !(stride_b & 7u);
}

cudaError_t launch_mul_mm_cp_async(uint32_t type, const uint8_t* A, uint64_t a_bytes, const void* B, float* D,
                                   uint32_t M, uint32_t N, uint32_t K, uint32_t stride_b, uint32_t stride_d,
                                   uint32_t* status, float* parts, cudaStream_t s, uint64_t* launches) {
    EncodeFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    // equal tiles of at most 160 tokens (128: Q6_K)
    const uint32_t bn = N <= 32 ? 32u : N <= 64 ? 64u : bn_most(type);
    const uint32_t per = (N + (N + bn - 1) / bn - 1) / ((N + bn - 1) / bn);
    CUtensorMap map;
    const cuuint64_t dims[2] = {K, N};
    const cuuint64_t strides[1] = {(cuuint64_t)stride_b * 2};
    const cuuint32_t box[2] = {kBK, bn};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(B), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    MoeGemmArgs g{A, A + a_bytes, 0, D, nullptr, nullptr, nullptr, M, K, 1u, stride_d, (M + kBM - 1) / kBM, status, N, per, 1u, 0u, nullptr};
    // Fewer tiles than SMs: K is split over as many work items as find an SM, of two 256-column blocks at least. The result
    // must not depend on which of them is done first: two add into a zeroed D, the parts of more go through the scratch.
    // (Q6_K 4096 x 11008 on its 32 row tiles alone: 88 us with 32 tokens, 32 split; MXFP4
    // 2880 x 2880, 32 tokens: 15 us added in any order, 17 in this one.)
    const uint64_t tiles = (uint64_t)((N + per - 1) / per) * g.row_tiles;
    const uint32_t nblk = (K + 255) >> 8;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t most = tiles < (uint64_t)sms ? (uint32_t)(sms / tiles) : 1u;
    g.slice = max((nblk + most - 1) / most, 2u);
    g.splits = (nblk + g.slice - 1) / g.slice;
    if (g.splits > 2 && tiles * g.splits * per * kBM * 4 > kExactPartBytes) {  // more SMs than the scratch is sized for
        g.slice = (nblk + 1) / 2;
        g.splits = 2;
    }
    if (g.splits > 2) {
        g.parts = parts;
    } else if (g.splits == 2) {
        if (cudaError_t e = launch_zero(D, M, N, stride_d, s, launches); e != cudaSuccess) return e;
    }
    const uint64_t items64 = tiles * g.splits;
    const uint32_t items = items64 > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)items64;
    cudaError_t e = launch_gemm_bn(type, bn, map, g, items, s);
    if (e == cudaSuccess && g.parts) e = launch_add_parts(parts, D, M, N, kBM, g.row_tiles, per, (uint32_t)tiles, g.splits, stride_d, s);
    if (e == cudaSuccess && launches) *launches += g.parts ? 2 : 1;
    return e;
}

}  // namespace zc
