// MXFP4 prefill GEMM on the block-scaled tensor-core path: D[t][m] = sum_k W[m][k] X[t][k] with the GGUF MXFP4
// weights as they are (E2M1 nibbles, one E8M0 scale byte per 32 elements: exactly the operand format of
// tcgen05.mma kind::mxf8f6f4 with block scaling) and the activations, rounded to bf16, split into two FP8 terms.
//
//   x = x_hi + x_lo, both E4M3 with their own power-of-two scale per 32 elements. A bf16 value has 8 significant
//   bits and an E4M3 value 4, so x_hi (x rounded to 4 significant bits) and x_lo (the remainder, again at most 4
//   significant bits) reproduce x exactly unless an element lies more than 2^14 below its block's maximum (then to
//   2^-22 of that maximum); the two products accumulate into the same f32 accumulator. No weight is dequantised: a
//   row's nibbles are only re-ordered (GGUF keeps element j and j + 16 in one byte, the tensor core wants 16
//   consecutive elements in 8 bytes of a 16-byte chunk), about one integer operation per weight instead of the five
//   of the bf16 route, whose tiles the integer pipe bounds (73 % busy, 3600 cycles per 256 columns of 128 rows).
//
//   1. mx_terms_kernel   X -> x_hi, x_lo (bytes [rows][K]) and their scale bytes in the 512-byte atoms the tensor
//                        core reads (128 tokens x 4 blocks: byte (t % 32) * 16 + (t / 32) * 4 + block), per tile
//   2. mx_gemm_kernel    persistent pairs of CTAs (cta_group::2) over (up to BN tokens of an expert or of the only matrix,
//                        256 weight rows) items: a CTA has 128 of the rows and half of the tokens. Per 128-column stage:
//                        the weight stage (16 KB, K-major, 128-byte swizzle) and its 512 scale bytes written by 128
//                        producer threads (one per row) from raw bytes; x_hi / x_lo tiles and their scale atoms by TMA;
//                        one warp copies the scale atoms into tensor memory (tcgen05.cp) and issues eight MMAs (four
//                        32-column steps x two terms, as wide as the tile has tokens); two accumulators let the
//                        epilogue of an item overlap the next item's MMAs.
// What bounds it: the issuing warp's twelve tensor-core instructions a stage (420 cycles, and some 200 of barrier polls)
// with few tokens, the turn-around of four stages with 160. Measured, down projection of 32 experts 2880 x 2880: 64 tokens,
// top 4, 99 us with the bf16 tiles, 62 here; 1024 tokens 135 and 96. What it took: CTA pairs (half the activation bytes per
// SM, and an issue serves twice the rows), a loader thread per stream (a TMA issue costs its thread 150 cycles), raw bytes
// by TMA three stages at a time (copied by warps they kept the shared-memory pipe from the producers: 1060 cycles to
// repack a stage instead of 550). Bringing the next item's weights to L2 ahead cost 5 %: TMA serves that too.
// Every mbarrier wait is bounded; a wait that gives up records {1, site}, raises the CTA's flag, and every role
// drains to the common exit where tensor memory is released.
//
// Replaces the tiled prefill GEMM dispatch for MXFP4 weights (src/compute/dmmv.zig:1045-1094 recordMulMmQ4K is
// its Q4_K form; element order and scale rule of MXFP4: src/compute/forward.zig:441-459).
#include <cuda_fp8.h>

#include "kernels.h"
#include "tc_common.cuh"

namespace zc {
namespace {

constexpr int kMxStageK = 128;             // columns per stage: four MXFP4 blocks, one scale atom
constexpr uint32_t kMxABytes = kBM * 128;  // 16 KB: 128 rows x 128 padded-FP4 bytes
constexpr uint32_t kMxAtom = 512;          // scale bytes of 128 rows or tokens, four blocks
constexpr int kMxGroups = 3;               // of producer warps; group j fills every third stage
// Raw bytes come three stages (204 bytes of a row) at a time, in their 16-byte aligned superset of up to 14 pieces: the
// load unit takes a copy instruction apart by the lines it meets, some 27 cycles where a run of bytes was one stage's 68.
// Rows 240 bytes apart: 8-byte reads of 16 rows meet two per bank pair.
constexpr uint32_t kMxPieces = 14, kMxRawRow = 240, kMxRawSlot = kBM * kMxRawRow, kMxUnit = kMxGroups;
// Warps: 0 tensor memory + MMA issue; 1 loader of x_hi, 3 of x_lo, 4 of the scale atoms, 2 and 5..7 of the raw
// weight bytes (one thread each: an issue costs its thread some 150 cycles); or, where TMA cannot fetch the
// raw bytes, 5..8 copy them. Then three groups of four producer warps (a thread per weight row; the groups work on different stages at the same
// time), then four epilogue warps.
constexpr int kMxFetchWarp0 = 5, kMxFetchWarps = 4;
constexpr int kMxProdWarp0 = kMxFetchWarp0 + kMxFetchWarps, kMxGroupWarps = 4, kMxEpiWarp0 = kMxProdWarp0 + kMxGroups * kMxGroupWarps;
constexpr int kMxThreads = (kMxEpiWarp0 + 4) * 32;

template <int BN>
struct MxTile {
    static constexpr uint32_t kXBytes = BN / 2 * 128;   // one term of the CTA's half of the tokens
    // Stages: what hides a slot's turn-around (commit, TMA latency, repacking: some 2000 cycles against 500 of MMAs)
    static constexpr int kStages = BN > 64 ? 4 : 6;
    static constexpr uint32_t kSfX = BN > 128 ? 2 * kMxAtom : kMxAtom;  // scale bytes of one term of a tile, four blocks
    // A | x_hi | x_lo | scales of A, x_hi, x_lo, padded to the 1024-byte alignment the swizzled tiles need
    static constexpr uint32_t kSfOffset = kMxABytes + 2 * kXBytes;
    static constexpr uint32_t kStageBytes = (kSfOffset + kMxAtom + 2 * kSfX + 1023u) & ~1023u;
    static constexpr uint32_t kRawOffset = kStages * kStageBytes;
    static constexpr uint32_t kAvail = 227u * 1024u - 1024 - 512 - kRawOffset;
    static constexpr uint32_t kRawSlots = kAvail / kMxRawSlot > 4 ? 4 : kAvail / kMxRawSlot;
    static_assert(kRawSlots >= 2);
    static constexpr uint32_t kBarOffset = kRawOffset + kRawSlots * kMxRawSlot;
    static constexpr uint32_t kSmemBytes = kBarOffset + 512 + 1024;
    // tensor memory: two accumulators, then per stage the scale columns of A, x_hi, x_lo
    static constexpr uint32_t kSfCols = 4 + 2 * (kSfX / 128);
    static constexpr uint32_t kSfCol0 = 2 * BN;
    static constexpr uint32_t kCols = kSfCol0 + kStages * kSfCols <= 128 ? 128 : kSfCol0 + kStages * kSfCols <= 256 ? 256 : 512;
    static_assert(kSmemBytes <= 227u * 1024u && kSfCol0 + kStages * kSfCols <= 512);
};

struct MxBars {
    // the pair's, in its even CTA: full, accum_empty; commits arrive in both CTAs
    uint64_t full[6];            // the stage's four producer warps of both CTAs + the loader's expect_tx
    uint64_t empty[6];           // the issuing warp's commit
    uint64_t full_w[4];          // raw slots: a copy-completion arrival per fetch thread
    uint64_t empty_w[4];         // all producer warps
    uint64_t accum_full[2];
    uint64_t accum_empty[2];     // one arrival per epilogue warp of both CTAs
    uint32_t tmem_base;
    volatile uint32_t failed;
};

struct MxArgs {
    MxGemm p;
    uint32_t rows, row_tiles;
};

__device__ __forceinline__ uint4 mx_tile(const MxGemm& p, const uint4* tiles, uint32_t t) {
    if (p.dense_n) return make_uint4(0u, t * p.dense_tile, min(p.dense_tile, p.dense_n - t * p.dense_tile), 0u);
    return __ldg(&tiles[t]);
}

// Shared-memory descriptor of a scale atom for tcgen05.cp: 32 rows of 16 bytes, no swizzle, 8-row groups 128 bytes
// apart.
__device__ __forceinline__ uint64_t sf_desc(uint32_t saddr) {
    const uint32_t lo = ((saddr >> 4) & 0x3FFFu) | (1u << 16);
    const uint32_t hi = (128u >> 4) | (1u << 14);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ void tmem_cp_sf(uint32_t tmem_col, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_col), "l"(desc) : "memory");
}

// Instruction descriptor of the block-scaled MMA: A = E2M1, B = E4M3, both K-major, E8M0 scales, M = 256, N = cols,
// K = 32; sf: which byte of the scale words this step uses.
__device__ __forceinline__ uint32_t mx_idesc(uint32_t cols, uint32_t sf) {
    return (sf << 4) | (5u << 7) | (0u << 10) | ((cols >> 3) << 17) | (1u << 23) | ((256u >> 4) << 24) | (sf << 29);
}
__device__ __forceinline__ void umma_mx(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                        uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
        : "memory");
}

// Eight nibble bytes of a block (two words) -> the four bytes of the low nibbles and of the high nibbles, two
// consecutive elements per byte, the lower element in the low nibble.
__device__ __forceinline__ void repack8(uint32_t q0, uint32_t q1, uint32_t& lo, uint32_t& hi) {
    const uint32_t even = __byte_perm(q0, q1, 0x6420), odd = __byte_perm(q0, q1, 0x7531);
    lo = (even & 0x0F0F0F0Fu) | ((odd << 4) & 0xF0F0F0F0u);
    hi = ((even >> 4) & 0x0F0F0F0Fu) | (odd & 0xF0F0F0F0u);
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// kTma: the raw bytes come by TMA. Eight rows are a multiple of 16 bytes (K % 64 == 0), so the matrix is a tensor of
// eight-row groups, and the segments of the rows c, c + 8, c + 16, .. of a tile are a box: eight boxes of 16 rows a unit,
// kept in the raw slot by c.
template <int BN, bool kTma>
__global__ void __launch_bounds__(kMxThreads, 1)
mx_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_sf,
               const __grid_constant__ CUtensorMap tmap_w, const MxArgs args) {
    // everything this kernel reads but the weights comes from the kernels before it
    chain_wait();
    const MxArgs& g = args;
    const uint32_t* header = g.p.header;
    const uint4* tiles = g.p.tiles;
    const uint32_t* list = g.p.list;
    after_wait(header);
    after_wait(tiles);
    after_wait(list);
    using T = MxTile<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    MxBars* bars = reinterpret_cast<MxBars*>(smem + T::kBarOffset);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t n_items = (g.p.dense_n ? (g.p.dense_n + g.p.dense_tile - 1) / g.p.dense_tile : header[0]) * g.row_tiles;
    const uint32_t nb = g.p.K >> 5;                        // blocks per row
    const int n_stages = (int)((nb + 3) >> 2);             // the last one may hold fewer than four blocks
    const uint64_t row_bytes = (uint64_t)nb * 17u;
    const uint32_t rank = cluster_ctarank(), step = gridDim.x >> 1;
    // The CTA's 128 rows of item w; a CTA wholly past M repeats the last ones (computed, dropped).
    auto first_row = [&](uint32_t w) { return min(((w % g.row_tiles) * 2 + rank) * (uint32_t)kBM, (g.p.M - 1) & ~(kBM - 1u)); };

    if (tid == 0) {
        for (int s = 0; s < T::kStages; ++s) {
            mbar_init(&bars->full[s], 2 * kMxGroupWarps + 1);
            mbar_init(&bars->empty[s], 1);
        }
        for (uint32_t s = 0; s < T::kRawSlots; ++s) {
            mbar_init(&bars->full_w[s], kTma ? 4 : kMxFetchWarps * 32);
            mbar_init(&bars->empty_w[s], kMxGroups * kMxGroupWarps);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars->accum_full[s], 1);
            mbar_init(&bars->accum_empty[s], 8);
        }
        bars->failed = 0;
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                     "r"(T::kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem = warp_uniform(bars->tmem_base);

    if (warp == 0 && rank == 0) {
        // ---- scale copies + MMA issuer of the pair (the converged warp walks, one elected lane issues) ----
        uint32_t st = 0, ph = 0, i = 0;
        bool ok = true;
        for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step, ++i) {
            const uint32_t ab = i & 1;
            // as many columns as the tile has tokens (N of a pair's MMA in steps of 32)
            const uint32_t cols = warp_uniform((mx_tile(g.p, tiles, w / g.row_tiles).z + 31u) & ~31u);
            ok = warp_poll(smem_u32(&bars->accum_empty[ab]), ((i >> 1) & 1) ^ 1, bars, g.p.status, 141);
            if (!ok) break;
            tc_fence_after();
            for (int s = 0; s < n_stages; ++s) {
                ok = warp_poll(smem_u32(&bars->full[st]), ph, bars, g.p.status, 142);
                if (!ok) break;
                tc_fence_after();
                const uint32_t stage = smem_u32(smem) + st * T::kStageBytes;
                const uint32_t sf_a = tmem + T::kSfCol0 + st * T::kSfCols, sf_hi = sf_a + 4, sf_lo = sf_hi + T::kSfX / 128;
                const uint64_t dsf = sf_desc(stage + T::kSfOffset);
                const uint64_t da = smem_desc(stage), dh = smem_desc(stage + kMxABytes);
                const int steps = min(4, (int)nb - 4 * s);
                if (elect_one()) {
                    tmem_cp_sf(sf_a, dsf);
                    tmem_cp_sf(sf_hi, dsf + kMxAtom / 16);
                    tmem_cp_sf(sf_lo, dsf + (kMxAtom + T::kSfX) / 16);
                    if constexpr (BN > 128) {  // the scales of tokens 128 and up
                        if (cols > 128) {
                            tmem_cp_sf(sf_hi + 4, dsf + 2 * kMxAtom / 16);
                            tmem_cp_sf(sf_lo + 4, dsf + (2 * kMxAtom + T::kSfX) / 16);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (k == steps) break;
                        umma_mx(tmem + ab * BN, da + 2 * k, dh + 2 * k, mx_idesc(cols, k), sf_a, sf_hi, (s | k) ? 1u : 0u);
                        umma_mx(tmem + ab * BN, da + 2 * k, dh + T::kXBytes / 16 + 2 * k, mx_idesc(cols, k), sf_a, sf_lo, 1u);
                    }
                    umma_commit_pair(&bars->empty[st]);
                    if (s + 1 == n_stages) umma_commit_pair(&bars->accum_full[ab]);
                }
                if (++st == T::kStages) {
                    st = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 1 || warp == 3) {
        if (lane == 0) {  // ---- loaders of the activation terms ----
            uint32_t st = 0, ph = 1;
            bool ok = true;
            const uint32_t term = warp == 1 ? 0u : 1u;
            for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step) {
                const uint4 tile = mx_tile(g.p, tiles, w / g.row_tiles);
                // the CTA's half of the columns
                const int y = (int)(term * g.rows + tile.y + rank * (((tile.z + 31u) & ~31u) >> 1));
                for (int s = 0; s < n_stages; ++s) {
                    ok = poll_or_fail(&bars->empty[st], ph, bars, g.p.status, 143);
                    if (!ok) break;
                    if (rank == 0 && term == 0) mbar_expect_tx(&bars->full[st], 2 * (2 * T::kXBytes + 2 * T::kSfX));  // of both CTAs
                    tma_load_2d_pair(smem + st * T::kStageBytes + kMxABytes + term * T::kXBytes, &tmap_x, s * kMxStageK, y,
                                     leader_addr(&bars->full[st]));
                    if (++st == T::kStages) {
                        st = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 4) {
        if (lane == 0) {  // ---- loader of the activations' scale atoms ----
            uint32_t st = 0, ph = 1;
            bool ok = true;
            for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step) {
                const uint32_t sf = w / g.row_tiles * (uint32_t)n_stages;
                for (int s = 0; s < n_stages; ++s) {
                    ok = poll_or_fail(&bars->empty[st], ph, bars, g.p.status, 148);
                    if (!ok) break;
                    tma_load_2d_pair(smem + st * T::kStageBytes + T::kSfOffset + kMxAtom, &tmap_sf, 0, (int)((sf + s) * (T::kSfX / 128)),
                                     leader_addr(&bars->full[st]));
                    if (++st == T::kStages) {
                        st = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (kTma && (warp == 2 || (warp >= kMxFetchWarp0 && warp < kMxFetchWarp0 + 3))) {
        if (lane == 0) {  // ---- loaders of the raw bytes, two boxes each ----
            const uint32_t c0 = warp == 2 ? 0u : 2u * (uint32_t)(warp - kMxFetchWarp0 + 1);
            uint32_t slot = 0, ph = 1;
            bool ok = true;
            for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step) {
                const int expert = (int)mx_tile(g.p, tiles, w / g.row_tiles).x, group = (int)(first_row(w) / 8);
                for (int s = 0; s < n_stages; s += (int)kMxUnit) {
                    ok = poll_or_fail(&bars->empty_w[slot], ph, bars, g.p.status, 146);
                    if (!ok) break;
                    uint8_t* const raw = smem + T::kRawOffset + slot * kMxRawSlot;
                    mbar_expect_tx(&bars->full_w[slot], kMxRawSlot / 4);
#pragma unroll
                    for (uint32_t c = c0; c < c0 + 2; ++c)
                        tma_load_3d(raw + c * (kMxRawSlot / 8), &tmap_w, (int)((c * (uint32_t)row_bytes + (uint32_t)s * 68u) & ~15u), group,
                                    expert, &bars->full_w[slot]);
                    if (++slot == T::kRawSlots) {
                        slot = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (!kTma && warp >= kMxFetchWarp0 && warp < kMxProdWarp0) {
        // ---- fetchers: the 16-byte pieces of all rows dealt to the threads row by row; rows past M repeat the last one
        // (computed, dropped); bytes past the matrix are zeros, not read ----
        const uint8_t* const end = g.p.A + g.p.a_bytes;
        uint32_t slot = 0, ph = 1;
        bool ok = true;
        for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step) {
            const uint32_t m0 = first_row(w);
            const uint8_t* rows = g.p.A + (uint64_t)mx_tile(g.p, tiles, w / g.row_tiles).x * g.p.expert_stride + (uint64_t)m0 * row_bytes;
            for (int s = 0; s < n_stages; s += (int)kMxUnit) {
                ok = poll_or_fail(&bars->empty_w[slot], ph, bars, g.p.status, 149);
                if (!ok) break;
                uint8_t* const raw = smem + T::kRawOffset + slot * kMxRawSlot;
                const uint32_t need = 68u * (uint32_t)min((int)kMxUnit, n_stages - s);
#pragma unroll 2
                for (uint32_t idx = (uint32_t)tid - kMxFetchWarp0 * 32; idx < kBM * kMxPieces; idx += kMxFetchWarps * 32) {
                    const uint32_t r = idx / kMxPieces, piece = (idx - r * kMxPieces) * 16;
                    const uint32_t o = min(r, g.p.M - 1 - m0) * (uint32_t)row_bytes + (uint32_t)s * 68u;
                    if (piece >= (o & 15u) + need) continue;
                    const uint8_t* sp = rows + (o & ~15u) + piece;
                    const uint32_t n = sp + 16 <= end ? 16u : (sp < end ? (uint32_t)(end - sp) : 0u);
                    cp_async16_zfill(raw + r * kMxRawRow + piece, n ? sp : g.p.A, n);
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bars->full_w[slot])) : "memory");
                if (++slot == T::kRawSlots) {
                    slot = 0;
                    ph ^= 1;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp >= kMxProdWarp0 && warp < kMxEpiWarp0) {
        // ---- weight producers: group = stage slot, thread = weight row; four blocks (68 bytes) per stage ----
        const uint32_t p = (uint32_t)(tid - kMxProdWarp0 * 32) & 127u, grp = (uint32_t)(warp - kMxProdWarp0) / kMxGroupWarps;
        // kTma: eight lanes take eight different c (distinct swizzles in the stage) of eight different groups (distinct banks
        // in the raw slot)
        const uint32_t row = kTma ? ((((p & 7u) + (p >> 3)) & 15u) << 3) | (p & 7u) : p;
        const uint32_t raw_at = kTma ? (row & 7u) * (kMxRawSlot / 8) + (row >> 3) * kMxRawRow : row * kMxRawRow;
        // Every group meets every unit and takes one of its stages, the one that is its turn among all stages (the last
        // unit of a row may hold none for it).
        bool dead = false;
        uint32_t st = grp, ph = 1, slot = 0, slot_ph = 0, turn = grp;
        for (uint32_t w = blockIdx.x >> 1; w < n_items; w += step) {
          const uint32_t row_off = (kTma ? row & 7u : min(row, g.p.M - 1 - first_row(w))) * (uint32_t)row_bytes;
          for (int u = 0; u < n_stages; u += (int)kMxUnit) {
            const int s = u + (int)turn;
            const int blocks = (int)nb - 4 * s;  // of the stage: four or, at the end of a row, fewer
            const uint32_t off = ((row_off + (uint32_t)u * 68u) & 15u) + turn * 68u;
            if (!dead) dead = !poll_or_fail(&bars->full_w[slot], slot_ph, bars, g.p.status, 147);
            // the row's 68 bytes: 8-byte reads from the offset rounded down to 8, then shifted to the first byte
            uint32_t v[20], wd[18];
            const uint8_t* src = smem + T::kRawOffset + slot * kMxRawSlot + raw_at + (off & ~7u);
#pragma unroll
            for (int k = 0; k < 10; ++k) {
                const uint2 t = *reinterpret_cast<const uint2*>(src + 8 * k);
                v[2 * k] = t.x;
                v[2 * k + 1] = t.y;
            }
            release_after((v[0] ^ v[2] ^ v[4]) ^ (v[6] ^ v[8] ^ v[10]) ^ (v[12] ^ v[14] ^ v[16]) ^ v[18], &bars->empty_w[slot], lane);
            if (++slot == T::kRawSlots) {
                slot = 0;
                slot_ph ^= 1;
            }
            if (s >= n_stages) continue;
            if (off & 4u) {
#pragma unroll
                for (int k = 0; k < 19; ++k) v[k] = v[k + 1];
            }
#pragma unroll
            for (int k = 0; k < 18; ++k) wd[k] = __funnelshift_r(v[k], v[k + 1], (off & 3u) * 8u);
            if (!dead) dead = !poll_or_fail(&bars->empty[st], ph, bars, g.p.status, 144);
            if (!dead) {
                uint8_t* stage = smem + st * T::kStageBytes;
                uint8_t* rowp = stage + row * 128;
                const uint32_t sw = row & 7;
                uint32_t sf = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    // block b: scale byte at 17 b, nibble bytes 17 b + 1 .. 17 b + 16
                    constexpr int kW[4] = {0, 4, 8, 13};
                    constexpr int kS[4] = {8, 16, 24, 0};
                    uint32_t q[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        q[i] = kS[b] ? __funnelshift_r(wd[kW[b] + i], wd[kW[b] + i + 1], kS[b]) : wd[kW[b] + i];
                    uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
                    repack8(q[0], q[1], lo.x, hi.x);
                    repack8(q[2], q[3], lo.y, hi.y);
                    *reinterpret_cast<uint4*>(rowp + (((2 * b) ^ sw) << 4)) = lo;
                    *reinterpret_cast<uint4*>(rowp + (((2 * b + 1) ^ sw) << 4)) = hi;
                    sf |= ((wd[(17 * b) >> 2] >> (8 * ((17 * b) & 3))) & 0xFFu) << (8 * b);
                }
                // a short stage: neutral scales (its missing blocks take part in no MMA)
                if (blocks < 4) sf = (sf & ((1u << (8 * blocks)) - 1u)) | (0x7F7F7F7Fu << (8 * blocks));
                *reinterpret_cast<uint32_t*>(stage + T::kSfOffset + (row & 31) * 16 + (row >> 5) * 4) = sf;
                fence_proxy_async();
            }
            __syncwarp();
            if (lane == 0 && !dead) mbar_arrive_cluster(leader_addr(&bars->full[st]));
            st += kMxGroups;
            if (st >= T::kStages) {
                st -= T::kStages;
                ph ^= 1;
            }
          }
          turn = (turn + 2 * (uint32_t)n_stages) % kMxGroups;  // minus the item's stages
        }
    } else if (warp >= kMxEpiWarp0) {
        // ---- epilogue: lane = weight row, column = pair of the tile ----
        const uint32_t q = warp & 3;
        uint32_t i = 0;
        for (uint32_t w = blockIdx.x >> 1; w < n_items; w += step, ++i) {
            const uint32_t ab = i & 1;
            const uint32_t tt = w / g.row_tiles;
            const uint4 tile = mx_tile(g.p, tiles, tt);
            const uint32_t m = ((w - tt * g.row_tiles) * 2 + rank) * kBM + q * 32 + lane;
            if (!poll_or_fail(&bars->accum_full[ab], (i >> 1) & 1, bars, g.p.status, 145)) break;
            __syncwarp();
            tc_fence_after();
#pragma unroll 1
            for (uint32_t c = 0; c * 32 < tile.z; ++c) {
                uint32_t v[32];
                tmem_ld32(tmem + ((q * 32u) << 16) + ab * BN + c * 32, v);
                // pair of column c*32 + lane: its output row starts at Y + token * y_token_stride + slot * M
                const uint32_t idx = c * 32 + lane;
                const uint32_t pair = idx >= tile.z ? 0u : (g.p.dense_n ? tile.y + idx : __ldg(&list[tile.y + idx]));
                const uint32_t tok = pair / g.p.n_used;
                const uint64_t at = (uint64_t)tok * g.p.y_token_stride + (uint64_t)(pair - tok * g.p.n_used) * g.p.M;
                tmem_ld_wait();
#pragma unroll
                for (int jj = 0; jj < 32; ++jj) {
                    const uint64_t y = __shfl_sync(0xFFFFFFFFu, at, jj);
                    if (c * 32 + jj < tile.z && m < g.p.M) g.p.Y[y + m] = __uint_as_float(v[jj]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_addr(&bars->accum_empty[ab]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (bars->failed) {  // given up with copies in flight: let them land before the CTA's shared memory is another's
        for (int i = 0; i < 100; ++i) __nanosleep(1000);
    }
    cluster_sync_all();  // the peer's MMAs read this CTA's stages, its commits arrive here
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kCols) : "memory");
    }
}

// ---- activation split ---------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t scale_exp(float maxabs) {
    // power of two s = 2^(e - 127) with maxabs / s in [128, 256): inside E4M3's range (448), four bits kept
    const uint32_t E = (__float_as_uint(maxabs) >> 23) & 0xFFu;
    if (maxabs == 0.f) return 127u;
    return E < 8u ? 1u : (E - 7u > 254u ? 254u : E - 7u);
}
__device__ __forceinline__ float pow2_neg(uint32_t e) { return __uint_as_float((254u - e) << 23); }  // 2^(127 - e)
__device__ __forceinline__ float pow2_pos(uint32_t e) { return __uint_as_float(e << 23); }           // 2^(e - 127)


struct MxTerms {
    const void* X;           // f32 or bf16 [T][stride]
    uint32_t T, K, stride, n_used;
    const uint2* where;      // per (token, slot) pair: {row of the list, tile << 8 | place in the tile}, row 0xFFFFFFFF:
                             // not listed; nullptr: token t is row t, in tiles of `tile` tokens
    uint32_t tile;
    uint8_t* x;              // [2 * rows][K]: x_hi, then x_lo
    uint8_t* sf;
    uint32_t rows, sf_x;
};

// One warp per (token, 256 columns), eight columns per lane: four lanes a block, sixteen a scale atom's four blocks. A
// token's terms are made once and written to the rows of all its pairs. Bound: the bytes, and in a short warp the latencies in
// a row (token, place in the list, stores): the two reads go out together, conversions are made in pairs. 4096 rows of 2880
// columns 21 -> 17 us, 1024 tokens to four rows each 11 -> 9 (L2 cold; the bytes take 11 and 6).
template <bool kBf16>
__global__ void __launch_bounds__(256) mx_terms_kernel(const MxTerms a) {
    chain_wait();
    const uint32_t chunks = (a.K + 255) / 256, lane = threadIdx.x & 31;
    const uint32_t id = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (id >= a.T * chunks) return;
    const uint32_t t = id / chunks, col = (id - t * chunks) * 256 + lane * 8;
    const bool live = col < a.K;  // whole blocks: K % 32 == 0
    const uint2 first = a.where ? a.where[(size_t)t * a.n_used] : make_uint2(0u, 0u);  // on its way together with the token
    float v[8] = {};
    if (live) {
        if constexpr (kBf16) {
            const uint4 q = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.X) + (size_t)t * a.stride + col);
            const uint32_t ww[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[2 * j] = __uint_as_float(ww[j] << 16);
                v[2 * j + 1] = __uint_as_float(ww[j] & 0xFFFF0000u);
            }
        } else {
            const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(a.X) + (size_t)t * a.stride + col);
            const float4 q0 = src[0], q1 = src[1];
            const float f[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __bfloat162float(__float2bfloat16_rn(f[j]));
        }
    }
    // one term: four lanes' common power of two, eight E4M3 bytes, what is left over
    auto term = [&](uint2& bytes) -> uint32_t {
        float mx = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(v[j]));
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
        const uint32_t e = scale_exp(mx);
        const float inv = pow2_neg(e), s = pow2_pos(e);
        uint32_t w[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const uint32_t q = __nv_cvt_float2_to_fp8x2(make_float2(v[j] * inv, v[j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
            const float2 f = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)q, __NV_E4M3)));
            v[j] -= f.x * s;
            v[j + 1] -= f.y * s;
            w[j >> 2] |= q << (8 * (j & 3));
        }
        bytes = make_uint2(w[0], w[1]);
        // the atom's four scale bytes, on the lanes that start a block
        uint32_t word = e << (8 * ((lane >> 2) & 3));
        word |= __shfl_xor_sync(0xFFFFFFFFu, word, 4);
        word |= __shfl_xor_sync(0xFFFFFFFFu, word, 8);
        return word;
    };
    uint2 hi, lo;
    const uint32_t sf_hi = term(hi), sf_lo = term(lo);
    const uint32_t atoms = (a.K + 127) / 128;
    for (uint32_t u = 0; u < a.n_used; ++u) {
        uint32_t row = t, tile, place;
        if (a.where) {
            const uint2 at = u ? a.where[(size_t)t * a.n_used + u] : first;
            row = at.x;
            tile = at.y >> 8;
            place = at.y & 255u;
        } else {
            tile = t / a.tile;
            place = t - tile * a.tile;
        }
        if (row == 0xFFFFFFFFu || !live) continue;
        *reinterpret_cast<uint2*>(a.x + (size_t)row * a.K + col) = hi;
        *reinterpret_cast<uint2*>(a.x + ((size_t)a.rows + row) * a.K + col) = lo;
        if ((lane & 15) == 0) {
            uint8_t* sf = a.sf + ((size_t)tile * atoms + (col >> 7)) * 2 * a.sf_x + (place >> 7) * kMxAtom + (place & 31) * 16 +
                          ((place & 127) >> 5) * 4;
            *reinterpret_cast<uint32_t*>(sf) = sf_hi;
            *reinterpret_cast<uint32_t*>(sf + a.sf_x) = sf_lo;
        }
    }
}

template <int BN, bool kTma>
cudaError_t launch_gemm(const CUtensorMap& map, const CUtensorMap& sf, const CUtensorMap& w, const MxArgs& g, uint64_t items,
                        cudaStream_t s) {
    auto kern = mx_gemm_kernel<BN, kTma>;
    static std::atomic<uint64_t> attr_done{0};  // per device ordinal
    static std::atomic<int> max_pairs[64];
    if (cudaError_t e = ensure_dynamic_smem(kern, (int)MxTile<BN>::kSmemBytes, attr_done); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kMxThreads, 1, 1);
    cfg.dynamicSmemBytes = MxTile<BN>::kSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int pairs = max_pairs_of(kern, cfg, max_pairs);
    if (pairs < 1) return cudaErrorNotSupported;
    cfg.numAttrs = 2;
    cfg.gridDim = dim3(2 * (uint32_t)(items < (uint64_t)pairs ? items : (uint64_t)pairs), 1, 1);
    return cudaLaunchKernelEx(&cfg, kern, map, sf, w, g);
}

struct MxLayout {
    uint64_t sf, total;
    uint32_t sf_x;
};
MxLayout mx_layout(uint64_t rows, uint32_t K, uint64_t tiles, uint32_t bn) {
    MxLayout l;
    l.sf_x = bn > 128 ? 2 * kMxAtom : kMxAtom;
    l.sf = (2 * rows * K + 1023) & ~1023ull;
    l.total = l.sf + tiles * ((K + 127) / 128) * 2 * l.sf_x;
    return l;
}

// Tokens per tile of the plain GEMM: equal tiles of at most 160.
uint32_t dense_bn(uint32_t N) { return N <= 64 ? 64u : 160u; }
uint32_t dense_tile(uint32_t N) {
    const uint32_t n = (N + dense_bn(N) - 1) / dense_bn(N);
    return (N + n - 1) / n;
}

}  // namespace

uint64_t mx_bytes(uint64_t rows, uint32_t K, uint64_t tiles, uint32_t bn) { return mx_layout(rows, K, tiles, bn).total; }

cudaError_t launch_mx_terms(const void* X, bool bf16, uint32_t T, uint32_t K, uint32_t stride, uint32_t n_used,
                            const uint2* where, uint32_t tile, uint64_t rows, uint64_t tiles, uint32_t bn, uint8_t* ws,
                            cudaStream_t s) {
    const MxLayout l = mx_layout(rows, K, tiles, bn);
    const MxTerms a{X, T, K, stride, n_used, where, tile, ws, ws + l.sf, (uint32_t)rows, l.sf_x};
    const uint64_t warps = (uint64_t)T * ((K + 255) / 256);
    if (warps > 0x7FFFFFFFull) return cudaErrorNotSupported;
    return launch_chained(bf16 ? mx_terms_kernel<true> : mx_terms_kernel<false>, dim3((uint32_t)((warps + 7) / 8)), dim3(256), 0, s, a);
}

cudaError_t launch_mx_gemm(const MxGemm& p, uint64_t rows, uint64_t tiles, uint32_t bn, const uint8_t* ws, cudaStream_t s) {
    EncodeFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const MxLayout l = mx_layout(rows, p.K, tiles, bn);
    CUtensorMap map;
    const cuuint64_t dims[2] = {p.K, 2 * rows};
    const cuuint64_t strides[1] = {p.K};
    const cuuint32_t box[2] = {(cuuint32_t)kMxStageK, bn / 2};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(ws), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorNotSupported;
    // the scale atoms as rows of 256 bytes: a stage's two terms are one box
    CUtensorMap sf;
    const uint32_t atoms = (p.K + 127) / 128;
    const cuuint64_t sdims[2] = {256, tiles * atoms * (l.sf_x / 128)};
    const cuuint64_t sstrides[1] = {256};
    const cuuint32_t sbox[2] = {256, l.sf_x / 128};
    if (enc(&sf, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(ws) + l.sf, sdims, sstrides, sbox, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorNotSupported;
    const MxArgs g{p, (uint32_t)rows, (p.M + 255) / 256};
    const uint64_t items = tiles * g.row_tiles;
    // eight-row groups of whole 16-byte multiples, none of them reaching past the matrix
    const bool tma = p.K % 64 == 0 && p.M % 8 == 0;
    CUtensorMap w = map;
    if (tma) {
        const cuuint64_t group = (cuuint64_t)(p.K / 32) * 17 * 8;
        const cuuint64_t wdims[3] = {group, p.M / 8, p.dense_n ? 1u : p.n_experts};
        const cuuint64_t wstrides[2] = {group, p.dense_n ? group * (p.M / 8) : p.expert_stride};
        const cuuint32_t wbox[3] = {kMxRawRow, 16, 1};
        const cuuint32_t wstr[3] = {1, 1, 1};
        if (enc(&w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(p.A), wdims, wstrides, wbox, wstr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorNotSupported;
        return bn == 32   ? launch_gemm<32, true>(map, sf, w, g, items, s)
               : bn == 64 ? launch_gemm<64, true>(map, sf, w, g, items, s) : launch_gemm<160, true>(map, sf, w, g, items, s);
    }
    return bn == 32   ? launch_gemm<32, false>(map, sf, w, g, items, s)
           : bn == 64 ? launch_gemm<64, false>(map, sf, w, g, items, s) : launch_gemm<160, false>(map, sf, w, g, items, s);
}

uint64_t mul_mm_mx_workspace_bytes(uint32_t N, uint32_t K) {
    const uint32_t tile = N ? dense_tile(N) : 1;
    return mx_bytes(N, K, (N + tile - 1) / tile, dense_bn(N));
}

bool mul_mm_mx_eligible(uint32_t type, const uint8_t* A, const void* B, uint32_t N, uint32_t K, uint32_t stride_b,
                        const void* workspace, uint64_t workspace_size) {
    if (type != T_MXFP4 || (K & 31u) || K < 128 || N < 64) return false;
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255u) || workspace_size < mul_mm_mx_workspace_bytes(N, K)) return false;
    return !(reinterpret_cast<uintptr_t>(A) & 15u) && !(reinterpret_cast<uintptr_t>(B) & 15u) && !(stride_b & 7u);
}

cudaError_t launch_mul_mm_mx(const uint8_t* A, uint64_t a_bytes, const void* B, float* D, uint32_t M, uint32_t N,
                             uint32_t K, uint32_t stride_b, uint32_t stride_d, void* workspace, uint32_t* status,
                             cudaStream_t s, uint64_t* launches) {
    const uint32_t bn = dense_bn(N), tile = dense_tile(N), tiles = (N + tile - 1) / tile;
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    cudaError_t e = launch_mx_terms(B, true, N, K, stride_b, 1, nullptr, tile, N, tiles, bn, ws, s);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
    MxGemm p{};
    p.A = A;
    p.a_bytes = a_bytes;
    p.Y = D;
    p.M = M;
    p.K = K;
    p.n_used = 1;
    p.y_token_stride = stride_d;
    p.dense_n = N;
    p.dense_tile = tile;
    p.status = status;
    e = launch_mx_gemm(p, N, tiles, bn, ws, s);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

}  // namespace zc
