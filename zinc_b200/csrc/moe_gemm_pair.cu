// Grouped dequant-GEMM of the MoE prefill on CTA pairs: Q4_K and Q6_K expert stacks, tokens grouped by routed expert
// (moe_gemm_tc.cu makes the groups and packs the activations as bf16). An item is (a tile of up to BN of an expert's pairs,
// 256 weight rows); each CTA of a pair has 128 of the rows and half of the pairs (tcgen05.mma cta_group::2). A stage is 128
// columns: the weights as bf16 in tensor memory, written by eight producer warps (a thread per row, its own lane), two
// activation tiles in shared memory by TMA.
//
// Raw blocks (256 columns) come by TMA. Q4_K rows have a 16-byte pitch: one box of 128 rows. Q6_K rows have not, but eight
// of them have: the matrix is a tensor of eight-row groups, the segments of the rows c, c + 8, c + 16, .. of a tile are a
// box of 16, and the slot keeps them by c.
//
// What bounds it, with the 16 pairs an expert of 256 has at 512 tokens: the producers' integer pipe, 1650 (Q4_K) and 2200
// (Q6_K) cycles for 256 columns of 128 rows. On one-CTA tiles it was 2800: a third in the producers' own copies, which held
// up their stores, a third waiting for the one stage a warp had (layer 316 us, 242 on pairs). Through shared memory every
// bf16 weight was written there and read by the MMA, 1024 cycles at 128 bytes each (226 us with tensor memory). Q6_K rows
// are read four bytes at a time: no selection by the offset's bits, two rows to a bank at worst (down projection 96.6 ->
// 92.9 us; 8 bytes 98.4).
// Warp roles (25 warps): 0 MMA issuer, 1 and 3 loaders of the activations, 2 and 4 of raw blocks (a thread each), 5-20
// producers (group j of four warps = columns 64 j .. of every block, a thread per row), 21-24 epilogue.
// Every mbarrier wait is bounded; a wait that gives up records {1, site}, raises the CTA's flag, and every role drains to
// the common exit where tensor memory is released.
#include "kernels.h"
#include "tc_common.cuh"

namespace zc {
namespace {

constexpr int kPairProdWarp0 = 5, kPairEpiWarp0 = kPairProdWarp0 + 16;
constexpr int kPairThreads = (kPairEpiWarp0 + 4) * 32;

template <int TYPE, int BN>
struct PairTile {
    static constexpr uint32_t kXBytes = BN / 2 * 128;      // 64 columns of the CTA's half of the pairs
    static constexpr uint32_t kStageBytes = 2 * kXBytes;
    static constexpr int kStages = BN > 64 ? 4 : 6;
    static constexpr uint32_t kRawRow = TYPE == T_Q4_K ? 144 : 240;  // odd multiples of 16 (8 rows of 16-byte reads: all banks)
    static constexpr uint32_t kRawSlot = kBM * kRawRow;
    static constexpr uint32_t kRawOffset = kStages * kStageBytes;
    static constexpr uint32_t kRawSlots = 4;
    static constexpr uint32_t kBarOffset = kRawOffset + kRawSlots * kRawSlot;
    static constexpr uint32_t kSmemBytes = kBarOffset + 512 + 1024;
    // tensor memory: two accumulators, then the stages' weights (two bf16 a column)
    static constexpr uint32_t kACol0 = 2 * BN, kACols = 64;
    static_assert(kSmemBytes <= 227u * 1024u && kACol0 + kStages * kACols <= 512);
};

// D[tmem] (+)= A[tmem] * B[smem desc]^T of a CTA pair, bf16 x bf16 -> f32, issued by one thread
__device__ __forceinline__ void umma_bf16_pair_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

struct PairBars {
    // the pair's, in its even CTA: full, accum_empty; commits arrive in both CTAs
    uint64_t full[6];   // the stage's eight producer warps of both CTAs + the loader's expect_tx
    uint64_t empty[6];
    uint64_t full_w[4], empty_w[4];  // raw slots: the loaders' expect_tx; the sixteen producer warps
    uint64_t accum_full[2], accum_empty[2];
    uint32_t tmem_base;
    volatile uint32_t failed;
};

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// The weight row of a tile that lane l of tensor memory holds.
template <int TYPE>
__device__ __forceinline__ uint32_t pair_row(uint32_t l) {
    return TYPE == T_Q4_K ? l : (l & 64u) + 8u * (l & 7u) + ((l >> 3) & 7u);
}

template <int TYPE, int BN>
__global__ void __launch_bounds__(kPairThreads, 1)
moe_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const MoePair args) {
    // everything this kernel reads but the weights comes from the kernels before it
    chain_wait();
    const MoePair& g = args;
    const uint32_t* header = g.header;
    const uint4* tiles = g.tiles;
    const uint32_t* list = g.list;
    after_wait(header);
    after_wait(tiles);
    after_wait(list);
    using T = PairTile<TYPE, BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    PairBars* bars = reinterpret_cast<PairBars*>(smem + T::kBarOffset);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t row_tiles = (g.M + 255) / 256, n_items = header[0] * row_tiles;
    const int nblk = (int)(g.K >> 8);
    const uint32_t row_bytes = (uint32_t)nblk * Raw<TYPE>::kBlock;
    const uint32_t rank = cluster_ctarank(), step = gridDim.x >> 1;

    if (tid == 0) {
        for (int s = 0; s < T::kStages; ++s) {
            mbar_init(&bars->full[s], 17);
            mbar_init(&bars->empty[s], 1);
        }
        for (uint32_t s = 0; s < T::kRawSlots; ++s) {
            mbar_init(&bars->full_w[s], TYPE == T_Q4_K ? 1 : 2);
            mbar_init(&bars->empty_w[s], 16);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars->accum_full[s], 1);
            mbar_init(&bars->accum_empty[s], 8);  // the epilogue warps of both CTAs
        }
        bars->failed = 0;
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem = warp_uniform(bars->tmem_base);

    if (warp == 0 && rank == 0) {
        // ---- MMA issuer of the pair (the converged warp walks, one elected lane issues) ----
        uint32_t st = 0, ph = 0, i = 0;
        bool ok = true;
        for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step, ++i) {
            const uint32_t ab = i & 1;
            // as many columns as the tile has pairs (N of a pair's MMA in steps of 32)
            const uint32_t cols = warp_uniform((__ldg(&tiles[w / row_tiles]).z + 31u) & ~31u);
            const uint32_t idesc = instr_desc_pair<32>() + ((cols - 32u) >> 3 << 17);
            ok = warp_poll(smem_u32(&bars->accum_empty[ab]), ((i >> 1) & 1) ^ 1, bars, g.status, 161);
            if (!ok) break;
            tc_fence_after();
            for (int s = 0; s < 2 * nblk; ++s) {
                ok = warp_poll(smem_u32(&bars->full[st]), ph, bars, g.status, 162);
                if (!ok) break;
                tc_fence_after();
                const uint64_t dx = smem_desc(smem_u32(smem) + st * T::kStageBytes);
                const uint32_t a = tmem + T::kACol0 + st * T::kACols;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)  // 16 columns a time; the activations are two tiles of 64
                        umma_bf16_pair_ta(tmem + ab * BN, a + 8 * k, dx + (k >> 2) * (T::kXBytes / 16) + 2 * (k & 3), idesc, (uint32_t)(s | k));
                    umma_commit_pair(&bars->empty[st]);
                    if (s + 1 == 2 * nblk) umma_commit_pair(&bars->accum_full[ab]);
                }
                if (++st == T::kStages) {
                    st = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 1 || warp == 3) {
        if (lane == 0) {  // ---- loaders of the activations: a tile of 64 columns of every stage each ----
            uint32_t st = 0, ph = 1;
            bool ok = true;
            const uint32_t half = warp == 1 ? 0u : 1u;
            for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step) {
                const uint4 tile = __ldg(&tiles[w / row_tiles]);
                const int y = (int)(tile.y + rank * (((tile.z + 31u) & ~31u) >> 1));  // the CTA's half of the columns
                for (int s = 0; s < 2 * nblk; ++s) {
                    ok = poll_or_fail(&bars->empty[st], ph, bars, g.status, 163);
                    if (!ok) break;
                    if (rank == 0 && half == 0) mbar_expect_tx(&bars->full[st], 4 * T::kXBytes);  // of both CTAs
                    tma_load_2d_pair(smem + st * T::kStageBytes + half * T::kXBytes, &tmap_x, s * 128 + (int)half * 64, y,
                                     leader_addr(&bars->full[st]));
                    if (++st == T::kStages) {
                        st = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 2 || (warp == 4 && TYPE != T_Q4_K)) {
        if (lane == 0) {  // ---- loaders of the raw blocks ----
            uint32_t slot = 0, ph = 1;
            bool ok = true;
            for (uint32_t w = blockIdx.x >> 1; w < n_items && ok; w += step) {
                const uint32_t t = w / row_tiles;
                const int expert = (int)__ldg(&tiles[t]).x, m0 = (int)(((w - t * row_tiles) * 2 + rank) * kBM);  // rows past M: zeros
                for (int b = 0; b < nblk; ++b) {
                    ok = poll_or_fail(&bars->empty_w[slot], ph, bars, g.status, 164);
                    if (!ok) break;
                    uint8_t* const raw = smem + T::kRawOffset + slot * T::kRawSlot;
                    if constexpr (TYPE == T_Q4_K) {
                        mbar_expect_tx(&bars->full_w[slot], T::kRawSlot);
                        tma_load_3d(raw, &tmap_w, b * 144, m0, expert, &bars->full_w[slot]);
                    } else {
                        const uint32_t c0 = warp == 2 ? 0u : 4u;
                        mbar_expect_tx(&bars->full_w[slot], T::kRawSlot / 2);
#pragma unroll
                        for (uint32_t c = c0; c < c0 + 4; ++c)
                            tma_load_3d(raw + c * (T::kRawSlot / 8), &tmap_w, (int)((c * row_bytes + (uint32_t)b * 210u) & ~15u), m0 / 8, expert,
                                        &bars->full_w[slot]);
                    }
                    if (++slot == T::kRawSlots) {
                        slot = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp >= kPairProdWarp0 && warp < kPairEpiWarp0) {
        // ---- producers ----
        // A thread's row goes to its own lane of tensor memory. Q6_K: eight lanes take the same c of eight groups (distinct
        // banks in the raw slot).
        const uint32_t q = (uint32_t)(warp - kPairProdWarp0) >> 2, row = pair_row<TYPE>((uint32_t)((warp & 3) * 32 + lane));
        const uint32_t raw_at = TYPE == T_Q4_K ? row * T::kRawRow : (row & 7u) * (T::kRawSlot / 8) + (row >> 3) * T::kRawRow;
        const uint32_t row_off = (row & 7u) * row_bytes;  // eight rows are a multiple of 16 bytes
        const uint32_t lane_col = tmem + (((uint32_t)(warp & 3) * 32u) << 16) + T::kACol0 + (q & 1u) * (T::kACols / 2);
        uint32_t st = q >> 1, ph = 1, slot = 0, slot_ph = 0;
        bool dead = false;
        for (uint32_t w = blockIdx.x >> 1; w < n_items; w += step) {
            for (int b = 0; b < nblk; ++b) {
                if (!dead) dead = !poll_or_fail(&bars->full_w[slot], slot_ph, bars, g.status, 165);
                const uint8_t* raw = smem + T::kRawOffset + slot * T::kRawSlot + raw_at;
                uint32_t o[32];
                auto put = [&](int c, const uint4& v) {
                    o[4 * c] = v.x;
                    o[4 * c + 1] = v.y;
                    o[4 * c + 2] = v.z;
                    o[4 * c + 3] = v.w;
                };
                if constexpr (TYPE == T_Q4_K) {
                    const uint4 hd = *reinterpret_cast<const uint4*>(raw);
                    const uint4 c0 = *reinterpret_cast<const uint4*>(raw + 16 + q * 32);
                    const uint4 c1 = *reinterpret_cast<const uint4*>(raw + 32 + q * 32);
                    release_after(hd.x ^ c0.x ^ c1.x, &bars->empty_w[slot], lane);
                    const GroupQ4k k = group_q4k(hd, q);
                    dequant_group_q4k(c0, c1, k.s_lo, k.m_lo, k.s_hi, k.m_hi, put);
                } else {
                    dequant_group_q6k<4>(raw, (row_off + (uint32_t)b * 210u) & 15u, (int)q, put);
                    // words 4 k + 3 are made of every word read but the first ones of ql and qh, which word 0 is made of
                    release_after(o[0] ^ o[3] ^ o[7] ^ o[11] ^ o[15] ^ o[19] ^ o[23] ^ o[27] ^ o[31], &bars->empty_w[slot], lane);
                }
                if (!dead) dead = !poll_or_fail(&bars->empty[st], ph, bars, g.status, 166);
                __syncwarp();
                tc_fence_after();
                if (!__any_sync(0xFFFFFFFFu, dead)) {
                    tmem_st32(lane_col + st * T::kACols, o);
                    tmem_st_wait();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0 && !dead) mbar_arrive_cluster(leader_addr(&bars->full[st]));
                st += 2;
                if (st >= T::kStages) {
                    st -= T::kStages;
                    ph ^= 1;
                }
                if (++slot == T::kRawSlots) {
                    slot = 0;
                    slot_ph ^= 1;
                }
            }
        }
    } else if (warp >= kPairEpiWarp0) {
        // ---- epilogue: lane = weight row, column = pair of the tile ----
        const uint32_t q = warp & 3;
        uint32_t i = 0;
        for (uint32_t w = blockIdx.x >> 1; w < n_items; w += step, ++i) {
            const uint32_t ab = i & 1, t = w / row_tiles;
            const uint4 tile = __ldg(&tiles[t]);
            const uint32_t m = ((w - t * row_tiles) * 2 + rank) * kBM + pair_row<TYPE>(q * 32 + lane);
            // pair of column c*32 + lane: its output row starts at Y + token * y_token_stride + slot * M
            auto place = [&](uint32_t c) {
                const uint32_t idx = c * 32 + lane, pair = idx >= tile.z ? 0u : __ldg(&list[tile.y + idx]);
                const uint32_t tok = pair / g.n_used;
                return (uint64_t)tok * g.y_token_stride + (uint64_t)(pair - tok * g.n_used) * g.M;
            };
            uint64_t at = place(0);  // fetched while the accumulator is on its way
            if (!poll_or_fail(&bars->accum_full[ab], (i >> 1) & 1, bars, g.status, 167)) break;
            __syncwarp();
            tc_fence_after();
#pragma unroll 1
            for (uint32_t c = 0; c * 32 < tile.z; ++c) {
                uint32_t v[32];
                tmem_ld32(tmem + ((q * 32u) << 16) + ab * BN + c * 32, v);
                if (c) at = place(c);
                tmem_ld_wait();
#pragma unroll
                for (int jj = 0; jj < 32; ++jj) {
                    if (jj % 8 == 0 && c * 32 + jj >= tile.z) break;
                    const uint64_t y = __shfl_sync(0xFFFFFFFFu, at, jj);
                    if (c * 32 + jj < tile.z && m < g.M) g.Y[y + m] = __uint_as_float(v[jj]);
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
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

template <int TYPE, int BN>
cudaError_t launch_pair(const CUtensorMap& x, const CUtensorMap& w, const MoePair& g, uint64_t items, cudaStream_t s) {
    using T = PairTile<TYPE, BN>;
    auto kern = moe_pair_kernel<TYPE, BN>;
    static std::atomic<uint64_t> attr_done{0};  // per device ordinal
    static std::atomic<int> max_pairs[64];
    if (cudaError_t e = ensure_dynamic_smem(kern, (int)T::kSmemBytes, attr_done); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kPairThreads, 1, 1);
    cfg.dynamicSmemBytes = T::kSmemBytes;
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
    return cudaLaunchKernelEx(&cfg, kern, x, w, g);
}

}  // namespace

bool moe_pair_eligible(uint32_t type, uint32_t M, uint32_t K) {
    return (type == T_Q4_K || (type == T_Q6_K && M % 8 == 0)) && K % 256 == 0 && (uint64_t)(K / 256) * 210 * 8 < (1u << 31);
}

cudaError_t launch_moe_pair(uint32_t type, const MoePair& g, const void* xp, uint64_t n_pairs, uint64_t max_tiles, uint32_t bn,
                            cudaStream_t s) {
    EncodeFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    CUtensorMap x, w;
    const cuuint64_t xd[2] = {g.K, n_pairs}, xs[1] = {(cuuint64_t)g.K * 2};
    const cuuint32_t xb[2] = {kBK, bn / 2}, one[3] = {1, 1, 1};
    if (enc(&x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(xp), xd, xs, xb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorNotSupported;
    const cuuint64_t row = (cuuint64_t)(g.K / 256) * (type == T_Q4_K ? 144 : 210);
    const bool rows = type == T_Q4_K;
    const cuuint64_t wd[3] = {rows ? row : 8 * row, rows ? g.M : g.M / 8, g.n_experts}, ws[2] = {rows ? row : 8 * row, g.expert_stride};
    const cuuint32_t wb[3] = {rows ? 144u : 240u, rows ? (cuuint32_t)kBM : 16u, 1};
    if (enc(&w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(g.A), wd, ws, wb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorNotSupported;
    const uint64_t items = max_tiles * ((g.M + 255) / 256);
    if (type == T_Q4_K)
        return bn == 32   ? launch_pair<T_Q4_K, 32>(x, w, g, items, s)
               : bn == 64 ? launch_pair<T_Q4_K, 64>(x, w, g, items, s) : launch_pair<T_Q4_K, 128>(x, w, g, items, s);
    return bn == 32   ? launch_pair<T_Q6_K, 32>(x, w, g, items, s)
           : bn == 64 ? launch_pair<T_Q6_K, 64>(x, w, g, items, s) : launch_pair<T_Q6_K, 128>(x, w, g, items, s);
}

}  // namespace zc
