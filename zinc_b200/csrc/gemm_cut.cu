// Prefill dequant-GEMM for few tiles: Q4_K and Q6_K weights, bf16 activations, K cut over the CTAs that the tiles leave idle.
// (src/compute/dmmv.zig:1045 recordMulMmQ4K; the large products take gemm_tc.cu.)
//
// A tile is 128 weight rows x up to 192 tokens. Its blocks of 256 columns are shared out over up to eight CTAs of a cluster, two
// clusters a tile at most; the CTAs of a cluster add up their parts through one another's shared memory, in their order, and the two
// clusters add to D, which a kernel in front has zeroed (two summands commute: the same bits every time). With one CTA a tile it stores.
// What bounds it: the producers (0.83 us a block of Q4_K, 1.39 of Q6_K) behind 3.3 us of launch, set-up and first copy, and 2 to 3 us for
// the zeroing kernel and the sums where K is cut. Against the kernels it stands in for, over 62 shapes between 256 x 1024 and 12288 x
// 12288 with 16 to 2048 tokens: 1.6 times as fast in the mean (0.98 at worst; figures at the rule below).
// Weights go from registers to tensor memory (the MMA takes A from there), activations by TMA, a stage is 128 columns; the raw blocks
// of Q6_K, whose rows have no 16-byte pitch, come as the rows c, c + 8, c + 16, .. of a tile in one box each, by a tensor map for each c
// (such rows lie eight rows' bytes apart, a multiple of 16), so that any number of rows can be described.
// Warp roles (20 warps): 0 MMA issuer, 1 loader of the activations, 2 and 3 of raw blocks, 4-19 producers (group j of four warps =
// columns 64 j .. of every block, a thread per row) and epilogue. Every mbarrier wait is bounded; a wait that gives up records {1, site},
// raises the flag of all CTAs of the cluster, none of which adds its sums then, and every role drains to the common exit, where copies
// and MMAs in flight are awaited and tensor memory is released.
#include <cstddef>

#include "kernels.h"
#include "tc_common.cuh"

namespace zc {
namespace {

constexpr int kCutProdWarp0 = 4, kCutThreads = (kCutProdWarp0 + 16) * 32;
constexpr uint32_t kCutMaxTokens = 192, kCutMaxStages = 4, kCutSmem = 227 * 1024, kCutBars = 512;

struct CutArgs {
    float* D;
    uint32_t M, N, nblk, stride_d;
    uint32_t tn, stages, raw_slots;   // tokens of a tile (a multiple of 16), stages, slots of raw blocks
    uint32_t parts, cluster;          // CTAs a tile; of them in a cluster
    uint32_t* status;
};
template <int TYPE>
struct CutMaps {
    CUtensorMap x;
    CUtensorMap w[TYPE == T_Q4_K ? 1 : 8];
};
template <int TYPE>
struct CutRaw {
    static constexpr uint32_t kRow = TYPE == T_Q4_K ? 144 : 240;  // odd multiples of 16 (8 rows of 16-byte reads: all banks)
    static constexpr uint32_t kSlot = kBM * kRow;
};

struct CutBars {
    uint64_t full[kCutMaxStages], full_x[kCutMaxStages], empty[kCutMaxStages];  // eight producer warps; the loader's expect_tx; a commit
    uint64_t full_w[2][4], empty_w[4];                    // raw slots: each loader's expect_tx; sixteen producer warps
    uint64_t accum, drained;
    uint32_t tmem_base;
    volatile uint32_t failed;
};
static_assert(sizeof(CutBars) <= kCutBars, "barriers");

// D[tmem] (+)= A[tmem] * B[smem desc]^T, bf16 x bf16 -> f32, issued by one thread
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t a, uint32_t rank) {
    float4 v;
    asm volatile(
        "{\n\t.reg .b32 r;\n\t"
        "mapa.shared::cluster.u32 r, %4, %5;\n\t"
        "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [r];\n\t}"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "r"(a), "r"(rank)
        : "memory");
    return v;
}
__device__ __forceinline__ void raise_cluster(volatile uint32_t* flag, uint32_t rank) {
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\tst.shared::cluster.u32 [r], %2;\n\t}" ::"r"(
                     smem_u32(const_cast<uint32_t*>(flag))),
                 "r"(rank), "r"(1u)
                 : "memory");
}
// The weight row of a tile that lane l of tensor memory holds: for Q6_K eight lanes take the same c of eight groups (distinct banks).
template <int TYPE>
__device__ __forceinline__ uint32_t cut_row(uint32_t l) {
    return TYPE == T_Q4_K ? l : (l & 64u) + 8u * (l & 7u) + ((l >> 3) & 7u);
}

// After a wait has given up: until the last copies into a ring of n slots have landed, of `issued` that one thread requested. (The
// barriers are arrived at by that thread only, so every copy's phase ends.)
__device__ __forceinline__ void cut_await_copies(uint64_t* bars, uint32_t n, uint32_t issued) {
    for (uint32_t i = issued > n ? issued - n : 0u; i < issued; ++i)
        for (uint32_t tries = 0; tries < kDrainLimit && !mbar_try_wait(&bars[i % n], (i / n) & 1); ++tries) {
        }
}

template <int TYPE>
__global__ void __launch_bounds__(kCutThreads, 1) gemm_cut_kernel(const __grid_constant__ CutMaps<TYPE> maps, const CutArgs g) {
    using R = CutRaw<TYPE>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t x_bytes = g.tn * 128u, stage_bytes = 2 * x_bytes;  // 64 columns; a stage
    uint8_t* const raw0 = smem + g.stages * stage_bytes;
    CutBars* bars = reinterpret_cast<CutBars*>(raw0 + g.raw_slots * R::kSlot);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t part = blockIdx.x, m0 = blockIdx.y * kBM, n0 = blockIdx.z * g.tn;
    const int b0 = (int)(part * g.nblk / g.parts), nb = (int)((part + 1) * g.nblk / g.parts) - b0;

    if (tid < (int)(offsetof(CutBars, tmem_base) / 8)) {  // a thread each
        static_assert(offsetof(CutBars, tmem_base) / 8 <= 32, "by the warp that goes on to the allocation");
        constexpr int kEmptyW = offsetof(CutBars, empty_w) / 8;
        mbar_init(bars->full + tid, tid < (int)kCutMaxStages ? 8u : tid >= kEmptyW && tid < kEmptyW + 4 ? 16u : 1u);
        if (tid == 0) bars->failed = 0;
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // Without a zeroing kernel in front (which has waited) the kernel before may still be running, and what it writes may be this one's
    // weights.
    if (g.parts == 1) chain_wait();
    chain_release();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = warp_uniform(bars->tmem_base), tmem_w = tmem + (g.tn <= 128 ? 128u : 256u);

    uint32_t requested = 0;  // copies, by a loader
    if (warp == 0) {
        // ---- MMA issuer (the converged warp walks, one elected lane issues) ----
        const uint32_t idesc = instr_desc<16>() + ((g.tn - 16u) >> 3 << 17);
        uint32_t st = 0, ph = 0;
        for (int s = 0; s < 2 * nb; ++s) {
            if (!warp_poll(smem_u32(lane == 1 ? &bars->full_x[st] : &bars->full[st]), ph, bars, g.status, 171)) break;
            tc_fence_after();
            const uint64_t dx = smem_desc(smem_u32(smem) + st * stage_bytes);
            const uint32_t a = tmem_w + st * 64;
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < 8; ++k)  // 16 columns a time; the activations are two tiles of 64
                    umma_bf16_ta(tmem, a + 8 * k, dx + (k >> 2) * (x_bytes / 16) + 2 * (k & 3), idesc, (uint32_t)(s | k));
                umma_commit(&bars->empty[st]);
                if (s + 1 == 2 * nb) umma_commit(&bars->accum);
            }
            if (++st == g.stages) {
                st = 0;
                ph ^= 1;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // ---- loader of the activations ----
            uint32_t st = 0, ph = 1;
            for (int s = 0; s < 2 * nb; ++s) {
                if (!poll_or_fail<true>(&bars->empty[st], ph, bars, g.status, 172)) break;
                mbar_expect_tx(&bars->full_x[st], stage_bytes);
                for (int h = 0; h < 2; ++h)
                    tma_load_2d(smem + st * stage_bytes + h * x_bytes, &maps.x, (b0 * 4 + s * 2 + h) * 64, (int)n0, &bars->full_x[st]);
                ++requested;
                if (++st == g.stages) {
                    st = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 2 || (warp == 3 && TYPE != T_Q4_K)) {
        if (lane == 0) {  // ---- loaders of the raw blocks; rows past M: zeros ----
            uint32_t slot = 0, ph = 1;
            uint64_t* const full_w = bars->full_w[warp - 2];
            for (int b = b0; b < b0 + nb; ++b) {
                if (!poll_or_fail<true>(&bars->empty_w[slot], ph, bars, g.status, 173)) break;
                uint8_t* const raw = raw0 + slot * R::kSlot;
                if constexpr (TYPE == T_Q4_K) {
                    mbar_expect_tx(&full_w[slot], R::kSlot);
                    tma_load_2d(raw, &maps.w[0], b * 144, (int)m0, &full_w[slot]);
                } else {
                    const uint32_t c0 = warp == 2 ? 0u : 4u, row_bytes = g.nblk * 210u;
                    mbar_expect_tx(&full_w[slot], R::kSlot / 2);
#pragma unroll
                    for (uint32_t c = c0; c < c0 + 4; ++c)
                        tma_load_2d(raw + c * (R::kSlot / 8), &maps.w[c], (int)((((c * row_bytes) & 15u) + (uint32_t)b * 210u) & ~15u), (int)(m0 / 8),
                                    &full_w[slot]);
                }
                ++requested;
                if (++slot == g.raw_slots) {
                    slot = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp >= kCutProdWarp0) {
        // ---- producers: a thread's row goes to its own lane of tensor memory ----
        const uint32_t q = (uint32_t)(warp - kCutProdWarp0) >> 2, quarter = (uint32_t)warp & 3u, row = cut_row<TYPE>(quarter * 32 + lane);
        const uint32_t raw_at = TYPE == T_Q4_K ? row * R::kRow : (row & 7u) * (R::kSlot / 8) + (row >> 3) * R::kRow;
        const uint32_t row_off = ((row & 7u) * g.nblk * 210u) & 15u;   // eight rows are a multiple of 16 bytes
        // Q6_K: the rows of a warp are of one loader's boxes
        uint64_t* const full_w = bars->full_w[TYPE == T_Q4_K ? 0 : (row & 7u) >> 2];
        const uint32_t lane_col = tmem_w + ((quarter * 32u) << 16) + (q & 1u) * 32;
        uint32_t st = (q >> 1) % g.stages, ph = 1, slot = 0, slot_ph = 0;
        bool dead = false;
        for (int b = b0; b < b0 + nb; ++b) {
            if (!dead) dead = !poll_or_fail<true>(&full_w[slot], slot_ph, bars, g.status, 174);
            const uint8_t* raw = raw0 + slot * R::kSlot + raw_at;
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
            if (!dead) dead = !poll_or_fail<true>(&bars->empty[st], ph, bars, g.status, 175);
            __syncwarp();
            tc_fence_after();
            if (!__any_sync(0xFFFFFFFFu, dead)) {
                tmem_st32(lane_col + st * 64, o);
                tmem_st_wait();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && !dead) mbar_arrive(&bars->full[st]);
            st += 2;
            if (st >= g.stages) {
                st -= g.stages;
                ph ^= 1;
            }
            if (++slot == g.raw_slots) {
                slot = 0;
                slot_ph ^= 1;
            }
        }
        // ---- the tile, or this CTA's part of it: lane = weight row, column = token ----
        if (!dead) dead = !poll_or_fail<true>(&bars->accum, 0, bars, g.status, 176);
        __syncwarp();
        tc_fence_after();
        dead = __any_sync(0xFFFFFFFFu, dead);
        const uint32_t tokens = min(g.tn, g.N - n0);
        float* const sums = reinterpret_cast<float*>(smem);  // [token][row], in the place of the stages: all of them have been read
        if (!dead) {
            const uint32_t m = m0 + row;
#pragma unroll 1
            for (uint32_t c = q; c * 32 < tokens; c += 4) {
                uint32_t v[32];
                tmem_ld32(tmem + ((quarter * 32u) << 16) + c * 32, v);
                tmem_ld_wait();
                if (g.parts == 1) {
                    if (m < g.M) {
                        float* d = g.D + (uint64_t)(n0 + c * 32) * g.stride_d + m;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (c * 32 + j < tokens) d[(uint64_t)j * g.stride_d] = __uint_as_float(v[j]);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (c * 32 + j < tokens) sums[(c * 32 + j) * kBM + row] = __uint_as_float(v[j]);
                }
            }
        }
    }
    if (g.parts > 1) {
        // ---- the parts of the cluster's CTAs, each CTA's share of the tokens, in the order of the parts ----
        if (g.cluster > 1) {
            if (bars->failed)
                for (uint32_t r = 0; r < g.cluster; ++r) raise_cluster(&bars->failed, r);
            __syncwarp();
            cluster_sync_all();
        } else {
            __syncthreads();
        }
        if (warp >= kCutProdWarp0) {
            chain_wait();  // D is zeroed
            const uint32_t tokens = min(g.tn, g.N - n0), rank = g.cluster > 1 ? cluster_ctarank() : 0u, pt = tid - kCutProdWarp0 * 32;
            const uint32_t t0 = tokens * rank / g.cluster, t1 = tokens * (rank + 1) / g.cluster;
            const bool vec = (g.stride_d & 3u) == 0 && (reinterpret_cast<uintptr_t>(g.D) & 15u) == 0;
            if (!bars->failed) {
                for (uint32_t i = t0 * 32 + pt; i < t1 * 32; i += 16 * 32) {
                    const uint32_t at = smem_u32(smem) + i * 16, m = m0 + (i & 31u) * 4;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (g.cluster == 1) {
                        v = *reinterpret_cast<const float4*>(smem + i * 16);
                    } else {
                        for (uint32_t r = 0; r < g.cluster; ++r) {
                            const float4 p = ld_cluster_f4(at, r);
                            v = make_float4(v.x + p.x, v.y + p.y, v.z + p.z, v.w + p.w);
                        }
                    }
                    float* d = g.D + (uint64_t)(n0 + (i >> 5)) * g.stride_d + m;
                    if (vec && m + 4 <= g.M) {
                        atomicAdd(reinterpret_cast<float4*>(d), v);
                    } else {
                        if (m < g.M) atomicAdd(d, v.x);
                        if (m + 1 < g.M) atomicAdd(d + 1, v.y);
                        if (m + 2 < g.M) atomicAdd(d + 2, v.z);
                        if (m + 3 < g.M) atomicAdd(d + 3, v.w);
                    }
                }
            }
            __syncwarp();
        }
    }
    chain_wait();
    tc_fence_before();
    __syncthreads();
    if (bars->failed) {  // nothing is in flight when shared and tensor memory become another's
        if (warp == 0) {
            if (elect_one()) umma_commit(&bars->drained);
            __syncwarp();
            for (uint32_t tries = 0; tries < kDrainLimit && !mbar_try_wait(&bars->drained, 0); ++tries) {
            }
        } else if (lane == 0 && warp == 1) {
            cut_await_copies(bars->full_x, g.stages, requested);
        } else if (lane == 0 && warp < kCutProdWarp0) {
            cut_await_copies(bars->full_w[warp - 2], g.raw_slots, requested);
        }
        __syncthreads();
    }
    if (g.cluster > 1) cluster_sync_all();  // the others read this CTA's sums
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// How the work is cut.
struct Cut {
    uint32_t tn, parts, cluster;
};

template <int TYPE>
cudaError_t launch_typed(const uint8_t* A, const void* B, float* D, uint32_t M, uint32_t N, uint32_t K, uint32_t stride_b, uint32_t stride_d,
                         const Cut& cut, uint32_t* status, cudaStream_t s, uint64_t* launches) {
    using R = CutRaw<TYPE>;
    EncodeFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    CutMaps<TYPE> maps;
    const cuuint32_t ones[2] = {1, 1};
    {
        const cuuint64_t dims[2] = {K, N}, strides[1] = {(cuuint64_t)stride_b * 2};
        const cuuint32_t box[2] = {64, cut.tn};
        if (enc(&maps.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(B), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorNotSupported;
    }
    const uint32_t nblk = K >> 8;
    const uint64_t row_bytes = (uint64_t)nblk * Raw<TYPE>::kBlock;
    for (uint32_t c = 0; c < (TYPE == T_Q4_K ? 1u : 8u); ++c) {
        const uint64_t rows = TYPE == T_Q4_K ? M : M > c ? (M - c + 7) / 8 : 0, off = c * row_bytes;
        // a map of no rows is not asked for anything but zeros: that of row 0, out of whose range the boxes then lie
        const cuuint64_t dims[2] = {rows ? (off & 15u) + row_bytes : 16, rows ? rows : 1}, strides[1] = {TYPE == T_Q4_K ? row_bytes : 8 * row_bytes};
        const cuuint32_t box[2] = {R::kRow, TYPE == T_Q4_K ? 128u : 16u};
        if (enc(&maps.w[c], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(A + (rows ? off & ~15ull : 0)), dims, strides, box, ones,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
            CUDA_SUCCESS)
            return cudaErrorNotSupported;
    }
    CutArgs g{D, M, N, nblk, stride_d, cut.tn, 0, 0, cut.parts, cut.cluster, status};
    const uint32_t stage = cut.tn * 256, most = (nblk + cut.parts - 1) / cut.parts, room = kCutSmem - 1024 - kCutBars;
    g.raw_slots = most < 2 ? 1 : 2;
    g.stages = (room - g.raw_slots * R::kSlot) / stage;
    g.stages = g.stages < kCutMaxStages ? g.stages : kCutMaxStages;
    g.stages = g.stages < 2 * most ? g.stages : 2 * most;
    if (TYPE == T_Q4_K && most > 2 && room - g.stages * stage >= 4 * R::kSlot) g.raw_slots = 4;
    if (g.stages < 2) return cudaErrorNotSupported;  // two hold a tile's sums, which take the place of the stages
    auto kern = gemm_cut_kernel<TYPE>;
    static std::atomic<uint64_t> attr_done{0};
    if (cudaError_t e = ensure_dynamic_smem(kern, kCutSmem, attr_done); e != cudaSuccess) return e;
    if (cut.parts > 1)
        if (cudaError_t e = launch_zero(D, M, N, stride_d, s, launches); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cut.parts, (M + kBM - 1) / kBM, (N + cut.tn - 1) / cut.tn);
    cfg.blockDim = dim3(kCutThreads, 1, 1);
    const uint32_t rings = g.stages * stage + g.raw_slots * R::kSlot;
    cfg.dynamicSmemBytes = rings + kCutBars + 1024;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cut.cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, maps, g);
}

// Clusters of 1 to 8 CTAs that the device holds at once.
const int* most_clusters() {
    static std::atomic<int> cache[64][9];
    static thread_local int out[9];
    int dev = 0;
    cudaGetDevice(&dev);
    for (int c = 1; c <= 8; ++c) {
        out[c] = dev < 64 ? cache[dev][c].load(std::memory_order_relaxed) : 0;
        if (out[c]) continue;
        static std::atomic<uint64_t> attr_done{0};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(kCutThreads, 1, 1);
        cfg.dynamicSmemBytes = kCutSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = c;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (ensure_dynamic_smem(gemm_cut_kernel<T_Q4_K>, kCutSmem, attr_done) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&out[c], gemm_cut_kernel<T_Q4_K>, &cfg) != cudaSuccess || out[c] < 1) {
            cudaGetLastError();
            out[c] = -1;  // none
        }
        if (dev < 64) cache[dev][c].store(out[c], std::memory_order_relaxed);
    }
    return out;
}

// Estimates, in us, of this kernel and of the others (gemm_tc.cu, moe_gemm_tc.cu), fitted to 180 shapes of both types with 16 to 11264 tokens
// (here within 10 % rms, 35 % at worst; the others 20 %). Measured, others / this: Q4_K 1024 x 4096, 77 tokens 12.1 / 8.4, 1622 x 1280, 327
// tokens 31.4 / 8.5, 1337 x 2048, 1491 tokens 27.9 / 12.2, 12288 x 4096, 512 tokens 51 / 44 (two rounds of CTAs), Q6_K 783 x 3584, 420
// tokens 36.7 / 13.7, 7398 x 3328, 233 tokens 38.0 / 20.3; the other way Q4_K 2787 x 10496, 196 tokens 19.6 / 26, Q6_K 4096 x 12288,
// 512 tokens 56 / 69, 2048 tokens 145 / 224.
float cut_us(uint32_t type, uint32_t tn, uint32_t most, uint32_t cluster, uint32_t parts, uint32_t rounds) {
    const float one = 3.3f + (float)most * (type == T_Q4_K ? 0.83f : 1.39f) + 0.018f * (float)tn;
    return (float)rounds * one + (parts > 1 ? 2.1f : 0.f) + (cluster > 1 ? 0.9f : 0.f);
}
float others_us(uint32_t type, uint32_t M, uint32_t N, uint32_t K, uint32_t sms, bool vec) {  // vec: D's columns on 16 bytes
    const uint32_t nblk = K >> 8, row_tiles = (M + kBM - 1) / kBM;
    if (N > 256) {  // CTA pairs over 256 rows x 512 tokens
        const uint32_t tiles = (row_tiles + 1) / 2 * ((N + 511) / 512), pairs = sms / 2;
        uint32_t G = tiles * nblk / 4;
        G = G < 1 ? 1 : G > pairs ? pairs : G;
        // whole tiles: 31 shapes within 8 % rms (Q4_K 4096 x 4096, 2048 tokens there 52.5, here 60.7)
        if (tiles <= pairs && tiles * 5 >= pairs * 3) return 16.f + 2.4f * (float)nblk;
        return 28.f + 2.2f * (float)(tiles * nblk) / (float)G;
    }
    if (type == T_Q6_K && (K & 2047u)) return 1e9f;  // one CTA per 128 x 128, by cp.async
    const bool swapped = type == T_Q4_K && N <= 128;  // 256 rows a tile
    const uint32_t tiles = swapped ? (M + 255) / 256 : row_tiles, least = swapped ? 2 : 4;
    uint32_t splits = sms / tiles;
    splits = splits < 1 ? 1 : splits > 8 ? 8 : splits;
    while (splits > 1 && nblk / splits < least) --splits;
    const float blocks = (float)((nblk + splits - 1) / splits), rounds = (float)((tiles * splits + sms - 1) / sms);
    // (single additions: 4075 x 4096, 100 tokens 26 us, 4976 x 5120, 128 tokens with vectors of four 17)
    return swapped ? 7.5f + 2.3f * blocks * rounds + (vec || splits == 1 ? 0.f : 0.12f * (float)N) : N <= 128 ? 6.f + 1.9f * blocks * rounds : 8.f + (type == T_Q4_K ? 1.55f : 1.8f) * blocks * rounds;
}

bool best_cut(uint32_t type, uint32_t M, uint32_t N, uint32_t K, uint32_t sms, bool vec, Cut& best) {
    const uint32_t nblk = K >> 8, row_tiles = (M + kBM - 1) / kBM;
    const int* held = most_clusters();
    // the estimates are some 10 % off either way, between 128 and 256 tokens of Q4_K more (4814 x 5120, 159 tokens: 20.2 us, the other 17.9)
    float least = (type == T_Q4_K && N > 128 && N <= 256 ? 0.8f : 0.9f) * others_us(type, M, N, K, sms, vec);
    bool found = false;
    uint32_t last = 0;
    for (uint32_t nt = (N + kCutMaxTokens - 1) / kCutMaxTokens, tries = 0; nt <= (N + 15) / 16 && tries < 16; ++nt) {
        const uint32_t tn = ((N + nt - 1) / nt + 15u) & ~15u, tiles = row_tiles * ((N + tn - 1) / tn);
        if (tn == last) continue;  // no fewer tokens a tile
        last = tn;
        ++tries;
        for (uint32_t parts = 1; parts <= 16 && parts <= nblk; parts += parts == 1 ? 1 : 2) {
            const uint32_t cluster = parts <= 2 ? 1 : parts / 2;
            if (held[cluster] < 1) continue;
            const uint32_t rounds = (tiles * (parts / cluster) + held[cluster] - 1) / held[cluster], most = (nblk + parts - 1) / parts;
            if (parts > 1 && rounds > 1) break;
            const float us = cut_us(type, tn, most, cluster, parts, rounds);
            if (us < least) {
                least = us;
                best = {tn, parts, cluster};
                found = true;
            }
        }
    }
    return found;
}

}  // namespace

cudaError_t launch_mul_mm_cut(uint32_t type, const uint8_t* A, const void* B, float* D, uint32_t M, uint32_t N, uint32_t K, uint32_t stride_b,
                              uint32_t stride_d, uint32_t* status, cudaStream_t s, uint64_t* launches) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    Cut cut;
    const bool vec = (stride_d & 3u) == 0 && (reinterpret_cast<uintptr_t>(D) & 15u) == 0;
    if (!best_cut(type, M, N, K, (uint32_t)sms, vec, cut)) return cudaErrorNotSupported;
    const cudaError_t e = type == T_Q4_K ? launch_typed<T_Q4_K>(A, B, D, M, N, K, stride_b, stride_d, cut, status, s, launches)
                                         : launch_typed<T_Q6_K>(A, B, D, M, N, K, stride_b, stride_d, cut, status, s, launches);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

}  // namespace zc
