// Streaming decode matvec for Q6_K on the integer tensor cores (dmmv_slice.cuh deals rows to CTAs and K to warps).
//
// Stands in for src/shaders/dmmv_q6k.comp:58-156 (and its use for the down projection and the LM
// head, src/compute/forward.zig:7420, 7714) for the Q6_K layout of src/compute/forward.zig:276-325:
// 210-byte blocks ql[128] qh[64] scales[16] (int8) d (f16), 16-weight sub-blocks.
//
// Arithmetic and operand layout: kquant_dot.cuh. Weights are never rounded; x is rounded to 21 bits.
//
// Blocks are only 2-byte aligned (210 = 13*16 + 2), so a unit is copied as the 16-byte aligned superset of
// each row's block into a 240-byte row slot and read back with 32-bit loads: lane (g = lane/4, t = lane%4)
// reads word t of every 16-byte group of rows g and g+8 (bank = 4 * (15 g mod 8) + t + const: conflict-free),
// one load when the block starts on a word boundary inside its slot, else two and a permutation or a funnel shift.
#include "dmmv_slice.cuh"
#include "kquant_dot.cuh"

namespace zc {

namespace {

constexpr int kRow6 = 240;                  // bytes per row slot: 224-byte superset + pad (15 x 16: odd)
constexpr int kPieces6 = 14;                // 16-byte pieces per row superset
constexpr int kPiecesLane6 = (16 * kPieces6 + 31) / 32;  // 7
constexpr int kZeroBytes6 = 128;

struct Tab6 {
    uint8_t* zeros;  // kZeroBytes6 of zeros (sums of the dead columns 6 and 7)
    uint8_t* x;      // kQ6kTable bytes per super-block
};

// One warp per super-block; lane l handles the 8 consecutive elements 8l .. 8l+7. bpe: blocks of one vector; with more
// than that (MoE down projection) the activation is several vectors, x + s * x_stride, each scaled by the slot's routing
// weight wts[s].
__device__ __forceinline__ void load_x6(X8& r, const float* __restrict__ x, uint32_t blk, uint32_t bpe, uint32_t x_stride,
                                        const uint32_t* __restrict__ wts, int lane) {
    const uint32_t slot = wts ? blk / bpe : 0u, lb = blk - slot * bpe;
    const float* xp = x + (size_t)slot * x_stride + (size_t)lb * 256 + 8 * lane;
    const float w = wts ? __uint_as_float(__ldg(wts + slot)) : 1.f;
    const float4 lo = __ldg(reinterpret_cast<const float4*>(xp)), hi = __ldg(reinterpret_cast<const float4*>(xp) + 1);
    r.lo = make_float4(lo.x * w, lo.y * w, lo.z * w, lo.w * w);
    r.hi = make_float4(hi.x * w, hi.y * w, hi.z * w, hi.w * w);
}

// kAligned: every row starts on a 16-byte boundary (K a multiple of 2048), so all rows of a unit share one offset inside
// their aligned supersets; otherwise each row has its own (rows are 2-byte aligned).
template <bool kAligned>
struct FmtQ6K {
    using Tab = Tab6;
    using X = X8;
    static constexpr uint32_t kSlot = 16 * kRow6;
    static constexpr uint32_t kMost = 16;
    static constexpr uint32_t kCols = 256;
    static constexpr bool kFlowOne = true;
    static constexpr uint32_t kDeepWarps = 12;
    static bool flow_pair(uint32_t K) { return K <= (kAligned ? 8192u : 7424u); }
    static uint32_t flow_tiles(uint32_t K) { return K <= 7424 ? 4 : 9; }
    static uint32_t table_bytes(uint32_t nblk) { return kZeroBytes6 + nblk * kQ6kTable + 128; }
    static __device__ __forceinline__ Tab carve(uint8_t* p, uint32_t) {
        Tab t;
        p += (128u - (smem_u32(p) & 127u)) & 127u;
        t.zeros = p;
        t.x = p + kZeroBytes6;
        return t;
    }
    static __device__ __forceinline__ uint32_t prep_count(const SliceArgs& a) { return a.nblk; }
    template <int kSeg>
    static __device__ __forceinline__ void load_x(X& r, const SliceArgs& a, const NoExtra&, uint32_t blk, int lane) {
        load_x6(r, a.x, blk, a.bpe, a.x_slot_stride, kSeg == 3 ? a.routing + a.nseg : nullptr, lane);
    }
    static __device__ __forceinline__ void clear(const Tab& t, int tid) {
        if (tid < kZeroBytes6 / 16) reinterpret_cast<uint4*>(t.zeros)[tid] = make_uint4(0u, 0u, 0u, 0u);
    }
    static __device__ __forceinline__ void prep(const Tab& t, const X& r, const SliceArgs& a, uint32_t blk, int lane) {
        prep_q6k(t.x, r, a.nblk, blk, lane);
    }

    // piece p = i * 32 + lane of a unit: row p / 14, 16-byte column p % 14 of the row's aligned superset
    struct Copier {
        uint32_t row[kPiecesLane6], col[kPiecesLane6], src[kPiecesLane6];
        __device__ __forceinline__ void init(const SliceArgs& a, int lane) {
#pragma unroll
            for (int i = 0; i < kPiecesLane6; ++i) {
                const uint32_t p = i * 32 + lane;
                row[i] = p / kPieces6;
                col[i] = (p - row[i] * kPieces6) * 16;
                src[i] = row[i] * a.bpe * 210u + col[i];
            }
        }
        __device__ __forceinline__ void copy(const SliceArgs& a, const Unit& u, uint8_t* slot, int) const {
            const uint32_t row_bytes = a.bpe * 210u, d = smem_u32(slot);
            const uint8_t* first = u.mat + (uint64_t)u.row0 * row_bytes + u.lb * 210u;  // the block in the tile's first row
            if constexpr (kAligned) {
                const uint32_t o = (u.lb * 210u) & 15u, room = row_bytes - (u.lb * 210u - o);
                const uint8_t* p = first - o;
                if (u.rows == 16 && room >= kPieces6 * 16u) {  // away from the ends of the matrix and of its rows
#pragma unroll
                    for (int i = 0; i < kPiecesLane6; ++i)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + row[i] * kRow6 + col[i]), "l"(p + src[i])
                                     : "memory");
                    return;
                }
#pragma unroll
                for (int i = 0; i < kPiecesLane6; ++i)
                    if (row[i] < u.rows && col[i] < room)  // rows are 16-byte aligned: a piece never crosses the row end
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + row[i] * kRow6 + col[i]), "l"(p + src[i])
                                     : "memory");
            } else {
                const uint32_t f = (uint32_t)reinterpret_cast<uintptr_t>(first);
                // the pieces of a tile away from the end of the buffer are read whole
                // (A path without the tests for 16 rows inside the buffer was slower: 30000 x 12032 78.5 -> 87 us.)
                const bool inside = first + (uint64_t)u.rows * row_bytes + 240 <= u.end;
#pragma unroll
                for (int i = 0; i < kPiecesLane6; ++i) {
                    const uint32_t o = (f + row[i] * row_bytes) & 15u;
                    if (row[i] < u.rows && col[i] < o + 210u) {  // the piece holds bytes of the block
                        const uint8_t* p = first + src[i] - o;
                        if (inside || p + 16 <= u.end) {
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + row[i] * kRow6 + col[i]), "l"(p)
                                         : "memory");
                        } else {  // the very end of the tensor: copy only the bytes that exist
                            uint8_t* q = slot + row[i] * kRow6 + col[i];
                            for (; p < u.end; ++p) *q++ = __ldg(p);
                        }
                    }
                }
            }
        }
    };

    struct Acc {
        float s[2];
        __device__ __forceinline__ void clear() { s[0] = s[1] = 0.f; }
    };
    struct Lane {
        uint32_t xb, sums, sum_step, xs_s, m0, m1;
        uint32_t g, t;
        float dscale;
        __device__ __forceinline__ void init(const SliceArgs& a, const Tab& s, int lane) {
            g = lane >> 2;
            t = lane & 3;
            const uint32_t x = smem_u32(s.x);
            xb = x + (g < 6 ? g : g - 2) * 64u + t * 16u;  // columns 6 and 7 are dead: m0 = m1 = 0
            m0 = g < 6 && (g & 1) == 0 ? 1u : 0u;
            m1 = g < 6 && (g & 1) ? 1u : 0u;
            sums = g < 6 ? x + a.nblk * 768u + g * 16u + 4u * t : smem_u32(s.zeros);
            sum_step = g < 6 ? 96u : 0u;
            xs_s = x + a.nblk * 864u;
            dscale = __uint_as_float((127u + 14u - 7u * t) << 23);  // digit t carries 2^(14 - 7t)
        }
        __device__ __forceinline__ void dot(const SliceArgs& a, const Unit& u, uint32_t slot, Acc& acc) const {
            uint32_t oA, oB;  // byte offset of the block inside each row's aligned superset
            if constexpr (kAligned) {
                oA = oB = (u.lb * 210u) & 15u;
            } else {
                const uint32_t row_bytes = a.bpe * 210u;
                const uint32_t f = (uint32_t)reinterpret_cast<uintptr_t>(u.mat) + u.row0 * row_bytes + u.lb * 210u;
                oA = (f + g * row_bytes) & 15u;
                oB = (f + (g + 8) * row_bytes) & 15u;
            }
            const uint32_t rA = slot + g * kRow6 + (oA & ~3u), rB = slot + (g + 8) * kRow6 + (oB & ~3u);
            const uint32_t x = xb + u.kb * 768u, sb = sums + u.kb * sum_step;
            const float xs = lds_f1(xs_s + u.kb * 4);
            if constexpr (kAligned) {  // the same for the whole warp
                if (oA & 2u) q6k_block<kHalfWord>(rA, rB, 0u, 0u, x, m0, m1, sb, 4 * t, xs, acc.s);
                else q6k_block<kWord>(rA, rB, 0u, 0u, x, m0, m1, sb, 4 * t, xs, acc.s);
            } else {
                q6k_block<kAnyByte>(rA, rB, (oA & 3u) * 8u, (oB & 3u) * 8u, x, m0, m1, sb, 4 * t, xs, acc.s);
            }
        }
        __device__ __forceinline__ void finish(const Acc& acc, float& v0, float& v1) const {
            v0 = acc.s[0] * dscale;
            v1 = acc.s[1] * dscale;
        }
    };
};

template <int EPI>
cudaError_t launch_plain(const SliceArgs& s, int sm_count, cudaStream_t st) {
    // 210 * K / 256 bytes per row: a multiple of 16 for K % 2048 == 0
    return ((s.K >> 8) % 8u) == 0 ? slice_launch<FmtQ6K<true>, 1, EPI, 0>(s, sm_count, st)
                                  : slice_launch<FmtQ6K<false>, 1, EPI, 0>(s, sm_count, st);
}

}  // namespace

bool q6k_dmmv_eligible(uint32_t type, int mode, const DmmvArgs& a) {
    if (type != T_Q6_K || (a.K & 255u)) return false;
    if (mode != MODE_PLAIN && mode != MODE_SIGMOID_ACC) return false;
    if (!a.status) return false;
    if (reinterpret_cast<uintptr_t>(a.A) & 15u) return false;  // supersets are fetched in 16-byte pieces from the base
    if (((a.K >> 8) % 8u) != 0 && !a.a_end) return false;      // unaligned rows: the end of the buffer must be known
    return a.K <= kFixedPointMaxK && slice_fits<FmtQ6K<true>>(a.K, 1, 1);
}

// MoE down projection + weighted accumulate (y += sum_s w_s W[routing[s]] x_s) through the streaming kernel.
bool q6k_moe_down_acc_eligible(uint32_t type, const DmmvArgs& a) {
    if (type != T_Q6_K || !a.routing || a.n_used == 0 || !a.a_end || !a.status) return false;
    if ((reinterpret_cast<uintptr_t>(a.A) & 15u) || (a.expert_stride & 15u) || (a.K & 255u)) return false;
    if ((a.x_expert_stride & 3u) || (reinterpret_cast<uintptr_t>(a.x) & 15u)) return false;
    if (a.A_sh && ((reinterpret_cast<uintptr_t>(a.A_sh) & 15u) || !a.a_sh_end)) return false;
    if ((uint64_t)a.M * (a.K >> 8) * a.n_used * 210u < kStreamMinBytes) return false;  // small expert sets: latency-bound either way
    return (uint64_t)a.K * a.n_used <= kFixedPointMaxK && slice_fits<FmtQ6K<false>>(a.K, a.n_used, 1);
}

cudaError_t launch_q6k_moe_down_acc(const DmmvArgs& a, cudaStream_t st, uint64_t* launches) {
    SliceArgs s = slice_args(a);
    s.nseg = a.n_used;
    const cudaError_t e = slice_launch<FmtQ6K<false>, 1, EPI_ACC, 3>(s, a.sm_count, st);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

cudaError_t launch_q6k_dmmv(int mode, const DmmvArgs& a, cudaStream_t st, uint64_t* launches) {
    const SliceArgs s = slice_args(a);
    const cudaError_t e = mode == MODE_PLAIN ? launch_plain<EPI_PLAIN>(s, a.sm_count, st) : launch_plain<EPI_SIGMOID_ACC>(s, a.sm_count, st);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

}  // namespace zc
