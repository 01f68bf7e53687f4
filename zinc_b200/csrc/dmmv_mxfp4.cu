// Streaming decode matvec for MXFP4 (17-byte blocks: E8M0 scale + 32 E2M1 nibbles) on the tensor cores
// (dmmv_slice.cuh deals rows to CTAs and K to warps).
//
// Stands in for the reference's dmmv_mxfp4.comp and its MoE forms (src/shaders/dmmv_mxfp4.comp,
// dmmv_mxfp4_moe*.comp) for the block layout of src/compute/forward.zig:431-465.
//
// Arithmetic and operand layout: mx_dot.cuh. A unit is 16 rows x 16 blocks (512 columns). Rows are only 2-byte aligned
// (17 K / 32 bytes): a unit's row segment is fetched as the 16-byte aligned superset and read back with funnel shifts.
#include "dmmv_slice.cuh"
#include "mx_dot.cuh"

namespace zc {

namespace {

constexpr int kPiecesRow = 18;
constexpr int kPiecesLane = 16 * kPiecesRow / 32;  // 9
constexpr uint32_t kRowSlot = kMxPitch, kSegBytes = kMxUnitBytes;
constexpr int kUnitBlocks = kMxUnitBlocks;

struct TabX {
    uint4* zeros;
    uint4* xf;
    float* xs;
};

// With several slots (MoE down projection) the activation is the slots' vectors, x + s * x_stride, each padded to whole units and
// scaled by the slot's routing weight wts[s], so that sum_s w_s W_s x_s becomes one long dot product.
struct FmtMX {
    using Tab = TabX;
    using X = MxX;
    static constexpr uint32_t kSlot = 16 * kRowSlot;
    static constexpr uint32_t kMost = 18;  // what the registers allow: three rows of six warps at K = 2561 to 3072
    static constexpr uint32_t kCols = 512;
    static constexpr bool kFlowOne = false;
    static constexpr uint32_t kDeepWarps = 32;
    static bool flow_pair(uint32_t) { return true; }
    static uint32_t flow_tiles(uint32_t K) { return K <= 2 * kCols ? 0 : 20; }
    static uint32_t table_bytes(uint32_t nblk) { return kMxZeros + nblk * kMxTable + 128; }
    static __device__ __forceinline__ Tab carve(uint8_t* p, uint32_t nblk) {
        Tab t;
        p += (128u - (smem_u32(p) & 127u)) & 127u;
        t.zeros = reinterpret_cast<uint4*>(p);
        t.xf = t.zeros + kMxZeros / 16;
        t.xs = reinterpret_cast<float*>(t.xf + (size_t)nblk * 128);
        return t;
    }
    static __device__ __forceinline__ uint32_t prep_count(const SliceArgs& a) { return 2 * a.nblk; }  // chunks of 256 elements
    template <int kSeg>
    static __device__ __forceinline__ void load_x(X& r, const SliceArgs& a, const NoExtra&, uint32_t chunk, int lane) {
        const uint32_t b = lane >> 2, j = lane & 3;
        const uint32_t slot = kSeg == 3 ? chunk / (2 * a.bpe) : 0u, lc = chunk - slot * 2 * a.bpe;
        const uint32_t e0 = lc * 256 + b * 32 + 4 * j;
        r.lo = r.hi = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e0 < a.K) {  // K is a multiple of 32: the whole block or none of it
            const float* xs = a.x + (size_t)slot * a.x_slot_stride + e0;
            const float w = kSeg == 3 ? __uint_as_float(__ldg(a.routing + a.nseg + slot)) : 1.f;
            const float4 lo = __ldg(reinterpret_cast<const float4*>(xs)), hi = __ldg(reinterpret_cast<const float4*>(xs + 16));
            r.lo = make_float4(lo.x * w, lo.y * w, lo.z * w, lo.w * w);
            r.hi = make_float4(hi.x * w, hi.y * w, hi.z * w, hi.w * w);
        }
    }
    static __device__ __forceinline__ void clear(const Tab& s, int tid) {
        if (tid < (int)kMxZeros / 16) s.zeros[tid] = make_uint4(0u, 0u, 0u, 0u);
    }
    static __device__ __forceinline__ void prep(const Tab& s, const X& r, const SliceArgs&, uint32_t chunk, int lane) {
        mx_prep(s.xf, s.xs, r, chunk, lane);
    }

    // piece p = i * 32 + lane of a unit: row p / 18, 16-byte column p % 18 of the row's aligned superset
    struct Copier {
        uint32_t rc[kPiecesLane], src[kPiecesLane];
        __device__ __forceinline__ void init(const SliceArgs& a, int lane) {
            const uint32_t row_bytes = (a.K >> 5) * 17u;
#pragma unroll
            for (int i = 0; i < kPiecesLane; ++i) {
                const uint32_t p = i * 32 + lane, r = p / kPiecesRow, c = p - r * kPiecesRow;
                rc[i] = r | (c << 8) | (((r * row_bytes) & 15u) << 16);
                src[i] = r * row_bytes + c * 16;
            }
        }
        __device__ __forceinline__ void copy(const SliceArgs& a, const Unit& u, uint8_t* slot, int) const {
            const uint32_t nb = a.K >> 5, row_bytes = nb * 17u, d = smem_u32(slot);
            const uint32_t seg = min((uint32_t)kUnitBlocks, nb - u.lb * kUnitBlocks) * 17u;  // bytes of this row segment
            const uint8_t* first = u.mat + (uint64_t)u.row0 * row_bytes + u.lb * kSegBytes;
            const uint32_t tb = (uint32_t)reinterpret_cast<uintptr_t>(first) & 15u;
            const bool inside = first + (uint64_t)u.rows * row_bytes + 304 <= u.end;  // away from the end of the buffer
#pragma unroll
            for (int i = 0; i < kPiecesLane; ++i) {
                const uint32_t r = rc[i] & 0xFFu, c16 = (rc[i] >> 4) & 0xFF0u, o = (tb + (rc[i] >> 16)) & 15u;
                if (r < u.rows && c16 < o + seg) {  // the piece holds bytes of the segment
                    const uint8_t* p = first + src[i] - o;
                    if (inside || p + 16 <= u.end) {
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + r * kRowSlot + c16), "l"(p) : "memory");
                    } else {  // the very end of the tensor: copy only the bytes that exist
                        uint8_t* q = slot + r * kRowSlot + c16;
                        for (; p < u.end; ++p) *q++ = __ldg(p);
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
        MxLane ln;
        __device__ __forceinline__ void init(const SliceArgs&, const Tab& s, int lane) { ln.init(smem_u32(s.xf), smem_u32(s.xs), smem_u32(s.zeros), lane); }
        __device__ __forceinline__ void dot(const SliceArgs& a, const Unit& u, uint32_t slot, Acc& acc) const {
            const uint32_t nb = a.K >> 5, row_bytes = nb * 17u;
            const uint32_t f = (uint32_t)reinterpret_cast<uintptr_t>(u.mat) + u.row0 * row_bytes + u.lb * kSegBytes;
            const uint32_t oA = (f + ln.g * row_bytes) & 15u, oB = (f + (ln.g + 8) * row_bytes) & 15u;
            ln.dot(slot + ln.g * kRowSlot + oA, slot + (ln.g + 8) * kRowSlot + oB, nb - u.lb * kUnitBlocks, u.kb, acc.s);
        }
        __device__ __forceinline__ void finish(const Acc& acc, float& v0, float& v1) const {
            v0 = acc.s[0];
            v1 = acc.s[1];
        }
    };
};

bool common_ok(const DmmvArgs& a) {
    if (!a.status || !a.a_end) return false;
    // rows are fetched as 16-byte-aligned supersets: the buffers themselves must start on that boundary
    if ((reinterpret_cast<uintptr_t>(a.A) & 15u) || (a.A2 && (reinterpret_cast<uintptr_t>(a.A2) & 15u))) return false;
    if ((a.K & 31u) || a.K == 0) return false;
    if ((a.A_sh && ((reinterpret_cast<uintptr_t>(a.A_sh) & 15u) || !a.a_sh_end)) ||
        (a.A2_sh && ((reinterpret_cast<uintptr_t>(a.A2_sh) & 15u) || !a.a2_sh_end)))
        return false;
    return true;
}

}  // namespace

bool mxfp4_dmmv_eligible(uint32_t type, int mode, const DmmvArgs& a) {
    return type == T_MXFP4 && mode == MODE_PLAIN && common_ok(a) && slice_fits<FmtMX>(a.K, 1, 1);
}

bool mxfp4_moe_gate_up_eligible(uint32_t type, const DmmvArgs& a) {
    if (type != T_MXFP4 || a.x_expert_stride != 0 || !a.routing || !a.A2 || (!a.y2 && !a.act) || !a.a2_end || !common_ok(a))
        return false;
    return a.n_used >= 1 && slice_fits<FmtMX>(a.K, 1, 2);
}

bool mxfp4_moe_down_acc_eligible(uint32_t type, const DmmvArgs& a) {
    if (type != T_MXFP4 || !a.routing || a.n_used == 0 || !common_ok(a)) return false;
    if ((a.x_expert_stride & 3u) || (reinterpret_cast<uintptr_t>(a.x) & 15u)) return false;  // float4 loads per slot
    return slice_fits<FmtMX>(a.K, a.n_used, 1);
}

cudaError_t launch_mxfp4_dmmv(const DmmvArgs& a, cudaStream_t st, uint64_t* launches) {
    const cudaError_t e = slice_launch<FmtMX, 1, EPI_PLAIN, 0>(slice_args(a), a.sm_count, st);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

cudaError_t launch_mxfp4_moe_gate_up(const DmmvArgs& a, cudaStream_t st, uint64_t* launches) {
    SliceArgs s = slice_args(a);
    s.nseg = a.n_used;
    const cudaError_t e = slice_launch<FmtMX, 2, EPI_PAIR, 2>(s, a.sm_count, st);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

cudaError_t launch_mxfp4_moe_down_acc(const DmmvArgs& a, cudaStream_t st, uint64_t* launches) {
    SliceArgs s = slice_args(a);
    s.nseg = a.n_used;
    const cudaError_t e = slice_launch<FmtMX, 1, EPI_ACC, 3>(s, a.sm_count, st);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

}  // namespace zc
