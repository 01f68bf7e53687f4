// Streaming decode matvec for MXFP4 (17-byte blocks: E8M0 scale + 32 E2M1 nibbles) on the tensor cores
// (dmmv_slice.cuh deals rows to CTAs and K to warps).
//
// Stands in for the reference's dmmv_mxfp4.comp and its MoE forms (src/shaders/dmmv_mxfp4.comp,
// dmmv_mxfp4_moe*.comp) for the block layout of src/compute/forward.zig:431-465.
//
// A byte of a block (two nibbles) becomes two fp16 weights with one conversion instruction, exactly. The activations are
// two fp16 terms per element (scaled by a power of two per 256 elements so that the largest lies in [2^9, 2^10): 22
// significant bits, absolute error 2^-34 of the largest). mma.sync m16n8k16 multiplies 16 rows by them in f32.
// Lane (g, t) owns one block of rows g and g + 8 at a time; its k slots carry that block's elements, and B is
// block-diagonal: column 2 t + p is term p for the k slots of lane t's block and zero elsewhere, so D column 2 t + p is
// that block's dot product with term p alone and lands on the lane that owns the block, which applies its scale.
// A unit is 16 rows x 16 blocks (512 columns); in step q lane t owns block q + 4 t: four blocks are 68 bytes, 17 words, so
// that the 32-bit reads of the four lanes of a row fall on different banks. Rows are only 2-byte aligned (17 K / 32
// bytes): a unit's row segment is fetched as the 16-byte aligned superset and read back with funnel shifts.
// (The E2M1 -> signed byte tables and int8 digits of an earlier form took twice the instructions per weight.)
#include "dmmv_slice.cuh"

namespace zc {

namespace {

constexpr int kUnitBlocks = 16;
constexpr uint32_t kSegBytes = kUnitBlocks * 17;  // 272
constexpr int kRowSlot = 304;                // 288-byte aligned superset + 16: rows 12 banks apart
constexpr int kPiecesRow = 18;
constexpr int kPiecesLane = 16 * kPiecesRow / 32;  // 9
constexpr int kZeroUnits = 64;               // zeros the lanes of dead columns read (one step's table is 512 bytes)

struct TabX {
    uint4* zeros;
    uint4* xf;       // terms of x in B-operand order: ((step * 4 + j) * 2 + term) * 4 + t, step = 4 * unit + q
    float* xs;       // per 256 elements: 2^-f
};

// One warp per 256 elements; lane = b * 4 + j holds, for block b of the chunk, the elements of MMA step j: 4j .. 4j+3 and
// 16 + 4j .. 16 + 4j+3. Elements at or beyond K read as zero. With several slots (MoE down projection) the activation is
// the slots' vectors, x + s * x_stride, each padded to whole units and scaled by the slot's routing weight wts[s], so
// that sum_s w_s W_s x_s becomes one long dot product.
struct XRegsX {
    float4 lo, hi;
};

struct FmtMX {
    using Tab = TabX;
    using X = XRegsX;
    static constexpr uint32_t kSlot = 16 * kRowSlot;
    static constexpr uint32_t kMost = 18;  // what the registers allow: three rows of six warps at K = 2561 to 3072
    static constexpr uint32_t kCols = 512;
    static constexpr bool kFlowOne = false;
    static constexpr uint32_t kDeepWarps = 32;
    static bool flow_pair(uint32_t) { return true; }
    static uint32_t flow_tiles(uint32_t K) { return K <= 2 * kCols ? 0 : 20; }
    static uint32_t table_bytes(uint32_t nblk) { return kZeroUnits * 16 + nblk * (2048 + 8) + 128; }
    static __device__ __forceinline__ Tab carve(uint8_t* p, uint32_t nblk) {
        Tab t;
        p += (128u - (smem_u32(p) & 127u)) & 127u;
        t.zeros = reinterpret_cast<uint4*>(p);
        t.xf = t.zeros + kZeroUnits;
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
    static __device__ __forceinline__ uint32_t pack(float a, float b) {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    static __device__ __forceinline__ uint32_t rest(float a, float b, uint32_t h) {
        const __half2 v = *reinterpret_cast<const __half2*>(&h);
        return pack(a - __low2float(v), b - __high2float(v));
    }
    static __device__ __forceinline__ void clear(const Tab& s, int tid) {
        if (tid < kZeroUnits) s.zeros[tid] = make_uint4(0u, 0u, 0u, 0u);
    }
    static __device__ __forceinline__ void prep(const Tab& s, const X& r, const SliceArgs&, uint32_t chunk, int lane) {
        const uint32_t b = lane >> 2, j = lane & 3;
        float4 lo = r.lo, hi = r.hi;
        float mx = fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(lo.y)), fmaxf(fabsf(lo.z), fabsf(lo.w))),
                         fmaxf(fmaxf(fabsf(hi.x), fabsf(hi.y)), fmaxf(fabsf(hi.z), fabsf(hi.w))));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        uint32_t E = (__float_as_uint(mx) >> 23) & 0xFFu;
        E = E < 32u ? 32u : E;
        const float scale = __uint_as_float((263u - E) << 23);
        lo = make_float4(lo.x * scale, lo.y * scale, lo.z * scale, lo.w * scale);
        hi = make_float4(hi.x * scale, hi.y * scale, hi.z * scale, hi.w * scale);
        // byte k of a block's word j holds elements 4j + k and 16 + 4j + k
        const uint4 h = make_uint4(pack(lo.x, hi.x), pack(lo.y, hi.y), pack(lo.z, hi.z), pack(lo.w, hi.w));
        const uint4 l = make_uint4(rest(lo.x, hi.x, h.x), rest(lo.y, hi.y, h.y), rest(lo.z, hi.z, h.z), rest(lo.w, hi.w, h.w));
        // block b of chunk c is block q + 4 t of unit c / 2
        const uint32_t q = b & 3, t = 2 * (chunk & 1) + (b >> 2), u = (((chunk >> 1) * 4 + q) * 4 + j) * 2;
        s.xf[u * 4 + t] = h;
        s.xf[(u + 1) * 4 + t] = l;
        if (lane == 0) s.xs[chunk] = __uint_as_float((E - 9u) << 23);
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
    static __device__ __forceinline__ uint32_t lds_u32(uint32_t saddr) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
        return v;
    }
    // the four bytes of x (a low and a high nibble each) as pairs of fp16
    static __device__ __forceinline__ void e2m1x8_to_f16(uint32_t x, uint32_t (&o)[4]) {
        asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %4;\n\t"
            "cvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, b;\n\tcvt.rn.f16x2.e2m1x2 %2, c;\n\tcvt.rn.f16x2.e2m1x2 %3, d;\n\t}"
            : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3])
            : "r"(x));
    }
    struct Lane {
        uint32_t xu, xu_step, xs_s, g, t;
        __device__ __forceinline__ void init(const SliceArgs&, const Tab& s, int lane) {
            g = lane >> 2;
            t = lane & 3;
            const bool live = (g >> 1) == t;
            xu = live ? smem_u32(s.xf + (g & 1) * 4 + t) : smem_u32(s.zeros + (g >> 1) + 1);
            xu_step = live ? 512u : 0u;  // 32 entries of 16 bytes per step
            xs_s = smem_u32(s.xs) + 4u * (t >> 1);
        }
        __device__ __forceinline__ void dot(const SliceArgs& a, const Unit& u, uint32_t slot, Acc& acc) const {
            const uint32_t nb = a.K >> 5, row_bytes = nb * 17u;
            const uint32_t f = (uint32_t)reinterpret_cast<uintptr_t>(u.mat) + u.row0 * row_bytes + u.lb * kSegBytes;
            const uint32_t oA = (f + g * row_bytes) & 15u, oB = (f + (g + 8) * row_bytes) & 15u;
            // this lane's blocks q + 4 t of the two rows: all at the same byte position within their words
            const uint32_t pa = slot + g * kRowSlot + oA + 68 * t, pb = slot + (g + 8) * kRowSlot + oB + 68 * t;
            const uint32_t left = nb - u.lb * kUnitBlocks;
            const float xs = lds_f1(xs_s + u.kb * 8);
#pragma unroll 2
            for (uint32_t q = 0; q < 4; ++q) {
                // 17 bytes at byte offset o (0..3) inside five aligned words: the scale is byte o, nibble word i is
                // bytes o + 1 + 4 i .. of them: one funnel shift by 8 (o + 1) bits (a shift of 32 hands back the
                // upper word)
                uint32_t wa[5], wb[5];
                const uint32_t qa = pa + 17 * q, qb = pb + 17 * q;
                const uint32_t sha = (qa & 3u) * 8u + 8u, shb = (qb & 3u) * 8u + 8u;
#pragma unroll
                for (int i = 0; i < 5; ++i) {
                    wa[i] = lds_u32((qa & ~3u) + 4 * i);
                    wb[i] = lds_u32((qb & ~3u) + 4 * i);
                }
                const uint32_t xq = xu + (u.kb * 4 + q) * xu_step;
                float d[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};  // two chains of MMAs
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t ha[4], hb[4];
                    e2m1x8_to_f16(__funnelshift_rc(wa[j], wa[j + 1], sha), ha);
                    e2m1x8_to_f16(__funnelshift_rc(wb[j], wb[j + 1], shb), hb);
                    const uint4 bx = lds_v4(xq + j * 128);
                    mma_f16(d, ha[0], hb[0], ha[1], hb[1], bx.x, bx.y);
                    mma_f16(e, ha[2], hb[2], ha[3], hb[3], bx.z, bx.w);
                }
                if (q + 4 * t < left) {  // blocks past the row end hold stale bytes: their scale must not be used
                    const uint32_t ea = (wa[0] >> (sha - 8u)) & 0xFFu, eb = (wb[0] >> (shb - 8u)) & 0xFFu;
                    acc.s[0] = fmaf(e8m0_to_f32(ea) * xs, (d[0] + e[0]) + (d[1] + e[1]), acc.s[0]);
                    acc.s[1] = fmaf(e8m0_to_f32(eb) * xs, (d[2] + e[2]) + (d[3] + e[3]), acc.s[1]);
                }
            }
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
