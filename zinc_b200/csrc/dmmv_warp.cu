// Streaming decode matvec for Q4_K on the integer tensor cores (dmmv_slice.cuh deals rows to CTAs and K to warps).
//
// Stands in for the reference's K-parallel decode shaders and their fused epilogues
// (src/shaders/dmmv_q4k.comp:59-240, dmmv_q4k_wide.comp, dmmv_q4k_fused_gate_up_swiglu.comp:195-218,
// dmmv_q8_0_sigmoid_acc.comp:95-132) for the Q4_K layout of src/compute/forward.zig:370-409.
//
// Arithmetic per super-block of a row, sub-blocks s = 0..7 of 32 weights:
//   y += 2^-f * ( d * sum_s sc_s * P_s  -  dmin * sum_s m_s * SX_s ),   P_s = sum_i q_i * X_i
// X_i = round(x_i * 2^f) is the block of x in 21-bit fixed point (f chosen per 256-element block
// from its largest magnitude), split into three digits X = b0*2^14 + b1*2^7 + b2 that fit int8
// (b0 signed, b1 and b2 in 0..127). The tensor core computes D_j,s = sum_i q_i * b_j,i exactly in s32
// for each digit j; the 6-bit scales are applied in integer arithmetic too (sum_s sc_s * D_j,s < 2^31),
// so one conversion and one f32 multiply-add per row, digit and super-block remain. SX_s = sum_i X_i
// is exact. Weights are never rounded; the only rounding before the f32 scaling is that of x to 21 bits.
//
// Tensor-core mapping (mma.sync m16n8k32, u8 x s8 -> s32): the 16 A rows are 16 weight rows. One 128-bit
// shared-memory read gives lane (g = lane/4, t = lane%4) bytes 16(t%2) .. +15 of the 32-byte qs group
// 2p + t/2 of row g (p = 0, 1), i.e. sixteen low nibbles (sub-block 4p + 2(t/2)) and sixteen high nibbles
// (sub-block 4p + 2(t/2) + 1; kept in place as 16 q, the factor is folded into the scale). An MMA thus
// carries two sub-blocks, k slots of lanes t < 2 one, of lanes t >= 2 the other; B is block-diagonal
// to match: column 2j + u holds digit j of x for the k slots of sub-block half u and zeros elsewhere, so
// D column 2j + u is digit j's dot product with sub-block u alone. Lane t < 3 therefore ends up with
// digit t of both sub-blocks for rows g and g+8 and applies their scales; eight MMAs per 16 x 256 tile.
#include "dmmv_slice.cuh"

namespace zc {

namespace {

constexpr uint32_t kCB = 2;                // super-blocks per unit (one at a time: 10 % more instructions per block)
constexpr int kRowSeg = kCB * 144 + 32;    // 320: rows land 64 B apart mod 128 B -> conflict-free 128-bit reads
constexpr int kZeroBytes = 256;            // zeros: B operand of the lanes whose column is dead for their k slots
constexpr int kFracBits = 20;              // |X| <= 2^20
constexpr int kPieces = kCB * 9;           // 16-byte pieces of a row of a unit
constexpr int kPiecesPerLane = (16 * kPieces + 31) / 32;

struct Tab {
    uint8_t* zeros;  // kZeroBytes of zeros, 128-byte aligned
    uint8_t* dig;    // three digit planes of K bytes each, elements in natural order
    float* sx;       // per 32-element sub-block sum of X
    float* xs;       // per super-block 2^-f
};

// Convert x into int8 digit planes. One warp per super-block; lane l handles the 8 consecutive elements
// 8l .. 8l+7 (a 32-byte coalesced read), so sub-block s is lanes 4s .. 4s+3.
struct XRegs {
    float4 lo, hi;
};
__device__ __forceinline__ void load_x(XRegs& r, const float* __restrict__ x, uint32_t blk, int lane) {
    const float* xp = x + (size_t)blk * 256 + 8 * lane;
    r.lo = __ldg(reinterpret_cast<const float4*>(xp));
    r.hi = __ldg(reinterpret_cast<const float4*>(xp) + 1);
}

// The same eight elements per lane, merged from split-K attention partials (up to four chunks; head_dim a
// multiple of 8, so a lane's elements share a head).
constexpr int kMergeChunks = 4;
__device__ __forceinline__ void load_x_merge(XRegs& r, const MergeArgs& m, uint32_t blk, int lane) {
    const uint32_t k0 = blk * 256 + 8 * lane, head = k0 / m.head_dim, d = k0 - head * m.head_dim;
    float4 pl[kMergeChunks], ph[kMergeChunks];
#pragma unroll
    for (int c = 0; c < kMergeChunks; ++c) {
        if ((uint32_t)c < m.n_chunks) {
            const float4* p = reinterpret_cast<const float4*>(
                m.partial + ((size_t)head * m.n_chunks + c) * m.head_dim + d);
            pl[c] = __ldg(p);
            ph[c] = __ldg(p + 1);
        } else {
            pl[c] = ph[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    float w[kMergeChunks];
    const float inv = attn_merge_weights<kMergeChunks>(
        m.partial + (size_t)m.n_heads * m.n_chunks * m.head_dim + (size_t)head * m.n_chunks * 2, m.sinks,
        m.sink_offset + head, m.n_chunks, w);
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
#pragma unroll
    for (int c = 0; c < kMergeChunks; ++c) {
        lo = make_float4(fmaf(w[c], pl[c].x, lo.x), fmaf(w[c], pl[c].y, lo.y), fmaf(w[c], pl[c].z, lo.z),
                         fmaf(w[c], pl[c].w, lo.w));
        hi = make_float4(fmaf(w[c], ph[c].x, hi.x), fmaf(w[c], ph[c].y, hi.y), fmaf(w[c], ph[c].z, hi.z),
                         fmaf(w[c], ph[c].w, hi.w));
    }
    r.lo = make_float4(lo.x * inv, lo.y * inv, lo.z * inv, lo.w * inv);
    r.hi = make_float4(hi.x * inv, hi.y * inv, hi.z * inv, hi.w * inv);
}

// Four values' low bytes as one word.
__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

__device__ __forceinline__ void prep_x(const Tab& s, const XRegs& r, uint32_t K, uint32_t blk, int lane) {
    const float4 lo = r.lo, hi = r.hi;
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    // |x| < 2^(E-126)  ->  |x * 2^f| < 2^20 with f = 146 - E (E = biased exponent of the block maximum)
    uint32_t E = (__float_as_uint(mx) >> 23) & 0xFFu;
    E = E < 32u ? 32u : E;
    const float scale = __uint_as_float((127u + 126u + kFracBits - E) << 23);
    int X[8];
    int sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        X[i] = __float2int_rn(v[i] * scale);
        sum += X[i];
    }
    uint2 d0, d1, d2;
    d0.x = pack4(X[0] >> 14, X[1] >> 14, X[2] >> 14, X[3] >> 14);
    d0.y = pack4(X[4] >> 14, X[5] >> 14, X[6] >> 14, X[7] >> 14);
    d1.x = pack4(X[0] >> 7, X[1] >> 7, X[2] >> 7, X[3] >> 7) & 0x7F7F7F7Fu;
    d1.y = pack4(X[4] >> 7, X[5] >> 7, X[6] >> 7, X[7] >> 7) & 0x7F7F7F7Fu;
    d2.x = pack4(X[0], X[1], X[2], X[3]) & 0x7F7F7F7Fu;
    d2.y = pack4(X[4], X[5], X[6], X[7]) & 0x7F7F7F7Fu;
    uint8_t* dst = s.dig + (size_t)blk * 256 + 8 * lane;
    *reinterpret_cast<uint2*>(dst) = d0;
    *reinterpret_cast<uint2*>(dst + K) = d1;
    *reinterpret_cast<uint2*>(dst + 2 * (size_t)K) = d2;
    // sub-block sums: four lanes per sub-block
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
    if ((lane & 3) == 0) s.sx[blk * 8 + (lane >> 2)] = (float)sum;
    if (lane == 0) s.xs[blk] = __uint_as_float((E + 1u - kFracBits) << 23);  // 2^-f = 2^(E-146)
}

struct FmtQ4K {
    using Tab = zc::Tab;
    using X = XRegs;
    static constexpr uint32_t kSlot = 16 * kRowSeg;
    static constexpr uint32_t kMost = 16;
    static constexpr uint32_t kCols = kCB * 256;
    static constexpr bool kFlowOne = false;
    static constexpr uint32_t kDeepWarps = 32;
    static bool flow_pair(uint32_t) { return true; }
    static uint32_t flow_tiles(uint32_t K) { return K <= kCols ? 0 : K <= 4096 ? 16 : 6; }
    static uint32_t table_bytes(uint32_t nblk) { return kZeroBytes + nblk * kCB * (768 + 32 + 4) + 128; }
    static __device__ __forceinline__ Tab carve(uint8_t* p, uint32_t nblk) {
        Tab t;
        p += (128u - (smem_u32(p) & 127u)) & 127u;
        t.zeros = p;
        t.dig = p + kZeroBytes;   // K is a multiple of 256: every plane starts 128-byte aligned
        t.sx = reinterpret_cast<float*>(t.dig + (size_t)nblk * kCB * 768);
        t.xs = t.sx + nblk * kCB * 8;
        return t;
    }
    static __device__ __forceinline__ uint32_t prep_count(const SliceArgs& a) { return a.K >> 8; }
    template <int kSeg>
    static __device__ __forceinline__ void load_x(X& r, const SliceArgs& a, const NoExtra&, uint32_t blk, int lane) {
        zc::load_x(r, a.x, blk, lane);
    }
    template <int kSeg>
    static __device__ __forceinline__ void load_x(X& r, const SliceArgs&, const MergeArgs& m, uint32_t blk, int lane) {
        load_x_merge(r, m, blk, lane);
    }
    static __device__ __forceinline__ void clear(const Tab& t, int tid) {
        if (tid < kZeroBytes / 16) reinterpret_cast<uint4*>(t.zeros)[tid] = make_uint4(0u, 0u, 0u, 0u);
    }
    static __device__ __forceinline__ void prep(const Tab& t, const X& r, const SliceArgs& a, uint32_t blk, int lane) {
        prep_x(t, r, a.K, blk, lane);
    }

    // piece p = i * 32 + lane of a unit: row p / 18, 16-byte column p % 18
    struct Copier {
        uint32_t src[kPiecesPerLane], dst[kPiecesPerLane];  // dst: row << 16 | offset in the slot
        __device__ __forceinline__ void init(const SliceArgs& a, int lane) {
#pragma unroll
            for (int i = 0; i < kPiecesPerLane; ++i) {
                const uint32_t p = i * 32 + lane, r = p / kPieces, c = p - r * kPieces;
                src[i] = r * (a.K >> 8) * 144u + c * 16;
                dst[i] = r << 16 | (r * kRowSeg + c * 16);
            }
        }
        __device__ __forceinline__ void copy(const SliceArgs& a, const Unit& u, uint8_t* slot, int) const {
            const uint32_t bpr = a.K >> 8, d = smem_u32(slot);
            const uint8_t* p = u.mat + (uint64_t)u.row0 * (bpr * 144u) + u.lb * (kCB * 144u);
            if (u.rows == 16 && (u.lb + 1) * kCB <= bpr) {
#pragma unroll
                for (int i = 0; i < kPiecesPerLane; ++i)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + (dst[i] & 0xFFFFu)), "l"(p + src[i]) : "memory");
            } else {  // a lower tile, or the last block of an odd number
                const uint32_t bytes = min(kCB, bpr - u.lb * kCB) * 144u;
#pragma unroll
                for (int i = 0; i < kPiecesPerLane; ++i) {
                    const uint32_t r = dst[i] >> 16, off = dst[i] & 0xFFFFu;
                    if (r < u.rows && off - r * kRowSeg < bytes)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + off), "l"(p + src[i]) : "memory");
                }
            }
        }
    };

    // per stream, rows g and g+8: digit t's share of d * sum_s sc_s P_s (to be scaled by 2^(10 - 7t)) and this lane's
    // share of dmin * sum_s m_s SX_s
    struct Acc {
        float M[2], m[2];
        __device__ __forceinline__ void clear() { M[0] = M[1] = m[0] = m[1] = 0.f; }
    };
    struct Lane {
        uint32_t xb_base, xb_step, xs_s, sx_s, msel, g, t;
        float dscale;
        __device__ __forceinline__ void init(const SliceArgs& a, const Tab& s, int lane) {
            g = lane >> 2;
            t = lane & 3;
            // B operand: lane (g, t) feeds column g for its k slots (elements 64(t/2) + 16(t%2) .. +15 of a 128-element
            // pair of qs groups, +32 for the high nibbles). Column g = 2j + u is live for the lanes with t/2 == u and
            // reads digit plane j; the other lanes read zeros, at a bank offset the live lanes of their quarter-warp
            // do not touch (live: 32h + {0..31, 64..95} mod 128 for nibble half h; zeros at 32 + 32h).
            const bool b_live = g < 6 && (g & 1) == (t >> 1);
            xb_base = b_live ? smem_u32(s.dig) + (g >> 1) * a.K + 64u * (t >> 1) + 16u * (t & 1) : smem_u32(s.zeros) + 32u;
            xb_step = b_live ? 256u : 0u;
            xs_s = smem_u32(s.xs);
            sx_s = smem_u32(s.sx) + 8u * t;
            msel = (2u * t) | ((2u * t + 1u) << 4) | 0x7700u;  // bytes 2t, 2t+1 of {mins 0..3, mins 4..7}
            // digit t's sum carries 2^(14 - 7t) and the 1/16 of the in-place high nibbles; lane t = 3 holds zeros
            dscale = __uint_as_float((127u + 10u - 7u * t) << 23);
        }
        __device__ __forceinline__ void dot(const SliceArgs& a, const Unit& u, uint32_t slot, Acc& acc) const {
            constexpr uint32_t kLo = 0x0F0F0F0Fu, kHi = 0xF0F0F0F0u;
#pragma unroll
            for (uint32_t bi = 0; bi < kCB; ++bi) {
                const uint32_t blk = u.kb * kCB + bi;
                if (bi > 0 && blk >= (a.K >> 8)) break;
                const uint32_t rA = slot + bi * 144 + g * kRowSeg, rB = slot + bi * 144 + (g + 8) * kRowSeg;
                const uint4 hA = lds_v4(rA), hB = lds_v4(rB);
                const uint32_t xb = xb_base + blk * xb_step;
                // 6-bit scales of sub-blocks 0..3 and 4..7, one per byte (getScaleMinK4, src/compute/forward.zig:229-238)
                const uint32_t scA[2] = {hA.y & 0x3F3F3F3Fu, (hA.w & 0x0F0F0F0Fu) | ((hA.y >> 2) & 0x30303030u)};
                const uint32_t scB[2] = {hB.y & 0x3F3F3F3Fu, (hB.w & 0x0F0F0F0Fu) | ((hB.y >> 2) & 0x30303030u)};
                int IloA = 0, IhiA = 0, IloB = 0, IhiB = 0;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const uint4 qa = lds_v4(rA + 16 + 64 * p + 16 * t), qb = lds_v4(rB + 16 + 64 * p + 16 * t);
                    const uint4 bl = lds_v4(xb + 128 * p), bh = lds_v4(xb + 128 * p + 32);
                    int lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
                    mma_u8s8(lo, qa.x & kLo, qb.x & kLo, qa.y & kLo, qb.y & kLo, bl.x, bl.y);
                    mma_u8s8(lo, qa.z & kLo, qb.z & kLo, qa.w & kLo, qb.w & kLo, bl.z, bl.w);
                    mma_u8s8(hi, qa.x & kHi, qb.x & kHi, qa.y & kHi, qb.y & kHi, bh.x, bh.y);
                    mma_u8s8(hi, qa.z & kHi, qb.z & kHi, qa.w & kHi, qb.w & kHi, bh.z, bh.w);
                    // D columns 2t, 2t+1 = digit t of sub-blocks 4p (+1 for the high nibbles) and 4p + 2 (+1)
                    const uint32_t sa = scA[p], sb2 = scB[p];
                    IloA += lo[0] * (int)(sa & 0xFFu) + lo[1] * (int)((sa >> 16) & 0xFFu);
                    IhiA += hi[0] * (int)((sa >> 8) & 0xFFu) + hi[1] * (int)(sa >> 24);
                    IloB += lo[2] * (int)(sb2 & 0xFFu) + lo[3] * (int)((sb2 >> 16) & 0xFFu);
                    IhiB += hi[2] * (int)((sb2 >> 8) & 0xFFu) + hi[3] * (int)(sb2 >> 24);
            }
            // the high nibbles were multiplied as 16 q: sum = (16 * lo + hi) / 16, the 1/16 sits in dscale
            const float PA = (float)(IloA * 16 + IhiA), PB = (float)(IloB * 16 + IhiB);
            // mins of sub-blocks 2t, 2t+1
            const uint32_t mnA = __byte_perm(hA.z & 0x3F3F3F3Fu, ((hA.w >> 4) & 0x0F0F0F0Fu) | ((hA.z >> 2) & 0x30303030u), msel);
            const uint32_t mnB = __byte_perm(hB.z & 0x3F3F3F3Fu, ((hB.w >> 4) & 0x0F0F0F0Fu) | ((hB.z >> 2) & 0x30303030u), msel);
            const float xs = lds_f1(xs_s + blk * 4);
            const float2 sxv = lds_f2(sx_s + blk * 32);
            const float dA = h2f(hA.x) * xs, dmA = h2f(hA.x >> 16) * xs;
            const float dB = h2f(hB.x) * xs, dmB = h2f(hB.x >> 16) * xs;
            const float mA = (float)(mnA & 0xFFu) * sxv.x + (float)((mnA >> 8) & 0xFFu) * sxv.y;
            const float mB = (float)(mnB & 0xFFu) * sxv.x + (float)((mnB >> 8) & 0xFFu) * sxv.y;
            acc.M[0] = fmaf(dA, PA, acc.M[0]);
            acc.M[1] = fmaf(dB, PB, acc.M[1]);
            acc.m[0] = fmaf(dmA, mA, acc.m[0]);
            acc.m[1] = fmaf(dmB, mB, acc.m[1]);
            }
        }
        __device__ __forceinline__ void finish(const Acc& acc, float& v0, float& v1) const {
            v0 = fmaf(acc.M[0], dscale, -acc.m[0]);
            v1 = fmaf(acc.M[1], dscale, -acc.m[1]);
        }
    };
};

bool base_ok(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
uint64_t units(uint32_t M, uint32_t K) { return (uint64_t)((M + 15) / 16) * ((K / 256 + kCB - 1) / kCB); }

}  // namespace

bool warp_dmmv_eligible(uint32_t type, int mode, const DmmvArgs& a) {
    if (type != T_Q4_K || (a.K & 255u)) return false;
    if (a.merge.partial && (mode != MODE_PLAIN || a.merge.n_chunks > (uint32_t)kMergeChunks || (a.merge.head_dim & 7u) ||
                            !base_ok(a.merge.partial)))
        return false;
    if (mode != MODE_PLAIN && mode != MODE_GATE_UP_SWIGLU && mode != MODE_SIGMOID_ACC) return false;
    if (!a.status || !base_ok(a.A) || !base_ok(a.A2)) return false;
    const int ns = mode == MODE_GATE_UP_SWIGLU ? 2 : 1;
    return a.K <= kFixedPointMaxK && units(a.M, a.K) * ns >= kFixedPointMinUnits && slice_fits<FmtQ4K>(a.K, 1, ns);
}

cudaError_t launch_warp_dmmv(uint32_t type, int mode, const DmmvArgs& a, cudaStream_t st, uint64_t* launches) {
    (void)type;
    SliceArgs s = slice_args(a);
    cudaError_t e;
    switch (mode) {
        case MODE_PLAIN:
            if (a.merge.partial) {
                uint32_t warps, grid, smem;
                if (!slice_plan<FmtQ4K>(s, 1, 0, a.sm_count, warps, grid, smem)) return cudaErrorInvalidConfiguration;
                static std::atomic<uint64_t> attr_done{0};
                auto kern = dmmv_slice_merge_kernel<FmtQ4K, 16>;
                if ((e = ensure_dynamic_smem(kern, kSliceSmem1, attr_done)) != cudaSuccess) return e;
                e = launch_chained(kern, dim3(grid), dim3(warps * 32), smem, st, s, a.merge);
            } else {
                e = slice_launch<FmtQ4K, 1, EPI_PLAIN, 0>(s, a.sm_count, st);
            }
            break;
        case MODE_GATE_UP_SWIGLU: e = slice_launch<FmtQ4K, 2, EPI_GATE_UP, 0>(s, a.sm_count, st); break;
        case MODE_SIGMOID_ACC: e = slice_launch<FmtQ4K, 1, EPI_SIGMOID_ACC, 0>(s, a.sm_count, st); break;
        default: return cudaErrorInvalidValue;
    }
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

// Grouped launch: n <= 3 Q4_K matrices with the same K and the same x, y_i = W_i x, in one kernel.
bool warp_dmmv_multi_eligible(uint32_t type, uint32_t n, const uint8_t* const* A, const uint32_t* M, uint32_t K,
                              const DmmvArgs& common) {
    if (type != T_Q4_K || n < 2 || n > 3 || (K & 255u) || K > kFixedPointMaxK || !common.status) return false;
    uint64_t u = 0;
    for (uint32_t i = 0; i < n; ++i) {
        if (!base_ok(A[i]) || M[i] == 0) return false;
        u += units(M[i], K);
    }
    return u >= kFixedPointMinUnits && slice_fits<FmtQ4K>(K, 1, 1);
}

cudaError_t launch_warp_dmmv_multi(uint32_t n, const uint8_t* const* A, float* const* y, const uint32_t* M,
                                   const DmmvArgs& common, cudaStream_t st, uint64_t* launches) {
    SliceArgs s = slice_args(common);
    s.nseg = n;
    for (uint32_t i = 0; i < n; ++i) {
        s.segA[i] = A[i];
        s.segY[i] = y[i];
        s.segM[i] = M[i];
    }
    const cudaError_t e = slice_launch<FmtQ4K, 1, EPI_PLAIN, 1>(s, common.sm_count, st);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

// MoE fused gate + up: y_gate[s][M], y_up[s][M] = Wg[routing[s]] x, Wu[routing[s]] x for the n_used slots, x shared.
bool warp_moe_gate_up_eligible(uint32_t type, const DmmvArgs& a) {
    if (type != T_Q4_K || a.x_expert_stride != 0 || !a.routing || !a.A2 || (!a.y2 && !a.act) || !a.status || a.n_used < 1)
        return false;
    if (!base_ok(a.A) || !base_ok(a.A2) || (a.expert_stride & 15u) || !base_ok(a.A_sh) || !base_ok(a.A2_sh) || (a.K & 255u))
        return false;
    return a.K <= kFixedPointMaxK && units(a.M, a.K) * a.n_used * 2 >= kFixedPointMinUnits && slice_fits<FmtQ4K>(a.K, 1, 2);
}

cudaError_t launch_warp_moe_gate_up(const DmmvArgs& a, cudaStream_t st, uint64_t* launches) {
    SliceArgs s = slice_args(a);
    s.nseg = a.n_used;
    const cudaError_t e = slice_launch<FmtQ4K, 2, EPI_PAIR, 2>(s, a.sm_count, st);
    if (e == cudaSuccess && launches) ++*launches;
    return e;
}

}  // namespace zc
