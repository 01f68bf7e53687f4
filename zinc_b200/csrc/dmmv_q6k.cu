// Streaming decode matvec for Q6_K on the integer tensor cores (dmmv_slice.cuh deals rows to CTAs and K to warps).
//
// Stands in for src/shaders/dmmv_q6k.comp:58-156 (and its use for the down projection and the LM
// head, src/compute/forward.zig:7420, 7714) for the Q6_K layout of src/compute/forward.zig:276-325:
// 210-byte blocks ql[128] qh[64] scales[16] (int8) d (f16), 16-weight sub-blocks.
//
// Arithmetic per super-block of a row:  y += 2^-f * d * sum_s sc_s * P_s,
//   P_s = sum_{i in s} (v_i - 32) * X_i = sum_j 2^(14-7j) (D_j,s - 32 * SB_j,s),   D_j,s = sum_i v_i * b_j,i
// v_i = 6-bit quant 0..63 fed to the tensor core as u8, X_i = round(x_i * 2^f) the block of x in 21-bit fixed
// point, b_j,i its three digits (s8), SB_j,s = sum_i b_j,i. The MMA accumulators start at -32 * SB_j,s, the
// int8 scales are applied in integer arithmetic (sum_s sc_s * (..) < 2^31), so one conversion and one f32
// multiply-add per row, digit and super-block remain; the only rounding before that is x to 21 bits.
//
// Blocks are only 2-byte aligned (210 = 13*16 + 2), so a unit is copied as the 16-byte aligned superset of
// each row's block into a 240-byte row slot and read back with 32-bit loads: lane (g = lane/4, t = lane%4)
// reads word t of every 16-byte group of rows g and g+8 (bank = 4 * (15 g mod 8) + t + const: conflict-free),
// one load when the block starts on a word boundary inside its slot, two and a funnel shift otherwise.
// That is the native A fragment of mma.sync m16n8k32 (bytes 4t .. 4t+3 and 16 + 4t .. of a 32-byte group):
// an MMA covers the 32 elements 128h + 32j .. of half h, quarter j, i.e. sub-blocks 8h + 2j (k slots 0..15)
// and 8h + 2j + 1 (k slots 16..31). B is block-diagonal to match: column 2d + u holds digit d of x in the k
// slots of sub-block half u and zeros in the other half, so D column 2d + u is digit d's dot product with
// sub-block u alone; lane t < 3 ends up with digit t of both sub-blocks for rows g and g+8.
#include "dmmv_slice.cuh"

namespace zc {

namespace {

constexpr int kRow6 = 240;                  // bytes per row slot: 224-byte superset + pad (15 x 16: odd)
constexpr int kPieces6 = 14;                // 16-byte pieces per row superset
constexpr int kPiecesLane6 = (16 * kPieces6 + 31) / 32;  // 7
constexpr int kZeroBytes6 = 128;
constexpr int kFracBits = 20;
constexpr int kBBytes = 1536;               // B operand table per super-block: [h 2][j pair 2][column 6][t 4][16 bytes]
constexpr int kNsxBytes = 256;              // accumulator start values per super-block: [h 2][digit 4][j 4][u 2] s32

struct Tab6 {
    uint8_t* zeros;  // kZeroBytes6 of zeros (B operand of the dead columns 6 and 7)
    uint8_t* bq;     // per super-block kBBytes: {b0, b1} register pairs in B-operand order
    int* nsx;        // per super-block kNsxBytes / 4: -32 * sum of digit d over sub-block (h, j, u)
    float* xs;       // per super-block 2^-f
};

struct XRegs6 {
    float4 lo, hi;
};
// One warp per super-block; lane l handles the 8 consecutive elements 8l .. 8l+7. bpe: blocks of one vector; with more
// than that (MoE down projection) the activation is several vectors, x + s * x_stride, each scaled by the slot's routing
// weight wts[s].
__device__ __forceinline__ void load_x6(XRegs6& r, const float* __restrict__ x, uint32_t blk, uint32_t bpe, uint32_t x_stride,
                                        const uint32_t* __restrict__ wts, int lane) {
    const uint32_t slot = wts ? blk / bpe : 0u, lb = blk - slot * bpe;
    const float* xp = x + (size_t)slot * x_stride + (size_t)lb * 256 + 8 * lane;
    const float w = wts ? __uint_as_float(__ldg(wts + slot)) : 1.f;
    const float4 lo = __ldg(reinterpret_cast<const float4*>(xp)), hi = __ldg(reinterpret_cast<const float4*>(xp) + 1);
    r.lo = make_float4(lo.x * w, lo.y * w, lo.z * w, lo.w * w);
    r.hi = make_float4(hi.x * w, hi.y * w, hi.z * w, hi.w * w);
}

__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// Lane l's elements 8l .. 8l+7 lie in half h = l/16, quarter j = (l/4)%4, sub-block half u = (l/2)%2, and are
// the k-slot groups t = 2(l%2) and t+1 of that sub-block half.
__device__ __forceinline__ void prep_x6(const Tab6& s, const XRegs6& r, uint32_t blk, int lane) {
    const uint32_t h = lane >> 4, j = (lane >> 2) & 3, u = (lane >> 1) & 1, t0 = 2 * (lane & 1);
    const float4 lo = r.lo, hi = r.hi;
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    float mx = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) mx = fmaxf(mx, fabsf(v[e]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    uint32_t E = (__float_as_uint(mx) >> 23) & 0xFFu;
    E = E < 32u ? 32u : E;
    const float scale = __uint_as_float((127u + 126u + kFracBits - E) << 23);
    int X[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) X[e] = __float2int_rn(v[e] * scale);
    uint32_t dw[3][2];
    int ds[3];
    dw[0][0] = pack4(X[0] >> 14, X[1] >> 14, X[2] >> 14, X[3] >> 14);
    dw[0][1] = pack4(X[4] >> 14, X[5] >> 14, X[6] >> 14, X[7] >> 14);
    dw[1][0] = pack4(X[0] >> 7, X[1] >> 7, X[2] >> 7, X[3] >> 7) & 0x7F7F7F7Fu;
    dw[1][1] = pack4(X[4] >> 7, X[5] >> 7, X[6] >> 7, X[7] >> 7) & 0x7F7F7F7Fu;
    dw[2][0] = pack4(X[0], X[1], X[2], X[3]) & 0x7F7F7F7Fu;
    dw[2][1] = pack4(X[4], X[5], X[6], X[7]) & 0x7F7F7F7Fu;
    ds[0] = ds[1] = ds[2] = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        ds[0] += X[e] >> 14;
        ds[1] += (X[e] >> 7) & 0x7F;
        ds[2] += X[e] & 0x7F;
    }
    uint8_t* bq = s.bq + (size_t)blk * kBBytes + h * 768 + (j >> 1) * 384 + (j & 1) * 8;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        uint8_t* dst = bq + (2 * d + u) * 64 + t0 * 16;
        // {b0, b1}: the digit word sits in the register that feeds the k slots of sub-block half u
        *reinterpret_cast<uint2*>(dst) = u ? make_uint2(0u, dw[d][0]) : make_uint2(dw[d][0], 0u);
        *reinterpret_cast<uint2*>(dst + 16) = u ? make_uint2(0u, dw[d][1]) : make_uint2(dw[d][1], 0u);
        const int sum = ds[d] + __shfl_xor_sync(0xFFFFFFFFu, ds[d], 1);
        if ((lane & 1) == 0) s.nsx[blk * 64 + h * 32 + d * 8 + j * 2 + u] = -32 * sum;
    }
    if ((lane & 1) == 0) s.nsx[blk * 64 + h * 32 + 24 + j * 2 + u] = 0;  // digit 3 does not exist: lane t = 3
    if (lane == 0) s.xs[blk] = __uint_as_float((E + 1u - kFracBits) << 23);
}

__device__ __forceinline__ uint32_t lds_u32s(uint32_t saddr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u16s(uint32_t saddr) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(saddr));
    return v;
}

// The 32-bit word at byte address saddr (2-byte aligned): one load when kFunnel is false (saddr is a multiple
// of 4), else the two words around it and a funnel shift by sh = 8 * (saddr % 4).
template <bool kFunnel>
__device__ __forceinline__ uint32_t lds_word(uint32_t saddr, uint32_t sh) {
    if constexpr (kFunnel) {
        const uint32_t base = saddr & ~3u;
        return __funnelshift_r(lds_u32s(base), lds_u32s(base + 4), sh);
    } else {
        return lds_u32s(saddr);
    }
}

// sign-extended byte n of w
template <int n>
__device__ __forceinline__ int sbyte(uint32_t w) {
    int r;  // prmt: selector nibble n takes byte n, 8 | n replicates that byte's sign bit
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0u), "n"(n | ((8 | n) << 4) | ((8 | n) << 8) | ((8 | n) << 12)));
    return r;
}

// One super-block of rows g (at slot address rA) and g+8 (rB) against the B table at xb / accumulator start
// values at nb; returns sum_s sc_s * (D_t,s - 32 SB_t,s) for digit t = lane % 4 and both rows.
template <bool kFunnel>
__device__ __forceinline__ void block6(uint32_t rA, uint32_t rB, uint32_t shA, uint32_t shB, uint32_t xb, uint32_t xh,
                                       uint32_t nb, int t, int& IA, int& IB) {
    constexpr uint32_t kNib = 0x0F0F0F0Fu, kTop = 0x30303030u;
    IA = IB = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t vA[4][2], vB[4][2];  // [quarter j][sub-block half m]
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint32_t o = 16 * m + 4 * t;
            const uint32_t la0 = lds_word<kFunnel>(rA + 64 * h + o, shA), la1 = lds_word<kFunnel>(rA + 64 * h + 32 + o, shA);
            const uint32_t ha = lds_word<kFunnel>(rA + 128 + 32 * h + o, shA);
            const uint32_t lb0 = lds_word<kFunnel>(rB + 64 * h + o, shB), lb1 = lds_word<kFunnel>(rB + 64 * h + 32 + o, shB);
            const uint32_t hb = lds_word<kFunnel>(rB + 128 + 32 * h + o, shB);
            vA[0][m] = (la0 & kNib) | ((ha << 4) & kTop);
            vA[1][m] = (la1 & kNib) | ((ha << 2) & kTop);
            vA[2][m] = ((la0 >> 4) & kNib) | (ha & kTop);
            vA[3][m] = ((la1 >> 4) & kNib) | ((ha >> 2) & kTop);
            vB[0][m] = (lb0 & kNib) | ((hb << 4) & kTop);
            vB[1][m] = (lb1 & kNib) | ((hb << 2) & kTop);
            vB[2][m] = ((lb0 >> 4) & kNib) | (hb & kTop);
            vB[3][m] = ((lb1 >> 4) & kNib) | ((hb >> 2) & kTop);
        }
        // int8 scales of the half's eight sub-blocks, rows g and g+8
        const uint32_t sA0 = lds_word<kFunnel>(rA + 192 + 8 * h, shA), sA1 = lds_word<kFunnel>(rA + 196 + 8 * h, shA);
        const uint32_t sB0 = lds_word<kFunnel>(rB + 192 + 8 * h, shB), sB1 = lds_word<kFunnel>(rB + 196 + 8 * h, shB);
        // {b0, b1} of quarters 0, 1 / 2, 3 (xh: 0 for the lanes of the dead columns, which read zeros at xb)
        const uint4 b01 = lds_v4(xb + (768 * h & xh)), b23 = lds_v4(xb + ((768 * h + 384) & xh));
        const uint4 n01 = lds_v4(nb + 128 * h), n23 = lds_v4(nb + 128 * h + 16);  // start values: (j, u) pairs
        int c0[4] = {(int)n01.x, (int)n01.y, (int)n01.x, (int)n01.y};
        int c1[4] = {(int)n01.z, (int)n01.w, (int)n01.z, (int)n01.w};
        int c2[4] = {(int)n23.x, (int)n23.y, (int)n23.x, (int)n23.y};
        int c3[4] = {(int)n23.z, (int)n23.w, (int)n23.z, (int)n23.w};
        mma_u8s8(c0, vA[0][0], vB[0][0], vA[0][1], vB[0][1], b01.x, b01.y);
        mma_u8s8(c1, vA[1][0], vB[1][0], vA[1][1], vB[1][1], b01.z, b01.w);
        mma_u8s8(c2, vA[2][0], vB[2][0], vA[2][1], vB[2][1], b23.x, b23.y);
        mma_u8s8(c3, vA[3][0], vB[3][0], vA[3][1], vB[3][1], b23.z, b23.w);
        // D columns 2t, 2t+1 = digit t of sub-blocks 8h + 2j, 8h + 2j + 1: scale bytes 2j, 2j+1 of the half
        IA += c0[0] * sbyte<0>(sA0) + c0[1] * sbyte<1>(sA0) + c1[0] * sbyte<2>(sA0) + c1[1] * sbyte<3>(sA0) +
              c2[0] * sbyte<0>(sA1) + c2[1] * sbyte<1>(sA1) + c3[0] * sbyte<2>(sA1) + c3[1] * sbyte<3>(sA1);
        IB += c0[2] * sbyte<0>(sB0) + c0[3] * sbyte<1>(sB0) + c1[2] * sbyte<2>(sB0) + c1[3] * sbyte<3>(sB0) +
              c2[2] * sbyte<0>(sB1) + c2[3] * sbyte<1>(sB1) + c3[2] * sbyte<2>(sB1) + c3[3] * sbyte<3>(sB1);
    }
}

// kAligned: every row starts on a 16-byte boundary (K a multiple of 2048), so all rows of a unit share one offset inside
// their aligned supersets; otherwise each row has its own (rows are 2-byte aligned).
template <bool kAligned>
struct FmtQ6K {
    using Tab = Tab6;
    using X = XRegs6;
    static constexpr uint32_t kSlot = 16 * kRow6;
    static constexpr uint32_t kMost = 16;
    static constexpr uint32_t kCols = 256;
    static constexpr bool kFlowOne = true;
    static uint32_t flow_tiles(uint32_t) { return 2; }
    static uint32_t table_bytes(uint32_t nblk) { return kZeroBytes6 + nblk * (kBBytes + kNsxBytes + 4) + 128; }
    static __device__ __forceinline__ Tab carve(uint8_t* p, uint32_t nblk) {
        Tab t;
        p += (128u - (smem_u32(p) & 127u)) & 127u;
        t.zeros = p;
        t.bq = p + kZeroBytes6;
        t.nsx = reinterpret_cast<int*>(t.bq + (size_t)nblk * kBBytes);
        t.xs = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(t.nsx) + (size_t)nblk * kNsxBytes);
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
    static __device__ __forceinline__ void prep(const Tab& t, const X& r, const SliceArgs&, uint32_t blk, int lane) {
        prep_x6(t, r, blk, lane);
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
        uint32_t xb_base, xb_step, xh, nsx_s, xs_s;
        int g, t;
        float dscale;
        __device__ __forceinline__ void init(const SliceArgs&, const Tab& s, int lane) {
            g = lane >> 2;
            t = lane & 3;
            // B operand: lane (g, t) feeds column g; columns 6 and 7 are dead (zeros, one address for the quarter-warp)
            const bool b_live = g < 6;
            xb_base = b_live ? smem_u32(s.bq) + (uint32_t)g * 64u + (uint32_t)t * 16u : smem_u32(s.zeros);
            xb_step = b_live ? (uint32_t)kBBytes : 0u;
            xh = b_live ? 0xFFFFFFFFu : 0u;
            nsx_s = smem_u32(s.nsx) + 32u * t;
            xs_s = smem_u32(s.xs);
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
            const uint32_t rA = slot + g * kRow6 + oA, rB = slot + (g + 8) * kRow6 + oB;
            const uint32_t xb = xb_base + u.kb * xb_step, nb = nsx_s + u.kb * (uint32_t)kNsxBytes;
            int IA, IB;
            if (kAligned && (oA & 2u) == 0) block6<false>(rA, rB, 0u, 0u, xb, xh, nb, t, IA, IB);  // the same for the whole warp
            else block6<true>(rA, rB, (oA & 3u) * 8u, (oB & 3u) * 8u, xb, xh, nb, t, IA, IB);
            const float xs = lds_f1(xs_s + u.kb * 4);
            acc.s[0] = fmaf(h2f(lds_u16s(rA + 208)) * xs, (float)IA, acc.s[0]);
            acc.s[1] = fmaf(h2f(lds_u16s(rB + 208)) * xs, (float)IB, acc.s[1]);
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
