// The parts of the K-quant matvecs that their kernels share: x as 21-bit fixed point in three digits, and the exact integer dot
// products of Q4_K and Q6_K blocks with it (src/shaders/dmmv_q6k.comp:58-156; layout: src/compute/forward.zig:276-325).
#pragma once

#include "stream_skel.cuh"

namespace zc {
namespace {

struct X8 {
    float4 lo, hi;
};
__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
__device__ __forceinline__ void put(uint8_t* p, uint32_t v) { *reinterpret_cast<uint32_t*>(p) = v; }
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// Lane l holds elements 8 l .. 8 l + 7 of a block of 256: X = round(x 2^f), |X| <= 2^20, as digits b0 2^14 + b1 2^7 + b2.
struct Digits {
    int X[8];
    uint32_t w[3][2];
    float inv;  // 2^-f
};
__device__ __forceinline__ Digits digits_of(const X8& r) {
    const float v[8] = {r.lo.x, r.lo.y, r.lo.z, r.lo.w, r.hi.x, r.hi.y, r.hi.z, r.hi.w};
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    uint32_t E = (__float_as_uint(mx) >> 23) & 0xFFu;
    E = E < 32u ? 32u : E;
    const float scale = __uint_as_float((273u - E) << 23);
    Digits d;
#pragma unroll
    for (int i = 0; i < 8; ++i) d.X[i] = __float2int_rn(v[i] * scale);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int* X = d.X + 4 * h;
        d.w[0][h] = pack4(X[0] >> 14, X[1] >> 14, X[2] >> 14, X[3] >> 14);
        d.w[1][h] = pack4(X[0] >> 7, X[1] >> 7, X[2] >> 7, X[3] >> 7) & 0x7F7F7F7Fu;
        d.w[2][h] = pack4(X[0], X[1], X[2], X[3]) & 0x7F7F7F7Fu;
    }
    d.inv = __uint_as_float((E - 19u) << 23);
    return d;
}

constexpr uint32_t kQ4kTable = 768 + 32 + 4;  // bytes per block of x
// Block blk of x into a Q4_K table: three digit planes of K bytes, sums per 32 elements, scale per 256.
__device__ __forceinline__ void prep_q4k(uint8_t* tab, const X8& r, uint32_t K, uint32_t blk, int lane) {
    const Digits d = digits_of(r);
#pragma unroll
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(tab + j * K + blk * 256 + 8 * lane) = make_uint2(d.w[j][0], d.w[j][1]);
    int sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) sum += d.X[i];
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
    if ((lane & 3) == 0) put(tab + 3 * K + (blk * 8 + (lane >> 2)) * 4, __float_as_uint((float)sum));
    if (lane == 0) put(tab + 3 * K + (K >> 8) * 32 + blk * 4, __float_as_uint(d.inv));
}

struct Q4kAcc {
    float M[2], m[2];
    __device__ __forceinline__ void clear() { M[0] = M[1] = m[0] = m[1] = 0.f; }
};

// A unit's rows lie 288 bytes apart. 128-bit reads take eight lanes, rows of two lane groups, at a time: rows two apart start
// 64 bytes apart modulo 128, so lane groups 2 i and 2 i + 1 get such rows (the low two bits of the group swapped).
__device__ __forceinline__ uint32_t q4k_row(uint32_t g) { return (g & 4u) | ((g & 1u) << 1) | ((g >> 1) & 1u); }

// One super-block of rows A and B: see the Q4_K streaming matvec for the layout of the operands.
__device__ __forceinline__ void q4k_block(uint32_t rA, uint32_t rB, uint32_t xb, uint32_t sxa, uint32_t xsa, uint32_t t, uint32_t msel, Q4kAcc& acc) {
    constexpr uint32_t kLo = 0x0F0F0F0Fu, kHi = 0xF0F0F0F0u;
    const uint4 hA = lds_v4(rA), hB = lds_v4(rB);
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
        const uint32_t sa = scA[p], sb = scB[p];
        IloA += lo[0] * (int)(sa & 0xFFu) + lo[1] * (int)((sa >> 16) & 0xFFu);
        IhiA += hi[0] * (int)((sa >> 8) & 0xFFu) + hi[1] * (int)(sa >> 24);
        IloB += lo[2] * (int)(sb & 0xFFu) + lo[3] * (int)((sb >> 16) & 0xFFu);
        IhiB += hi[2] * (int)((sb >> 8) & 0xFFu) + hi[3] * (int)(sb >> 24);
    }
    const float PA = (float)(IloA * 16 + IhiA), PB = (float)(IloB * 16 + IhiB);
    const uint32_t mnA = __byte_perm(hA.z & 0x3F3F3F3Fu, ((hA.w >> 4) & 0x0F0F0F0Fu) | ((hA.z >> 2) & 0x30303030u), msel);
    const uint32_t mnB = __byte_perm(hB.z & 0x3F3F3F3Fu, ((hB.w >> 4) & 0x0F0F0F0Fu) | ((hB.z >> 2) & 0x30303030u), msel);
    const float xs = lds_f1(xsa);
    const float2 sxv = lds_f2(sxa);
    const float dA = h2f(hA.x) * xs, dmA = h2f(hA.x >> 16) * xs;
    const float dB = h2f(hB.x) * xs, dmB = h2f(hB.x >> 16) * xs;
    const float mA = (float)(mnA & 0xFFu) * sxv.x + (float)((mnA >> 8) & 0xFFu) * sxv.y;
    const float mB = (float)(mnB & 0xFFu) * sxv.x + (float)((mnB >> 8) & 0xFFu) * sxv.y;
    acc.M[0] = fmaf(dA, PA, acc.M[0]);
    acc.M[1] = fmaf(dB, PB, acc.M[1]);
    acc.m[0] = fmaf(dmA, mA, acc.m[0]);
    acc.m[1] = fmaf(dmB, mB, acc.m[1]);
}

constexpr uint32_t kQ6kTable = 768 + 96 + 4;  // bytes per block of x
// Block blk of nb into a Q6_K table: the digits in the order the lanes read them (768 bytes a block), their sums over the
// sub-blocks in two parts (96), the scales (4). Lane l: half h = l / 16, quarter j = (l / 4) % 4, sub-block half u = (l / 2) % 2, k slots t0, t0 + 1 with t0 = 2 (l % 2)
// kTwice: written to another CTA of the cluster too, whose shared memory is `also` on from this one's.
template <bool kTwice = false>
__device__ __forceinline__ void prep_q6k(uint8_t* tab, const X8& r, uint32_t nb, uint32_t blk, int lane, uint32_t also = 0) {
    const Digits d = digits_of(r);
    const uint32_t h = lane >> 4, j = (lane >> 2) & 3, u = (lane >> 1) & 1, t0 = 2 * (lane & 1);
    uint8_t* const b = tab + blk * 768 + h * 384 + u * 64 + t0 * 16 + j * 4;
    int s[3] = {0, 0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        s[0] += d.X[i] >> 14;
        s[1] += (d.X[i] >> 7) & 0x7F;
        s[2] += d.X[i] & 0x7F;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        put(b + k * 128, d.w[k][0]);
        put(b + k * 128 + 16, d.w[k][1]);
        if constexpr (kTwice) {
            st_cluster(smem_u32(b) + also + k * 128, d.w[k][0]);
            st_cluster(smem_u32(b) + also + k * 128 + 16, d.w[k][1]);
        }
        const int sum = s[k] + __shfl_xor_sync(0xFFFFFFFFu, s[k], 1);  // of sub-block 8 h + 2 j + u: -1024 .. 2032 = 64 hi + lo
        if ((lane & 1) == 0) {
            uint8_t* q = tab + nb * 768 + blk * 96 + k * 32 + 8 * h + 2 * j + u;
            q[0] = (uint8_t)(sum & 63);
            q[16] = (uint8_t)(sum >> 6);
            if constexpr (kTwice) {
                st_cluster_u8(smem_u32(q) + also, sum & 63);
                st_cluster_u8(smem_u32(q) + also + 16, sum >> 6);
            }
        }
    }
    if (lane == 0) {
        put(tab + nb * 864 + blk * 4, __float_as_uint(d.inv));
        if constexpr (kTwice) st_cluster(smem_u32(tab) + also + nb * 864 + blk * 4, __float_as_uint(d.inv));
    }
}

// Where a row's words lie: on word boundaries, in the middle of words (2 bytes past `a`), or anywhere (sh = 8 x the byte past `a`).
// `a` is a multiple of 4.
enum { kWord, kHalfWord, kAnyByte };
template <int kAt>
__device__ __forceinline__ uint32_t lds_word(uint32_t a, uint32_t sh) {
    if constexpr (kAt == kWord) return lds_u32(a);
    else if constexpr (kAt == kHalfWord) return __byte_perm(lds_u32(a), lds_u32(a + 4), 0x5432);
    else return __funnelshift_r(lds_u32(a), lds_u32(a + 4), sh);
}
template <int n>
__device__ __forceinline__ int signed_byte(uint32_t w) {
    int r;  // selector nibble n takes byte n, 8 | n replicates that byte's sign bit
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0u), "n"(n | ((8 | n) << 4) | ((8 | n) << 8) | ((8 | n) << 12)));
    return r;
}
// D(16x8,s32) += A(16x32,s8,row) * B(32x8,s8,col), k 16 .. 31 zero
__device__ __forceinline__ void mma_s8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%6}, {%7,%6}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(0u), "r"(b0));
}
// One Q6_K super-block of rows A and B (kAt, shA, shB: where they start): adds 2^-f d sum_s sc_s P_s, digit t's part of it, to acc.
//   P_s = sum_{i in s} (v_i - 32) X_i = sum_j 2^(14-7j) (D_j,s - 32 SB_j,s),   D_j,s = sum_i v_i b_j,i,   SB_j,s = sum_i b_j,i
// v_i: 6-bit quant 0..63, fed to the tensor core as u8; b_j,i: digits of X (s8). Lane (g = lane / 4, t = lane % 4) reads word t of
// every 16-byte group of its rows: the native A fragment of mma.sync m16n8k32 (bytes 4 t .. and 16 + 4 t .. of 32). An MMA covers
// elements 128 h + 32 j .. of half h, quarter j: sub-blocks 8 h + 2 j (k slots 0..15) and 8 h + 2 j + 1 (16..31). B is
// block-diagonal: column 2 d + u holds digit d in the k slots of sub-block half u and zeros in the other half, so that D column
// 2 d + u is digit d's dot product with sub-block u alone; lane t < 3 has digit t of both sub-blocks for its two rows. x's digits
// come as one word per MMA; m0 and m1 (1 or 0) put it into the register of its half (the other one, and both in the dead columns
// 6 and 7, are zero; by products, as logic operations are what tall matvecs are short of: 65536 x 6144 72.6 us in an earlier form
// with twice the table, 77.2 with masks, 67.5 so). The scales are applied in integers (sums < 2^31), and so is the offset: one
// MMA of the scales with the digits' sums SB, whose two parts of digit t lane t gets. So one conversion and one f32 multiply-add
// per row, digit and block remain. (The offset as start values of the accumulators took 32 moves per block.)
template <int kAt>
__device__ __forceinline__ void q6k_block(uint32_t rA, uint32_t rB, uint32_t shA, uint32_t shB, uint32_t xb, uint32_t m0, uint32_t m1,
                                          uint32_t sums, uint32_t t4, float xs, float (&acc)[2]) {
    constexpr uint32_t kNib = 0x0F0F0F0Fu, kPairs = 0x33333333u;
    int off[4] = {0, 0, 0, 0};
    mma_s8s8(off, lds_word<kAt>(rA + 192 + t4, shA), lds_word<kAt>(rB + 192 + t4, shB), lds_u32(sums));
    int IA = (off[0] + off[1] * 64) * -32, IB = (off[2] + off[3] * 64) * -32;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t vA[4][2], vB[4][2];
        auto six = [&](uint32_t l0, uint32_t l1, uint32_t q, uint32_t (&v)[4][2], int m) {
            const uint32_t e = q & kPairs, o = (q >> 2) & kPairs;  // the top bits of quarters 0 and 2, of 1 and 3
            v[0][m] = (l0 & kNib) | ((e << 4) & ~kNib);
            v[1][m] = (l1 & kNib) | ((o << 4) & ~kNib);
            v[2][m] = ((l0 >> 4) & kNib) | (e & ~kNib);
            v[3][m] = ((l1 >> 4) & kNib) | (o & ~kNib);
        };
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint32_t o = 16 * m + 64 * h, oh = 16 * m + 128 + 32 * h;
            six(lds_word<kAt>(rA + t4 + o, shA), lds_word<kAt>(rA + t4 + o + 32, shA), lds_word<kAt>(rA + t4 + oh, shA), vA, m);
            six(lds_word<kAt>(rB + t4 + o, shB), lds_word<kAt>(rB + t4 + o + 32, shB), lds_word<kAt>(rB + t4 + oh, shB), vB, m);
        }
        const uint32_t sA0 = lds_word<kAt>(rA + 192 + 8 * h, shA), sA1 = lds_word<kAt>(rA + 196 + 8 * h, shA);
        const uint32_t sB0 = lds_word<kAt>(rB + 192 + 8 * h, shB), sB1 = lds_word<kAt>(rB + 196 + 8 * h, shB);
        const uint4 b = lds_v4(xb + 384 * h);
        int c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0}, c2[4] = {0, 0, 0, 0}, c3[4] = {0, 0, 0, 0};
        mma_u8s8(c0, vA[0][0], vB[0][0], vA[0][1], vB[0][1], b.x * m0, b.x * m1);
        mma_u8s8(c1, vA[1][0], vB[1][0], vA[1][1], vB[1][1], b.y * m0, b.y * m1);
        mma_u8s8(c2, vA[2][0], vB[2][0], vA[2][1], vB[2][1], b.z * m0, b.z * m1);
        mma_u8s8(c3, vA[3][0], vB[3][0], vA[3][1], vB[3][1], b.w * m0, b.w * m1);
        IA += c0[0] * signed_byte<0>(sA0) + c0[1] * signed_byte<1>(sA0) + c1[0] * signed_byte<2>(sA0) + c1[1] * signed_byte<3>(sA0) +
              c2[0] * signed_byte<0>(sA1) + c2[1] * signed_byte<1>(sA1) + c3[0] * signed_byte<2>(sA1) + c3[1] * signed_byte<3>(sA1);
        IB += c0[2] * signed_byte<0>(sB0) + c0[3] * signed_byte<1>(sB0) + c1[2] * signed_byte<2>(sB0) + c1[3] * signed_byte<3>(sB0) +
              c2[2] * signed_byte<0>(sB1) + c2[3] * signed_byte<1>(sB1) + c3[2] * signed_byte<2>(sB1) + c3[3] * signed_byte<3>(sB1);
    }
    const uint32_t dA = kAt == kWord ? 0u : kAt == kHalfWord ? 2u : shA >> 3, dB = kAt == kWord ? 0u : kAt == kHalfWord ? 2u : shB >> 3;
    acc[0] = fmaf(h2f(lds_u16(rA + 208 + dA)) * xs, (float)IA, acc[0]);
    acc[1] = fmaf(h2f(lds_u16(rB + 208 + dB)) * xs, (float)IB, acc[1]);
}

}  // namespace
}  // namespace zc
