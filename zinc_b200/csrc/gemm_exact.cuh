// Prefill GEMM with exact weights and f32 (or bf16) activations on the 5th-generation tensor cores:
// D[n][m] = sum_k W[m][k] * X[n][k], f32 accuracy.
//
// The tensor cores take fp16 operands, so both sides are brought to fp16 without losing f32 accuracy:
//   W  inside a 256-column block a K-quant weight is an integer times the row's d: sc * q (Q4_K 945 at most, Q5_K
//      1953), 2^-10 of it, is exact in fp16 and the f16 block scale d is applied in f32 afterwards. Q6_K (13 bits) is two
//      exact fp16 terms, the second the rounding residue of the first; so is Q8_0 (d * q over the largest d's power of two
//      in the block, 19 bits) for a d of 2^-14 of the largest or more, below that to 2^-25 of the largest weight's power
//      of two. MXFP4 is a power of two times E2M1, one term: exact where the 32-column block's scale is 2^-23 of the largest
//      in the 256 columns or more, below that to 2^-25 of the largest. A row's min term of Q4_K / Q5_K,
//      -dmin * m_s * (sum of x over sub-block s), is 32 more columns of the block: (dmin / d) * m_s in two terms
//      against the sub-block sums of x in two terms.
//   X  a token is scaled by a power of two (its largest element to [2^14, 2^15)) and split into two fp16 terms: 22
//      significant bits down to 2^-17 of the token's largest element, below that an absolute error of 2^-39 of it. bf16
//      activations are one term, exact down to 2^-31 of the largest. (With the largest at 2^4, as it was first, a token with
//      one element 2^16 above the others lost half their bits.)
//      The sub-block sums are scaled by 2^-5 and the min terms too, which with the weights' 2^-10 is the same factor; it
//      leaves dmin / d a range of 2^15 before it no longer fits fp16, and the block's scale goes up by powers of two beyond.
// An infinite activation makes its token's row NaN.
// A run of columns is one accumulation in tensor memory; eight warps of their own then add scale * sum to f32 registers
// ("promote") while further runs fill other accumulators and the producer warps unpack what follows. (With both in the same
// warps a block took the sum of the two: MXFP4 4096 x 4096, 512 tokens 53.2 us, now 43.2, Q6_K 50.1 and 45.6; Q4_K, which has
// little to unpack and long MMAs, 39.8 and 40.0 there, 30.7 and 27.0 at 256 tokens.) The tensor core cuts an accumulator's last bits off at every
// instruction, so the length of a run decides how far the result is from the exact one (relative L2, activations N(0, 1),
// K = 4096):
//   kRuns 1  a block of 256 columns: 1.8e-7 (MXFP4) to 1e-6 (Q8_0 beyond 128 tokens), where one f32 chain per output
//            (gemm_simple_kernel) has 1.1e-6. For zc_mul_mm.
//   kRuns 4  64 columns, their small terms first: 1.2e-7 to 1.8e-7, where f32 sums by lanes (dmmv_kernel) have 1.0e-7 to
//            1.3e-7 and runs of a block 3.6e-7 to 1e-6. For zc_dmmv_batch, in tiles of at most 128 tokens, where a block's
//            four accumulators fit: Q4_K 12288 x 4096, 105 tokens 36.4 us. (Measured while the same warps unpacked and
//            promoted, 37.3 us: runs of a block 36.7; adding a block's four runs before the registers' sum 1.4e-7 and 42 us, with
//            the sum's roundings kept too 1.3e-7 and 49 us: the runs' own roundings are what is left.)
//
// Persistent CTA pairs (cta_group::2, 256 weight rows per pair): tiles of 256 rows x n_tile tokens, their
// (tile, block) units dealt in equal contiguous ranges to the pairs. A tile that is split over two pairs is summed with
// atomic adds into D, which the preparation kernel zeroes; where there are three pairs or more to a tile, the parts go
// through the scratch and are added in their order. Either way the result does not depend on timing.
// Bound: tensor pipe (2 or 3 fp16 products per weight and token) and the shared memory that feeds it from about 160 tokens to
// a tile on (Q4_K, 192 tokens: 3900 cycles a block, of which 34 MMAs take 3264); below that the chain raw block -> unpacked
// stage -> MMA, 2600 to 3000 cycles a block whatever the tokens. Around it: the preparation kernel (4.5 to 8 us), 2 us from
// the launch to the first raw block, 2 to 4 us of epilogue.
#pragma once

#include <atomic>

#include "kernels.h"
#include "tc_common.cuh"

namespace zc {
namespace {

constexpr int kXProdWarp0 = 4, kXPromoters = 8;  // warps: issuer, the two loaders, a spare one; the producers; the promoters
constexpr uint32_t kXBarBytes = 768;
// Blocks whose rows' scales are kept. A producer that passes on block b's has filled block b - 1, so with two stages a set the
// MMAs of block b - 3 are under way, which waited for the promotion of block b - 5: eight (a power of two of more than four).
constexpr uint32_t kXScales = 8;

template <int TYPE>
struct XW;  // kTerms: fp16 terms per weight; kBlock: bytes of 256 columns; kBox: bytes a TMA box (or a fetched row) holds
template <>
struct XW<T_Q4_K> {
    static constexpr int kTerms = 1;
    static constexpr bool kMin = true;
    static constexpr uint32_t kBlock = 144, kTmaRow = 144, kFetchRow = 176;
};
template <>
struct XW<T_Q5_K> {
    static constexpr int kTerms = 1;
    static constexpr bool kMin = true;
    static constexpr uint32_t kBlock = 176, kTmaRow = 176, kFetchRow = 208;
};
template <>
struct XW<T_Q6_K> {
    static constexpr int kTerms = 2;
    static constexpr bool kMin = false;
    static constexpr uint32_t kBlock = 210, kTmaRow = 240, kFetchRow = 240;
};
template <>
struct XW<T_Q8_0> {
    static constexpr int kTerms = 2;
    static constexpr bool kMin = false;
    static constexpr uint32_t kBlock = 272, kTmaRow = 272, kFetchRow = 304;
};
template <>
struct XW<T_MXFP4> {
    static constexpr int kTerms = 1;
    static constexpr bool kMin = false;
    static constexpr uint32_t kBlock = 136, kTmaRow = 176, kFetchRow = 176;
};

// Row strides are odd multiples of 16 bytes, so that 16-byte reads of 8 consecutive rows meet no bank twice.
template <int TYPE, int BN, bool kFetch, int kRuns>
struct XTile {
    static constexpr uint32_t kRow = kFetch ? XW<TYPE>::kFetchRow : XW<TYPE>::kTmaRow;
    // With few tokens a block's MMAs are short and the chain unpack -> MMA -> stage free again would set the pace:
    // every producer set has two stages there (the room the activation slots do not need).
    static constexpr int kABuf = BN == 64 ? 2 : 1;
    static constexpr int kWSlots = 2;
    // Producer warps. The warps that promote get the registers that the others give back (setmaxnreg); tiles beyond 192 tokens
    // need so many there (half a tile's sums) that there is room for eight producers of two sets each, which such a tile's
    // long MMAs leave the time for.
    static constexpr int kProducers = BN <= 192 ? 16 : 8, kSets = 16 / kProducers, kPromWarp0 = kXProdWarp0 + kProducers;
    static constexpr int kThreads = (kPromWarp0 + kXPromoters) * 32;
    static constexpr int kLaunchRegs = BN <= 192 ? 72 : 96, kControlRegs = BN <= 192 ? 72 : 48, kProducerRegs = BN <= 192 ? 48 : 56,
                         kPromoterRegs = BN <= 192 ? 120 : 160;
    static_assert(4 * kControlRegs + kProducers * kProducerRegs + kXPromoters * kPromoterRegs <= kThreads / 32 * kLaunchRegs &&
                      kThreads * kLaunchRegs <= 65536,
                  "what the block was launched with");
    static constexpr uint32_t kWBytes = kBM * kRow;
    // tensor-memory columns of one accumulator, and how many of them there are
    static constexpr int kPStride = BN == 64 || kRuns == 4 ? 128 : 256, kPBufs = kRuns == 4 ? 4 : 2;
    static_assert(kRuns == 1 || BN <= (XW<TYPE>::kTerms == 1 ? 128 : 64), "an accumulator for every run, a stage for every fill of a block");
    static constexpr uint32_t kMinOffset = kABuf * kAStages * kABytes;
    static constexpr uint32_t kMinBytes = kBM * 64;  // 32 columns: 64-byte rows, 64-byte swizzle; two of them
    static constexpr uint32_t kWOffset = kMinOffset + (XW<TYPE>::kMin ? 2 * kMinBytes : 0);
    static constexpr uint32_t kBOffset = kWOffset + ((kWSlots * kWBytes + 1023u) & ~1023u);
    // The rest is a ring of activation slots of 64 columns of a CTA's n_tile / 2 tokens (128 bytes per token and term):
    // as many as fit (small tiles need more of them in flight), at most 16.
    static constexpr uint32_t kSmemBytes = 232448u;
    static constexpr uint32_t kBRoom = (kSmemBytes - 1024u - kXBarBytes - kXScales * kBM * 4u - kBOffset) & ~1023u;
    static_assert(kBRoom >= 2 * BN * 128, "two slots of the widest tile");
    static constexpr uint32_t kScaleOffset = kBOffset + kBRoom, kBarOffset = kScaleOffset + kXScales * kBM * 4u;
};

struct XBars {
    uint64_t full_a[2 * kAStages], empty_a[2 * kAStages];
    uint64_t full_m[2], empty_m[2];
    uint64_t full_w[2], empty_w[2];
    uint64_t full_b[16], empty_b[16];
    uint64_t accum[4], pfree[4];
    uint64_t scales[kXScales];
    uint32_t tmem_base;
    volatile uint32_t failed;
};
static_assert(sizeof(XBars) <= kXBarBytes, "the tiles reserve these bytes for the barrier block");

struct XArgs {
    const uint8_t* A;
    const uint8_t* a_end;     // first byte past the matrix (fetched rows)
    float* D;
    const float* inv_scale;   // [N]: 1 / the token's power of two
    uint32_t M, N, K, nblk;
    uint32_t stride_d;
    uint32_t n_row_pairs, n_tiles, n_tile;  // n_tile tokens per tile (a multiple of 16)
    uint32_t groups;          // > 0: the pairs form groups, each with one pair more than it has tiles
    float* parts;             // null, or [pair][token of the tile][256 rows]: every pair has a part of one tile
    uint32_t terms;           // fp16 terms of an activation: 2 (f32) or 1 (bf16)
    uint32_t* status;
};

// which of `pairs` equal ranges (part_begin) of the units holds unit u
__device__ __forceinline__ uint32_t x_part_of(uint32_t u, uint32_t units, uint32_t pairs) {
    return (uint32_t)(((uint64_t)(u + 1) * pairs - 1) / units);
}

struct XSegment {
    uint32_t tile, b0, b1;
};
__device__ __forceinline__ bool x_next_segment(uint32_t& u, uint32_t u1, uint32_t nblk, XSegment& sg) {
    if (u >= u1) return false;
    sg.tile = u / nblk;
    sg.b0 = u - sg.tile * nblk;
    sg.b1 = min(nblk, sg.b0 + (u1 - u));
    u += sg.b1 - sg.b0;
    return true;
}

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t rotl(uint32_t v, int r) { return __funnelshift_l(v, v, r & 31); }

__device__ __forceinline__ void put_chunk(uint8_t* rowp, int sw, int c, uint4 o) {
    *reinterpret_cast<uint4*>(rowp + ((c ^ sw) << 4)) = o;
}

// 64 columns of Q4_K / Q5_K (w: nibble words, h: the fifth bits' words or unused): chunk i of the stage row holds
// word i's low nibbles (columns 4i + {0, 2, 1, 3}) and high nibbles (32 + 4i + ...): the order a byte mask yields,
// which the activations follow. 1024 + q comes from or-ing q into the fp16 pattern of 1024; one fma leaves s * q.
template <bool kFive>
__device__ __forceinline__ void x_deq_k4(const uint32_t (&w)[8], const uint32_t (&h)[8], int j, float s_lo, float s_hi,
                                         uint8_t* stage, int row) {
    const __half2 lo = __float2half2_rn(s_lo), lo_c = __float2half2_rn(-1024.f * s_lo);
    const __half2 hi = __float2half2_rn(s_hi * 0.0625f), hi_c = __float2half2_rn(-64.f * s_hi);
    uint8_t* rowp = stage + row * 128;
    const int sw = row & 7;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t a = w[i], b = w[i] >> 8;
        uint32_t l0 = (a & 0x000F000Fu) | 0x64006400u, l1 = (b & 0x000F000Fu) | 0x64006400u;
        uint32_t h0 = (a & 0x00F000F0u) | 0x64006400u, h1 = (b & 0x00F000F0u) | 0x64006400u;
        if constexpr (kFive) {  // bit 2j (low) and 2j + 1 (high) of byte 4i + ... of the qh plane
            const uint32_t fl = rotl(h[i], 4 - 2 * j), fh = rotl(h[i], 7 - 2 * j);
            l0 |= fl & 0x00100010u;
            l1 |= (fl >> 8) & 0x00100010u;
            h0 |= fh & 0x01000100u;
            h1 |= rotl(fh, 24) & 0x01000100u;
        }
        uint4 o;
        o.x = h2_bits(__hfma2(bits_h2(l0), lo, lo_c));
        o.y = h2_bits(__hfma2(bits_h2(l1), lo, lo_c));
        o.z = h2_bits(__hfma2(bits_h2(h0), hi, hi_c));
        o.w = h2_bits(__hfma2(bits_h2(h1), hi, hi_c));
        put_chunk(rowp, sw, i, o);
    }
}

// 32 columns as two fp16 terms: chunks 0..3 of the stage row the rounded product v * s, chunks 4..7 its residue.
// q[i]: the pairs (columns 4i + {0, 2}) and (4i + {1, 3}) as fp16 integers; s: scale of columns 4i .. 4i+3.
__device__ __forceinline__ void x_put_two(const uint32_t (&q)[16], const __half2 (&s)[8], uint8_t* stage, int row) {
    uint8_t* rowp = stage + row * 128;
    const int sw = row & 7;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        uint32_t a[4], r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const __half2 v = bits_h2(q[4 * c + e]), sc = s[2 * c + (e >> 1)];
            const __half2 p = __hmul2(v, sc);
            a[e] = h2_bits(p);
            r[e] = h2_bits(__hfma2(v, sc, __hneg2(p)));
        }
        put_chunk(rowp, sw, c, make_uint4(a[0], a[1], a[2], a[3]));
        put_chunk(rowp, sw, c + 4, make_uint4(r[0], r[1], r[2], r[3]));
    }
}

// Columns 32 gg .. of a Q6_K block at p + off (layout: ql[128] qh[64] scales[16] d, element order as dequantRow,
// src/compute/forward.zig:335-383): half n of the block, low or high nibbles of ql, bit pair of qh.
__device__ __forceinline__ void x_deq_q6k(const uint8_t* p, uint32_t off, int gg, uint8_t* stage, int row) {
    const int n = gg >> 2, hi = (gg >> 1) & 1, up = gg & 1;  // columns 128 n + 64 hi + 32 up ..
    uint32_t ql[8], qh[8];
    {
        const uint32_t o = off + 64u * n + 32u * up;
        lds_words<8>(p + (o & ~15u), o & 15u, ql);
    }
    {
        const uint32_t o = off + 128u + 32u * n;
        lds_words<8>(p + (o & ~15u), o & 15u, qh);
    }
    const uint32_t scw = *reinterpret_cast<const unsigned short*>(p + off + 192u + 8u * n + 4u * hi + 2u * up);
    const __half2 k1056 = bits_h2(0x64206420u);  // 1024 + 32
    const __half2 s0 = __float2half2_rn((float)(int)(int8_t)(scw & 0xFFu)), s1 = __float2half2_rn((float)(int)(int8_t)(scw >> 8));
    const int rot = 4 - 4 * hi - 2 * up;
    uint32_t q[16];
    __half2 s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t l = ql[i] >> (4 * hi), t = rotl(qh[i], rot);
        const uint32_t a = (l & 0x000F000Fu) | (t & 0x00300030u) | 0x64006400u;
        const uint32_t b = ((l >> 8) & 0x000F000Fu) | ((t >> 8) & 0x00300030u) | 0x64006400u;
        q[2 * i] = h2_bits(__hsub2(bits_h2(a), k1056));
        q[2 * i + 1] = h2_bits(__hsub2(bits_h2(b), k1056));
        s[i] = i < 4 ? s0 : s1;
    }
    x_put_two(q, s, stage, row);
}

// Columns 32 gg .. of eight Q8_0 blocks: block gg at p + off, dn = its d over the row block's power of two.
__device__ __forceinline__ void x_deq_q8(const uint8_t* p, uint32_t off, float dn, uint8_t* stage, int row) {
    uint32_t w[8];
    lds_words<8>(p + (off & ~15u), off & 15u, w);
    const __half2 k1152 = bits_h2(0x64806480u);  // 1024 + 128
    const __half2 d2 = __float2half2_rn(dn);
    uint32_t q[16];
    __half2 s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t u = w[i] ^ 0x80808080u;
        q[2 * i] = h2_bits(__hsub2(bits_h2((u & 0x00FF00FFu) | 0x64006400u), k1152));
        q[2 * i + 1] = h2_bits(__hsub2(bits_h2(((u >> 8) & 0x00FF00FFu) | 0x64006400u), k1152));
        s[i] = d2;
    }
    x_put_two(q, s, stage, row);
}

// One MXFP4 block (16 nibble bytes in q[4]: low nibbles = columns 0..15, high = 16..31) -> chunks c0 .. c0 + 3: the
// E2M1 bits s|ee|m placed at fp16 bits 15 and 11..9 read as the value times 2^-14; `sc` = 2^14 times the block's
// power of two.
__device__ __forceinline__ void x_deq_mx(const uint32_t (&q)[4], __half2 sc, int c0, uint8_t* stage, int row) {
    uint8_t* rowp = stage + row * 128;
    const int sw = row & 7;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {  // nibble plane e: (byte 0, 2) low, (1, 3) low, (0, 2) high, (1, 3) high
            const uint32_t v = e == 0 ? q[i] : e == 1 ? q[i] >> 8 : e == 2 ? q[i] >> 4 : q[i] >> 12;
            o[e] = h2_bits(__hmul2(bits_h2(((v << 9) & 0x0E000E00u) | ((v << 12) & 0x80008000u)), sc));
        }
        put_chunk(rowp, sw, c0 + i, make_uint4(o[0], o[1], o[2], o[3]));
    }
}

// acc += s * v, two at a time
__device__ __forceinline__ void fma_f32x2(float2& acc, float s, float v0, float v1) {
    asm("{\n\t.reg .b64 a, b, c;\n\t"
        "mov.b64 a, {%2, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "f"(s), "f"(v0), "f"(v1));
}
// Shared-memory matrix descriptor: K-major, 64-byte swizzle, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_64(uint32_t saddr) {
    const uint32_t lo = ((saddr >> 4) & 0x3FFFu) | (1u << 16);
    const uint32_t hi = (512u >> 4) | (1u << 14) | (4u << 29);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float2* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "f"(v[0].x), "f"(v[0].y),
                 "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y)
                 : "memory");
}

template <int TYPE, int BN, bool kFetch, int kRuns>
__global__ void __launch_bounds__(XTile<TYPE, BN, kFetch, kRuns>::kThreads, 1)
gemm_exact_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_m,
                  const __grid_constant__ CUtensorMap tmap_w, const XArgs g) {
    using T = XTile<TYPE, BN, kFetch, kRuns>;
    constexpr int kTerms = XW<TYPE>::kTerms;
    constexpr bool kMin = XW<TYPE>::kMin;
    constexpr uint32_t kBlock = XW<TYPE>::kBlock, kRow = T::kRow;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* smem_b = smem + T::kBOffset;
    uint8_t* smem_w = smem + T::kWOffset;
    XBars* bars = reinterpret_cast<XBars*>(smem + T::kBarOffset);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t nblk = g.nblk;
    const uint32_t U = g.n_tiles * nblk, G = gridDim.x >> 1, slot = blockIdx.x >> 1;
    uint32_t u_begin, u_end;
    if (g.groups) {
        const uint32_t e = x_part_of(slot, G, g.groups), at = (uint32_t)part_begin(e, G, g.groups);
        const uint32_t n = (uint32_t)part_begin(e + 1, G, g.groups) - at, u0 = (at - e) * nblk;  // n pairs share n - 1 tiles
        u_begin = u0 + (uint32_t)part_begin(slot - at, (n - 1) * nblk, n);
        u_end = u0 + (uint32_t)part_begin(slot - at + 1, (n - 1) * nblk, n);
    } else {
        u_begin = (uint32_t)part_begin(slot, U, G);
        u_end = (uint32_t)part_begin(slot + 1, U, G);
    }
    auto tile_m0 = [&](uint32_t tile) { return ((tile % g.n_row_pairs) * 2 + rank) * (uint32_t)kBM; };
    auto tile_n0 = [&](uint32_t tile) { return (tile / g.n_row_pairs) * g.n_tile; };
    const uint32_t b_bytes = g.n_tile * 64 * g.terms;  // an activation slot
    const uint32_t b_slots = min(T::kBRoom / b_bytes, 16u);

    if (tid == 0) {
        for (int s = 0; s < T::kABuf * kAStages; ++s) {
            mbar_init(&bars->full_a[s], 8);  // the four producer warps of the owning set, both CTAs
            mbar_init(&bars->empty_a[s], 1);
        }
        for (uint32_t s = 0; s < b_slots; ++s) {
            mbar_init(&bars->full_b[s], 1);  // the even CTA's loader expects the bytes of both CTAs
            mbar_init(&bars->empty_b[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars->full_w[s], kFetch ? T::kProducers * 32 : 1);
            mbar_init(&bars->empty_w[s], T::kProducers);
            mbar_init(&bars->full_m[s], 2 * T::kProducers);
            mbar_init(&bars->empty_m[s], 1);
        }
        for (int s = 0; s < T::kPBufs; ++s) {
            mbar_init(&bars->accum[s], 1);
            mbar_init(&bars->pfree[s], 2 * kXPromoters);  // of both CTAs
        }
        for (uint32_t s = 0; s < kXScales; ++s) mbar_init(&bars->scales[s], 4);  // the producer warps that have them
        bars->failed = 0;
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                     "r"((uint32_t)(T::kPBufs * T::kPStride))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;

    if constexpr (T::kControlRegs < T::kLaunchRegs) {
        if (warp < kXProdWarp0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(T::kControlRegs));
    }
    if (warp == 0) {
        if (rank == 0) {
            // ---- MMA issuer (even CTA). Two-term activations: up to 128 tokens the terms lie side by side on the MMA's
            // N (half the instructions; an instruction costs the issuer some 70 cycles whatever its N), above that they
            // are two instructions into the same columns. ----
            const bool two = g.terms == 2, merged = kRuns == 1 && two && g.n_tile <= 128;
            const uint32_t n_mma = merged ? 2 * g.n_tile : g.n_tile;
            const uint32_t idesc = (1u << 4) | ((n_mma >> 3) << 17) | ((256u >> 4) << 24);  // fp16 x fp16 -> f32
            const uint32_t lo = two && !merged ? (g.n_tile / 2) * 128 / 16 : 0;  // descriptor step to the low terms
            const uint32_t full_a = smem_u32(bars->full_a), full_b = smem_u32(bars->full_b);
            const uint64_t desc_a = smem_desc(smem_u32(smem)), desc_b = smem_desc(smem_u32(smem_b));
            uint32_t sb = 0, pb = 0;
            bool ok = true;
            const uint32_t total = u_end - u_begin;
            for (uint32_t gb = 0; gb < total && ok; ++gb) {
                if constexpr (kRuns == 1) {
                    const uint32_t d = tmem + (gb & 1) * T::kPStride;
                    uint64_t db = 0;
                    constexpr int kSteps = kTerms == 1 ? 4 : 8;
#pragma unroll
                    for (int st = 0; st < kSteps; ++st) {
                        // fill number f of set st % 4; its stage f % kABuf
                        const uint32_t f = kTerms == 1 ? gb : 2 * gb + (st >> 2);
                        const uint32_t sa = (st & 3) * T::kABuf + f % T::kABuf;
                        const bool open = kTerms == 1 || (st & 1) == 0;  // an activation slot serves two 32-column steps
                        const bool close = kTerms == 1 || (st & 1) == 1;
                        // lane 0 watches the weight stage, lane 1 the activation slot, lane 2 the accumulator
                        uint32_t bar = full_a + sa * 8, par = (f / T::kABuf) & 1;
                        if (open && lane == 1) {
                            bar = full_b + sb * 8;
                            par = pb;
                        }
                        if (st == 0 && lane == 2 && gb >= 2) {
                            bar = smem_u32(&bars->pfree[gb & 1]);
                            par = ((gb >> 1) - 1) & 1;
                        }
                        ok = warp_poll<true>(bar, par, bars, g.status, 181);
                        if (!ok) break;
                        tc_fence_after();
                        if (open) db = desc_b + sb * (b_bytes >> 4);
                        if (elect_one()) {
                            const uint64_t da = desc_a + sa * (kABytes >> 4);
                            if constexpr (kTerms == 1) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    umma_bf16_pair(d, da + 2 * k, db + 2 * k, idesc, (uint32_t)(st | k));
                                    if (lo) umma_bf16_pair(d, da + 2 * k, db + lo + 2 * k, idesc, 1u);
                                }
                            } else {
                                const uint64_t dx = db + 4 * (st & 1);
#pragma unroll
                                for (int k = 0; k < 2; ++k) {
                                    umma_bf16_pair(d, da + 2 * k, dx + 2 * k, idesc, (uint32_t)(st | k));
                                    umma_bf16_pair(d, da + 4 + 2 * k, dx + 2 * k, idesc, 1u);
                                    if (lo) umma_bf16_pair(d, da + 2 * k, dx + lo + 2 * k, idesc, 1u);
                                }
                            }
                            umma_commit_pair(&bars->empty_a[sa]);
                            if (close) umma_commit_pair(&bars->empty_b[sb]);
                            if (!kMin && st == kSteps - 1) umma_commit_pair(&bars->accum[gb & 1]);
                        }
                        if (close && ++sb == b_slots) {
                            sb = 0;
                            pb ^= 1;
                        }
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {  // a run: one stage or two of 32 columns
                        // fill number f of the sets, its stage f % kABuf
                        const uint32_t f = kTerms == 1 ? gb : 2 * gb + (c >> 1);
                        const uint32_t set = kTerms == 1 ? c : 2 * (c & 1);
                        const uint32_t sa = set * T::kABuf + f % T::kABuf, sa2 = sa + (kTerms - 1) * T::kABuf;
                        const uint32_t d = tmem + c * T::kPStride;
                        // lanes 0 and 3 watch the weight stages, lane 1 the activation slot, lane 2 the accumulator
                        uint32_t bar = full_a + (lane == 3 ? sa2 : sa) * 8, par = (f / T::kABuf) & 1;
                        if (lane == 1) {
                            bar = full_b + sb * 8;
                            par = pb;
                        }
                        if (lane == 2 && gb > 0) {
                            bar = smem_u32(&bars->pfree[c]);
                            par = (gb - 1) & 1;
                        }
                        ok = warp_poll<true>(bar, par, bars, g.status, 181);
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {  // small terms first: what they add up to is all that the accumulator rounds them by
                            const uint64_t da = desc_a + sa * (kABytes >> 4), db = desc_b + sb * (b_bytes >> 4);
                            if constexpr (kTerms == 1) {
                                if (lo) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k) umma_bf16_pair(d, da + 2 * k, db + lo + 2 * k, idesc, (uint32_t)k);
                                }
#pragma unroll
                                for (int k = 0; k < 4; ++k) umma_bf16_pair(d, da + 2 * k, db + 2 * k, idesc, lo | (uint32_t)k);
                            } else {
                                const uint64_t da2 = desc_a + sa2 * (kABytes >> 4);
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    umma_bf16_pair(d, (k < 2 ? da : da2) + 4 + 2 * (k & 1), db + 2 * k, idesc, (uint32_t)k);
                                if (lo) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k)
                                        umma_bf16_pair(d, (k < 2 ? da : da2) + 2 * (k & 1), db + lo + 2 * k, idesc, 1u);
                                }
#pragma unroll
                                for (int k = 0; k < 4; ++k) umma_bf16_pair(d, (k < 2 ? da : da2) + 2 * (k & 1), db + 2 * k, idesc, 1u);
                                umma_commit_pair(&bars->empty_a[sa2]);
                            }
                            umma_commit_pair(&bars->empty_a[sa]);
                            umma_commit_pair(&bars->empty_b[sb]);
                            if (!kMin || c < 3) umma_commit_pair(&bars->accum[c]);
                        }
                        if (++sb == b_slots) {
                            sb = 0;
                            pb ^= 1;
                        }
                    }
                }
                if constexpr (kMin) {  // into the last run; merged: these columns hold the sums' terms; the low-term columns see zeros
                    if (!ok) break;
                    ok = warp_poll<true>(lane == 1 ? full_b + sb * 8 : smem_u32(&bars->full_m[gb & 1]), lane == 1 ? pb : (gb >> 1) & 1, bars,
                                   g.status, 184);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t last = kRuns == 4 ? 3 : gb & 1, d = tmem + last * T::kPStride;
                        const uint64_t dm = smem_desc_64(smem_u32(smem + T::kMinOffset + (gb & 1) * T::kMinBytes));
                        const uint64_t ds = desc_b + sb * (b_bytes >> 4);
                        umma_bf16_pair(d, dm, ds, idesc, 1u);
                        umma_bf16_pair(d, dm + 2, ds + 2, idesc, 1u);
                        umma_commit_pair(&bars->empty_m[gb & 1]);
                        umma_commit_pair(&bars->empty_b[sb]);
                        umma_commit_pair(&bars->accum[last]);
                    }
                    if (++sb == b_slots) {
                        sb = 0;
                        pb ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- loader of the activations (each CTA its half of a tile's tokens): lane l serves slot l, so that every free
        // slot is seen in one round of polls ----
        constexpr uint32_t steps = 4u + (kMin ? 1u : 0u);
        const uint32_t half = (g.n_tile / 2) * 128;
        const bool merged = kRuns == 1 && g.terms == 2 && g.n_tile <= 128;
        const uint32_t fills = (u_end - u_begin) * steps;
        const uint32_t full = smem_u32(&bars->full_b[lane & 15]), full_lead = leader_addr(&bars->full_b[lane & 15]);
        const uint32_t empty = smem_u32(&bars->empty_b[lane & 15]);
        uint8_t* dst = smem_b + (lane & 15) * b_bytes;
        uint32_t f = (uint32_t)lane < b_slots ? (uint32_t)lane : fills, par = 1, idle = 0;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        while (__any_sync(0xFFFFFFFFu, f < fills)) {
            const bool go = f < fills && mbar_test_addr(empty, par);
            if (go) {
                const uint32_t blk = f / steps, st = f - blk * steps, u = u_begin + blk, tile = u / nblk, b = u - tile * nblk;
                const int n0 = (int)(tile_n0(tile) + rank * (g.n_tile / 2));
                const bool sums = kMin && st == 4, both = g.terms == 2 && (merged || !sums);
                if (rank == 0)  // the bytes of both CTAs
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(both ? 4 * half : 2 * half) : "memory");
                if (sums) {  // merged: the low-term columns get rows past the sums, zeros
                    tma_load_2d_pair(dst, &tmap_m, (int)(b * 64), n0, full_lead);
                    if (both) tma_load_2d_pair(dst + half, &tmap_m, (int)(b * 64), (int)g.N, full_lead);
                } else {
                    tma_load_2d_pair(dst, &tmap_x, (int)((b * 4 + st) * 64), n0, full_lead);
                    if (both) tma_load_2d_pair(dst + half, &tmap_x, (int)((b * 4 + st) * 64), (int)g.N + n0, full_lead);
                }
                f += b_slots;
                par ^= 1;
            }
            if (__any_sync(0xFFFFFFFFu, go)) {
                idle = 0;
            } else {  // bounded like every other wait
                __nanosleep(40);  // the unpacking warps' stores go through the same pipe as polls (1 %)
                ++idle;
                if ((idle & 255u) == 255u && __any_sync(0xFFFFFFFFu, bars->failed != 0)) break;
                if (idle >= 4u * kWaitLimit) {
                    bars->failed = 1;
                    if (g.status) {
                        g.status[0] = 1;
                        g.status[1] = 185;
                    }
                    break;
                }
            }
        }
    } else if (warp == 2) {
        if (!kFetch && lane == 0) {
            // ---- loader of the raw weight blocks, where rows have a 16-byte pitch. The weights do not depend on the
            // preparation kernel: they arrive and are unpacked while it still runs. ----
            uint32_t u = u_begin, i = 0;
            XSegment ws{0, 0, 0};
            bool ok = true;
            while (ok && x_next_segment(u, u_end, nblk, ws)) {
                const int m0 = (int)tile_m0(ws.tile);
                for (uint32_t b = ws.b0; b < ws.b1; ++b, ++i) {
                    const int sw = i & 1;
                    ok = wait_or_fail(&bars->empty_w[sw], ((i >> 1) & 1) ^ 1, bars, g.status, 191);
                    if (!ok) break;
                    mbar_expect_tx(&bars->full_w[sw], T::kWBytes);
                    // Q8_0 boxes are wider than 256 bytes: their map counts 16-bit elements
                    constexpr int kUnit = TYPE == T_Q8_0 ? 2 : 1;
                    tma_load_2d(smem_w + sw * T::kWBytes, &tmap_w, (int)(((b * kBlock) & ~15u) / kUnit), m0, &bars->full_w[sw]);
                }
            }
        }
    } else if (warp >= kXProdWarp0 && warp < T::kPromWarp0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(T::kProducerRegs));
        // ---- producers: thread = (row, set j0 or the sets j0 and j0 + 2). One-term types: set j holds columns 64 j .. of a block.
        // Two-term types: columns 32 j .. and 128 + 32 j .., one after the other. ----
        constexpr int kSets = T::kSets, kStep = 4 / kSets;
        const int j0 = (warp - kXProdWarp0) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t full_a0 = leader_addr(&bars->full_a[j0 * T::kABuf]);
        const uint32_t full_m = kMin ? leader_addr(&bars->full_m[0]) : 0u;
        float* const scales = reinterpret_cast<float*>(smem + T::kScaleOffset) + row;
        const uint64_t pitch = TYPE == T_Q8_0 || TYPE == T_MXFP4 ? (uint64_t)(g.K >> 5) * (kBlock / 8) : (uint64_t)(g.K >> 8) * kBlock;
        auto row_off = [&](uint32_t tile) {  // rows past M: computed, dropped
            return (uint64_t)min(tile_m0(tile) + (uint32_t)row, g.M - 1) * pitch;
        };
        if constexpr (kMin) {  // columns 24..31 of the min step are zeros
            if (j0 < 2)
                *reinterpret_cast<uint4*>(smem + T::kMinOffset + j0 * T::kMinBytes + row * 64 + ((3 ^ ((row >> 1) & 3)) << 4)) =
                    make_uint4(0, 0, 0, 0);
        }
        // fetched rows: the 16-byte pieces of the aligned supersets of the 128 rows' blocks, dealt to the threads row by
        // row (a warp's copy instruction then meets a handful of cache lines instead of 32)
        uint32_t uf = u_begin, f_b = 0, f_pw = 1;
        int f_sw = 0;
        XSegment f_seg{0, 0, 0};
        bool f_live = false;
        uint32_t f_m0 = 0;
        uint64_t c_off = 0;
        auto fetch = [&]() -> bool {
            if (!f_live) return true;
            if (!poll_or_fail(&bars->empty_w[f_sw], f_pw, bars, g.status, 186)) return false;
            uint8_t* dst = smem_w + f_sw * T::kWBytes;
            constexpr int kPieces = (kBlock + 15 + 15) / 16, kFetchers = T::kProducers * 32;
            static_assert(!kFetch || kPieces * 16 <= (int)kRow, "a fetched row fits its slot");
            const uint32_t pi = (uint32_t)tid - kXProdWarp0 * 32;
#pragma unroll
            for (int i = 0; i < (kBM * kPieces + kFetchers - 1) / kFetchers; ++i) {
                const uint32_t idx = pi + (uint32_t)kFetchers * i, r = idx / kPieces, piece = idx - r * kPieces;
                if ((kBM * kPieces) % kFetchers == 0 || r < (uint32_t)kBM) {
                    const uint64_t o = (uint64_t)min(f_m0 + r, g.M - 1) * pitch + (uint64_t)f_b * kBlock;
                    const uint8_t* sp = g.A + (o & ~(uint64_t)15) + piece * 16;
                    const uint32_t n = sp + 16 <= g.a_end ? 16u : (sp < g.a_end ? (uint32_t)(g.a_end - sp) : 0u);
                    cp_async16_zfill(dst + r * kRow + piece * 16, n ? sp : g.A, n);
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bars->full_w[f_sw])) : "memory");
            f_sw ^= 1;
            if (f_sw == 0) f_pw ^= 1;
            if (++f_b == f_seg.b1) {
                f_live = x_next_segment(uf, u_end, nblk, f_seg);
                f_b = f_seg.b0;
                if (f_live) f_m0 = tile_m0(f_seg.tile);
            }
            return true;
        };
        bool ok = true;
        if constexpr (kFetch) {
            f_live = x_next_segment(uf, u_end, nblk, f_seg);
            f_b = f_seg.b0;
            if (f_live) f_m0 = tile_m0(f_seg.tile);
            ok = fetch();
        }
        uint32_t u = u_begin, b = 0;
        XSegment sg{0, 0, 0};
        const uint32_t total = u_end - u_begin;
        // the scale of the row's block, for the warps that promote
        auto pass_on = [&](uint32_t gb, float sc) {
            if (j0 == 0) {
                scales[(gb & (kXScales - 1)) * kBM] = sc;
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->scales[gb & (kXScales - 1)]);
            }
        };
        for (uint32_t gb = 0; gb < total && ok; ++gb, ++b) {
            if (gb == 0 || b == sg.b1) {
                x_next_segment(u, u_end, nblk, sg);
                b = sg.b0;
                if constexpr (kFetch) c_off = row_off(sg.tile);
            }
            const int sw = gb & 1;
            if (!poll_or_fail(&bars->full_w[sw], (gb >> 1) & 1, bars, g.status, 187)) break;
            if constexpr (kFetch) {
                if (!fetch()) break;  // the next block, into the slot the previous one left
            }
            const uint8_t* wp = smem_w + sw * T::kWBytes + row * kRow;
            const uint32_t off = kFetch ? (uint32_t)((c_off + (uint64_t)b * kBlock) & 15u) : (b * kBlock) & 15u;
            // one-term types: fill number gb of a set, two-term types: 2 gb and 2 gb + 1
            const int ab = T::kABuf == 1 ? 0 : (int)(gb & 1);
            const uint32_t pa = ((gb / T::kABuf) & 1) ^ 1;
            float s_cur;
            if constexpr (kMin) {  // Q4_K / Q5_K rows and blocks are multiples of 16 bytes: off = 0
                const uint4 hd = *reinterpret_cast<const uint4*>(wp);
                uint4 c[2 * kSets];
                uint32_t read = hd.x;
#pragma unroll
                for (int e = 0; e < kSets; ++e) {
                    c[2 * e] = *reinterpret_cast<const uint4*>(wp + kBlock - 128 + (j0 + kStep * e) * 32);
                    c[2 * e + 1] = *reinterpret_cast<const uint4*>(wp + kBlock - 112 + (j0 + kStep * e) * 32);
                    read ^= c[2 * e].x ^ c[2 * e + 1].x;
                }
                uint4 h0 = c[0], h1 = c[1];
                if constexpr (TYPE == T_Q5_K) {
                    h0 = *reinterpret_cast<const uint4*>(wp + 16);
                    h1 = *reinterpret_cast<const uint4*>(wp + 32);
                }
                release_after(read ^ h0.y ^ h1.y, &bars->empty_w[sw], lane);
                const __half2 dd = *reinterpret_cast<const __half2*>(&hd.x);
                const float d = __low2float(dd), dmin = __high2float(dd);
                // The block's scale is d; where dmin is more than 2^15 of it (and there are mins at all), d times the
                // power of two that brings the ratio to [2^14, 2^15): the q terms go down by as much, exactly as far
                // as fp16 reaches (a ratio of 2^25) and beyond that to 2^-29 of a min term.
                float ratio = 0.f, q_scale = 1.f / 1024.f;
                bool mins = true;
                s_cur = d;
                if (fabsf(dmin) > 32768.f * fabsf(d)) {
                    mins = (hd.z | (hd.w & 0xF0F0F0F0u)) != 0u;
                    if (mins && d == 0.f) {
                        s_cur = dmin * (1.f / 32768.f);
                        q_scale = 0.f;
                    } else if (mins) {
                        const uint32_t e = __float_as_uint(__fdividef(fabsf(dmin), fabsf(d))) >> 23;
                        s_cur = d * __uint_as_float((e - 14u) << 23);
                        q_scale = __uint_as_float((258u - e) << 23);
                    }
                }
                if (mins && s_cur != 0.f) {  // dmin / s_cur: an approximate reciprocal and a Newton step
                    const float r = __fdividef(1.f, s_cur);
                    ratio = dmin * fmaf(fmaf(-s_cur, r, 1.f), r, r);
                }
                ratio *= -1.f / 32.f;
                pass_on(gb, s_cur);
                uint32_t vh[kSets], vl[kSets];
#pragma unroll
                for (int e = 0; e < kSets; ++e) {
                    const int j = j0 + kStep * e;
                    // the 6-bit scales and mins of sub-blocks 2j and 2j + 1 (getScaleMinK4, src/compute/forward.zig:229-238),
                    // four at a time as bytes
                    uint32_t scw, mnw;
                    if (j < 2) {
                        scw = hd.y & 0x3F3F3F3Fu;
                        mnw = hd.z & 0x3F3F3F3Fu;
                    } else {
                        scw = (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u);
                        mnw = ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u);
                    }
                    scw >>= 16 * (j & 1);
                    mnw >>= 16 * (j & 1);
                    const uint32_t s0 = scw & 0xFFu, s1 = (scw >> 8) & 0xFFu, mn0 = mnw & 0xFFu, mn1 = (mnw >> 8) & 0xFFu;
                    const uint32_t w[8] = {c[2 * e].x, c[2 * e].y, c[2 * e].z, c[2 * e].w, c[2 * e + 1].x, c[2 * e + 1].y, c[2 * e + 1].z, c[2 * e + 1].w};
                    const uint32_t hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                    if (!poll_or_fail(&bars->empty_a[j0 * T::kABuf + kStep * e * T::kABuf + ab], pa, bars, g.status, 188)) { ok = false; break; }
                    x_deq_k4<TYPE == T_Q5_K>(w, hw, j, q_scale * (float)s0, q_scale * (float)s1, smem + (j0 * T::kABuf + kStep * e * T::kABuf + ab) * kABytes, row);
                    const float v0 = ratio * (float)mn0, v1 = ratio * (float)mn1;
                    const __half2 hi = __floats2half2_rn(v0, v1);
                    vh[e] = h2_bits(hi);
                    vl[e] = h2_bits(__floats2half2_rn(v0 - __low2float(hi), v1 - __high2float(hi)));
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(full_a0 + (kStep * e * T::kABuf + ab) * 8);
                }
                if (!ok) break;
                if (!poll_or_fail(&bars->empty_m[gb & 1], ((gb >> 1) & 1) ^ 1, bars, g.status, 189)) break;
                // chunks 0, 1, 2: high, low, high terms
                uint8_t* mp = smem + T::kMinOffset + (gb & 1) * T::kMinBytes + row * 64 + 4 * j0;
                const int x = (row >> 1) & 3;
#pragma unroll
                for (int e = 0; e < kSets; ++e) {
                    *reinterpret_cast<uint32_t*>(mp + 8 * e + ((0 ^ x) << 4)) = vh[e];
                    *reinterpret_cast<uint32_t*>(mp + 8 * e + ((1 ^ x) << 4)) = vl[e];
                    *reinterpret_cast<uint32_t*>(mp + 8 * e + ((2 ^ x) << 4)) = vh[e];
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(full_m + (gb & 1) * 8);
            } else if constexpr (TYPE == T_MXFP4) {
                uint32_t emax = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (8 * b + i < (g.K >> 5)) emax = max(emax, (uint32_t)wp[off + 17 * i]);
                s_cur = e8m0_to_f32(emax);
                pass_on(gb, s_cur);
                uint32_t q[2 * kSets][4], read = emax;  // every word read: nibbles, the block's scales, these sets' own
                __half2 sc[2 * kSets];
#pragma unroll
                for (int i = 0; i < 2 * kSets; ++i) {
                    const int blk = 2 * (j0 + kStep * (i >> 1)) + (i & 1);
                    const uint32_t o = off + 17u * blk, e = wp[o];
                    const int diff = (int)emax - (int)e;
                    lds_words<4>(wp + ((o + 1) & ~15u), (o + 1) & 15u, q[i]);
                    read ^= e ^ q[i][0] ^ q[i][3];
                    const bool live = 8 * b + blk < (g.K >> 5);
                    sc[i] = __float2half2_rn(live && diff < 60 ? __uint_as_float((uint32_t)(127 + 14 - diff) << 23) : 0.f);
                    if (!live) q[i][0] = q[i][1] = q[i][2] = q[i][3] = 0u;
                }
                release_after(read, &bars->empty_w[sw], lane);
#pragma unroll
                for (int e = 0; e < kSets; ++e) {
                    uint8_t* stage = smem + (j0 * T::kABuf + kStep * e * T::kABuf + ab) * kABytes;
                    if (!poll_or_fail(&bars->empty_a[j0 * T::kABuf + kStep * e * T::kABuf + ab], pa, bars, g.status, 188)) { ok = false; break; }
                    x_deq_mx(q[2 * e], sc[2 * e], 0, stage, row);
                    x_deq_mx(q[2 * e + 1], sc[2 * e + 1], 4, stage, row);
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(full_a0 + (kStep * e * T::kABuf + ab) * 8);
                }
            } else {
                float up = 1.f;  // Q8_0: 1 / s_cur, a power of two
                if constexpr (TYPE == T_Q8_0) {
                    uint32_t top = 0;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (8 * b + i < (g.K >> 5)) top = max(top, (uint32_t)*reinterpret_cast<const unsigned short*>(wp + off + 34 * i) & 0x7FFFu);
                    const uint32_t e = __float_as_uint(h2f(top)) >> 23;  // f32 exponent of the largest |d|
                    s_cur = __uint_as_float(e << 23);
                    up = e ? __uint_as_float((254u - e) << 23) : 0.f;
                } else {
                    s_cur = h2f(*reinterpret_cast<const unsigned short*>(wp + off + 208));
                }
                pass_on(gb, s_cur);
#pragma unroll
                for (int f = 0; f < 2 * kSets; ++f) {  // in the order in which the issuer takes them: the second halves last
                    const int hf = f / kSets, st = kStep * (f % kSets), gg = j0 + st + 4 * hf;
                    // two stages: fill hf goes to stage hf, once a block
                    const int ab2 = T::kABuf == 1 ? 0 : hf;
                    uint8_t* stage2 = smem + (j0 * T::kABuf + st * T::kABuf + ab2) * kABytes;
                    const uint32_t pa2 = T::kABuf == 1 ? (uint32_t)hf ^ 1u : (gb & 1) ^ 1u;
                    if (!poll_or_fail(&bars->empty_a[j0 * T::kABuf + st * T::kABuf + ab2], pa2, bars, g.status, 188)) { ok = false; break; }
                    if constexpr (TYPE == T_Q6_K) {
                        x_deq_q6k(wp, off, gg, stage2, row);
                    } else if (8 * b + gg < (g.K >> 5)) {
                        const uint32_t o = off + 34u * gg;
                        x_deq_q8(wp, o + 2, h2f(*reinterpret_cast<const unsigned short*>(wp + o)) * up, stage2, row);
                    } else {  // past K
#pragma unroll
                        for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(stage2 + row * 128 + c * 16) = make_uint4(0, 0, 0, 0);
                    }
                    // the weights and their scales are in the stores above; the block's scale is in nothing yet
                    if (f == 2 * kSets - 1) release_after(__float_as_uint(s_cur), &bars->empty_w[sw], lane);
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(full_a0 + (st * T::kABuf + ab2) * 8);
                }
                if (!ok) break;
            }
        }
    } else if (warp >= T::kPromWarp0) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(T::kPromoterRegs));
        // ---- promoters: thread = (row, half of the tile's tokens): registers += the row's scale x the runs' sums ----
        const int hp = (warp - T::kPromWarp0) >> 2, row = (warp & 3) * 32 + lane;
        const bool merged = kRuns == 1 && g.terms == 2 && g.n_tile <= 128;
        const uint32_t pfree0 = leader_addr(&bars->pfree[0]), half = g.n_tile / 2;
        const float* const scales = reinterpret_cast<const float*>(smem + T::kScaleOffset) + row;
        const uint32_t lane_base = ((uint32_t)(warp & 3) * 32u) << 16;
        float2 acc[BN / 4];
#pragma unroll
        for (int i = 0; i < BN / 4; ++i) acc[i] = make_float2(0.f, 0.f);
        uint32_t u = u_begin, b = 0;
        XSegment sg{0, 0, 0};
        const uint32_t total = u_end - u_begin;
        bool ok = true;
        for (uint32_t gb = 0; gb < total && ok; ++gb) {
            if (gb == 0 || b == sg.b1) {
                x_next_segment(u, u_end, nblk, sg);
                b = sg.b0;
            }
            if (!poll_or_fail(&bars->scales[gb & (kXScales - 1)], (gb / kXScales) & 1, bars, g.status, 192)) break;
            const float sc = scales[(gb & (kXScales - 1)) * kBM];
#pragma unroll 1
            for (int r = 0; r < kRuns && ok; ++r) {
                const uint32_t buf = kRuns == 4 ? (uint32_t)r : gb & 1;
                ok = poll_or_fail(&bars->accum[buf], (kRuns == 4 ? gb : gb >> 1) & 1, bars, g.status, 190);
                if (!ok) break;
                __syncwarp();
                tc_fence_after();
                // columns of these tokens; merged: those of their low terms n_tile / 2 further on (either CTA's
                // tokens are [high | low] there)
                const uint32_t ta = tmem + lane_base + buf * T::kPStride + (merged ? hp * g.n_tile : hp * half);
                if (BN <= 128 && merged) {
#pragma unroll
                    for (int c = 0; c < BN / 32; ++c) {
                        if ((uint32_t)c * 16 < half) {
                            uint32_t v0[16], v1[16];
                            tmem_ld16(ta + c * 16, v0);
                            tmem_ld16(ta + c * 16 + half, v1);
                            tmem_ld_wait();
#pragma unroll
                            for (int e = 0; e < 16; e += 2)
                                fma_f32x2(acc[c * 8 + e / 2], sc, __uint_as_float(v0[e]) + __uint_as_float(v1[e]),
                                          __uint_as_float(v0[e + 1]) + __uint_as_float(v1[e + 1]));
                        }
                    }
                } else {  // pairs of loads where the registers allow it: a load's latency is what a run's promotion consists of
                    constexpr int kLoads = BN <= 128 ? 2 : 1;
#pragma unroll
                    for (int c = 0; c < BN / 32; c += kLoads) {
                        if ((uint32_t)c * 16 < half) {
                            uint32_t v[kLoads][16];
#pragma unroll
                            for (int l = 0; l < kLoads; ++l) tmem_ld16(ta + (c + l) * 16, v[l]);
                            tmem_ld_wait();
#pragma unroll
                            for (int l = 0; l < kLoads; ++l)
#pragma unroll
                                for (int e = 0; e < 16; e += 2)
                                    fma_f32x2(acc[(c + l) * 8 + e / 2], sc, __uint_as_float(v[l][e]), __uint_as_float(v[l][e + 1]));
                        }
                    }
                }
                if (r == kRuns - 1 && b + 1 == sg.b1) break;  // the columns are needed once more
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(pfree0 + buf * 8);
            }
            if (!ok) break;
            if (++b == sg.b1) {
                // ---- the segment's sums leave: a whole tile is stored, the parts of a split tile add up in D or wait in
                // their slots for add_parts_kernel. They go back to the columns that the last run was read from, so that a
                // loop of a few instructions can store them: with one store per register in a row, code that is fetched for
                // one pass, 64 columns a thread took 3.9 us and 96 6.2 (now 2.1 and 3.8). ----
                asm volatile("griddepcontrol.wait;" ::: "memory");  // D zeroed, scales written
                const bool whole = sg.b0 == 0 && sg.b1 == nblk;
                const uint32_t m = tile_m0(sg.tile) + row;
                const uint32_t n0 = tile_n0(sg.tile) + hp * half;
                float* out = g.parts ? g.parts + ((uint64_t)slot * g.n_tile + hp * half) * 256 + rank * kBM + row : g.D + (uint64_t)n0 * g.stride_d + m;
                const uint32_t out_stride = g.parts ? 256u : g.stride_d;
                // the tokens' scales, one per lane (a load per column would be held back by the add before it)
                float inv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    inv[i] = 32u * i + lane < half && n0 + 32 * i + lane < g.N ? __ldcg(g.inv_scale + n0 + 32 * i + lane) : 0.f;
                const uint32_t last = kRuns == 4 ? 3u : gb & 1;
                const uint32_t ta = tmem + lane_base + last * T::kPStride + (merged ? hp * g.n_tile : hp * half);
#pragma unroll
                for (int c = 0; c < BN / 16; ++c) {
                    if ((uint32_t)c * 8 < half) tmem_st8(ta + c * 8, acc + c * 4);
                    acc[c * 4] = acc[c * 4 + 1] = acc[c * 4 + 2] = acc[c * 4 + 3] = make_float2(0.f, 0.f);
                }
                tmem_st_wait();
                const uint32_t cols = m < g.M && n0 < g.N ? min(half, g.N - n0) : 0u;  // that this thread stores
                const bool plain = whole || g.parts;
#pragma unroll 1
                for (uint32_t c = 0; c < half; c += 8) {
                    uint32_t v[8];
                    tmem_ld8(ta + c, v);
                    const float iv = c < 64 ? (c < 32 ? inv[0] : inv[1]) : (c < 96 ? inv[2] : inv[3]);
                    float x[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = __shfl_sync(0xFFFFFFFFu, iv, (c & 31) + e);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] *= __uint_as_float(v[e]);
                    if (plain) {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (c + e < cols) out[(uint64_t)e * out_stride] = x[e];
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (c + e < cols) atomicAdd(out + (uint64_t)e * out_stride, x[e]);
                    }
                    out += 8 * (uint64_t)out_stride;
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(pfree0 + last * 8);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's MMAs read this CTA's stages, its commits arrive here
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(T::kPBufs * T::kPStride)) : "memory");
    }
}

template <int TYPE, int BN, bool kFetch, int kRuns>
cudaError_t x_launch(const ExactGemm& p, const XPlan& plan, const ExactPrep& prep, cudaStream_t s) {
    using T = XTile<TYPE, BN, kFetch, kRuns>;
    auto kern = gemm_exact_kernel<TYPE, BN, kFetch, kRuns>;
    static std::atomic<uint64_t> attr_done{0};
    static std::atomic<int> max_pairs[64];
    if (cudaError_t e = ensure_dynamic_smem(kern, (int)T::kSmemBytes, attr_done); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(T::kThreads, 1, 1);
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
    // the promoters wait for registers that the others give back: the sum is that of T's static_assert (the build fails where a kernel
    // got another number: build.py)
    static const bool registers = [&] {
        cudaFuncAttributes fa{};
        return cudaFuncGetAttributes(&fa, kern) == cudaSuccess && fa.numRegs == T::kLaunchRegs;
    }();
    if (!registers) return cudaErrorNotSupported;
    const uint32_t n = plan.n_tiles;
    const XDeal deal = x_deal(n, plan.n_tile, plan.nblk, (uint32_t)pairs, x_cost(p, XW<TYPE>::kTerms == 2, plan.n_tile));
    const uint32_t G = deal.pairs, per = deal.per;
    const bool split = n % G != 0, parts = per > 2;
    cfg.numAttrs = 2;
    cfg.gridDim = dim3(2 * G, 1, 1);
    XArgs g{};
    g.A = p.A;
    g.a_end = p.A + (uint64_t)p.M * (p.K / block_size(TYPE)) * bytes_per_block(TYPE);
    g.D = p.D;
    g.inv_scale = plan.inv_scale;
    g.M = p.M;
    g.N = p.N;
    g.K = p.K;
    g.nblk = plan.nblk;
    g.stride_d = p.stride_d;
    g.n_row_pairs = plan.n_row_pairs;
    g.n_tiles = plan.n_tiles;
    g.n_tile = plan.n_tile;
    g.terms = p.bf16 ? 1u : 2u;
    g.groups = deal.groups;
    g.parts = parts ? plan.parts : nullptr;
    g.status = p.status;
    EncodeFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    CUtensorMap mx, mm, mw;
    const cuuint32_t estr[2] = {1, 1};
    const cuuint32_t box[2] = {64, plan.n_tile / 2};
    // rows: the high (or only) terms of all tokens, then the low terms
    const cuuint64_t xd[2] = {(cuuint64_t)plan.nblk * 256, (cuuint64_t)p.N * g.terms}, xs[1] = {(cuuint64_t)plan.nblk * 512};
    if (enc(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, plan.x, xd, xs, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    mm = mx;
    if constexpr (XW<TYPE>::kMin) {
        const cuuint64_t md[2] = {(cuuint64_t)plan.nblk * 64, p.N}, ms[1] = {(cuuint64_t)plan.nblk * 128};
        if (enc(&mm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, plan.sums, md, ms, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    mw = mx;
    if constexpr (!kFetch) {
        constexpr int kUnit = TYPE == T_Q8_0 ? 2 : 1;
        const cuuint64_t row_bytes = (cuuint64_t)plan.nblk * XW<TYPE>::kBlock;
        const cuuint64_t wd[2] = {row_bytes / kUnit, p.M}, ws[1] = {row_bytes};
        const cuuint32_t wbox[2] = {XW<TYPE>::kTmaRow / kUnit, kBM};
        if (enc(&mw, kUnit == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                const_cast<uint8_t*>(p.A), wd, ws, wbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    // the preparation goes out last, so that the GEMM's launch follows it at once and overlaps it
    if (cudaError_t e = prep.launch(prep.args, split && !parts, s); e != cudaSuccess) return e;
    if (cudaError_t e = cudaLaunchKernelEx(&cfg, kern, mx, mm, mw, g); e != cudaSuccess) return e;
    if (plan.launches) *plan.launches += parts ? 3 : 2;
    return parts ? launch_add_parts(plan.parts, p.D, p.M, p.N, 2 * kBM, plan.n_row_pairs, plan.n_tile, n, per, p.stride_d, s) : cudaSuccess;
}

template <int TYPE, bool kFetch>
cudaError_t x_launch_bn(const ExactGemm& p, const XPlan& plan, const ExactPrep& prep, cudaStream_t s) {
    if (p.fine) {
        // Two-term types: tiles of at most 64 tokens, whose sets have two stages, a fill of a block each.
        if constexpr (XW<TYPE>::kTerms == 1) {
            if (plan.n_tile > 64) return x_launch<TYPE, 128, kFetch, 4>(p, plan, prep, s);
        }
        return plan.n_tile <= 64 ? x_launch<TYPE, 64, kFetch, 4>(p, plan, prep, s) : cudaErrorInvalidConfiguration;
    }
    if (plan.n_tile <= 64) return x_launch<TYPE, 64, kFetch, 1>(p, plan, prep, s);
    if (plan.n_tile <= 128) return x_launch<TYPE, 128, kFetch, 1>(p, plan, prep, s);
    return plan.n_tile <= 192 ? x_launch<TYPE, 192, kFetch, 1>(p, plan, prep, s) : x_launch<TYPE, 256, kFetch, 1>(p, plan, prep, s);
}

}  // namespace
}  // namespace zc
