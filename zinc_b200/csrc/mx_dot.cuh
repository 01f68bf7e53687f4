// The dot product of MXFP4 blocks (17 bytes: E8M0 scale + 32 E2M1 nibbles; src/compute/forward.zig:431-465) with one vector on the
// tensor cores, as the decode kernels share it.
//
// A byte of a block (two nibbles) becomes two fp16 weights with one conversion instruction, exactly. The activations are
// two fp16 terms per element (scaled by a power of two per 256 elements so that the largest lies in [2^9, 2^10): 22
// significant bits, absolute error 2^-34 of the largest). mma.sync m16n8k16 multiplies 16 rows by them in f32.
// Lane (g, t) owns one block of rows g and g + 8 at a time; its k slots carry that block's elements, and B is
// block-diagonal: column 2 t + p is term p for the k slots of lane t's block and zero elsewhere, so D column 2 t + p is
// that block's dot product with term p alone and lands on the lane that owns the block, which applies its scale.
// A unit is 16 rows x 16 blocks (512 columns); in step q lane t owns block q + 4 t: four blocks are 68 bytes, 17 words, so
// that the 32-bit reads of the four lanes of a row fall on different banks.
// (The E2M1 -> signed byte tables and int8 digits of an earlier form took twice the instructions per weight.)
#pragma once

#include "stream_skel.cuh"

namespace zc {
namespace {

constexpr uint32_t kMxUnitBlocks = 16, kMxUnitBytes = kMxUnitBlocks * 17;  // 272 bytes of a row
constexpr uint32_t kMxPitch = 304;           // 288-byte aligned superset + 16: rows 12 banks apart
constexpr uint32_t kMxTable = 2048 + 8;      // bytes per unit's columns of x: terms, scales
constexpr uint32_t kMxZeros = 1024;          // zeros the lanes of dead columns read (one step's table is 512 bytes)

// One warp per 256 elements; lane = b * 4 + j holds, for block b of the chunk, the elements of MMA step j: 4j .. 4j+3 and
// 16 + 4j .. 16 + 4j+3. Elements at or beyond K read as zero.
struct MxX {
    float4 lo, hi;
};
__device__ __forceinline__ uint32_t mx_pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t mx_rest(float a, float b, uint32_t h) {
    const __half2 v = *reinterpret_cast<const __half2*>(&h);
    return mx_pack(a - __low2float(v), b - __high2float(v));
}
// Terms of x in B-operand order, xf[((step * 4 + j) * 2 + term) * 4 + t] with step = 4 * unit + q, and xs, per 256 elements 2^-f.
// kTwice: written to another CTA of the cluster too, whose shared memory is `also` on from this one's.
template <bool kTwice = false>
__device__ __forceinline__ void mx_prep(uint4* xf, float* xs, const MxX& r, uint32_t chunk, int lane, uint32_t also = 0) {
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
    const uint4 h = make_uint4(mx_pack(lo.x, hi.x), mx_pack(lo.y, hi.y), mx_pack(lo.z, hi.z), mx_pack(lo.w, hi.w));
    const uint4 l = make_uint4(mx_rest(lo.x, hi.x, h.x), mx_rest(lo.y, hi.y, h.y), mx_rest(lo.z, hi.z, h.z), mx_rest(lo.w, hi.w, h.w));
    // block b of chunk c is block q + 4 t of unit c / 2
    const uint32_t q = b & 3, t = 2 * (chunk & 1) + (b >> 2), u = (((chunk >> 1) * 4 + q) * 4 + j) * 2;
    xf[u * 4 + t] = h;
    xf[(u + 1) * 4 + t] = l;
    if (lane == 0) xs[chunk] = __uint_as_float((E - 9u) << 23);
    if constexpr (kTwice) {
        const uint32_t o = smem_u32(xf + u * 4 + t) + also;
        st_cluster(o, h);
        st_cluster(o + 64, l);
        if (lane == 0) st_cluster(smem_u32(xs + chunk) + also, (E - 9u) << 23);
    }
}

// the four bytes of x (a low and a high nibble each) as pairs of fp16
__device__ __forceinline__ void e2m1x8_to_f16(uint32_t x, uint32_t (&o)[4]) {
    asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, b;\n\tcvt.rn.f16x2.e2m1x2 %2, c;\n\tcvt.rn.f16x2.e2m1x2 %3, d;\n\t}"
        : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3])
        : "r"(x));
}
__device__ __forceinline__ uint32_t mx_lds(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
// Where a lane reads x, and the sums it makes of a unit's rows g and g + 8.
struct MxLane {
    uint32_t xu, xu_step, xs_s, g, t;
    __device__ __forceinline__ void init(uint32_t xf, uint32_t xs, uint32_t zeros, int lane) {
        g = lane >> 2;
        t = lane & 3;
        const bool live = (g >> 1) == t;
        xu = live ? xf + ((g & 1) * 4 + t) * 16u : zeros + ((g >> 1) + 1) * 16u;
        xu_step = live ? 512u : 0u;  // 32 entries of 16 bytes per step
        xs_s = xs + 4u * (t >> 1);
    }
    // pa, pb: the unit's first byte of rows g and g + 8 in shared memory; left: blocks from there to the end of the row; kb: the unit's
    // place in x
    __device__ __forceinline__ void dot(uint32_t pa, uint32_t pb, uint32_t left, uint32_t kb, float (&acc)[2]) const {
        // this lane's blocks q + 4 t of the two rows: all at the same byte position within their words
        pa += 68 * t;
        pb += 68 * t;
        const float xs = lds_f1(xs_s + kb * 8);
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
                wa[i] = mx_lds((qa & ~3u) + 4 * i);
                wb[i] = mx_lds((qb & ~3u) + 4 * i);
            }
            const uint32_t xq = xu + (kb * 4 + q) * xu_step;
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
                acc[0] = fmaf(e8m0_to_f32(ea) * xs, (d[0] + e[0]) + (d[1] + e[1]), acc[0]);
                acc[1] = fmaf(e8m0_to_f32(eb) * xs, (d[2] + e[2]) + (d[3] + e[3]), acc[1]);
            }
        }
    }
};

}  // namespace
}  // namespace zc
