// Row matvec: y (+)= W x for the sizes and types the streaming kernels leave: every matrix below 2 MB, and Q5_K and Q8_0 of
// any size (src/shaders/dmmv_q8_0.comp:80-108, dmmv_q5k.comp and their siblings).
//
// A warp covers 256 columns of a row per step, eight weights per lane, all lanes' bytes contiguous. Weights become floats
// exactly (a byte permuted under the exponent of 2^23, one subtraction) and meet x in f32, two at a time. NR rows per warp
// share the loads of x; WK warps of a CTA share a row's steps, so that short matrices still fill the SMs and a row is a
// few loads deep.
// Bound: HBM and instruction issue for large matrices, below a few MB the latency of a launch: the first steps' weights are
// requested before the dependency wait, so that only x and the arithmetic lie behind it (in a chain of launches Q8_0 512 x
// 2048 2.6 us, 2.9 requested after the wait; 2048 x 2048 3.6 and 4.8). Weights are not written by the kernel in front.
#include "common.cuh"
#include "kernels.h"
#include "stream_common.cuh"

namespace zc {
namespace {

constexpr int kRowWarps = 8;

struct RowArgs {
    const uint8_t* A;
    const float* x;
    float* y;
    uint32_t M, K, acc_mode;
};

// bytes I and I + 1 of u as exact floats u[I] - bias, u[I + 1] - bias
template <int I>
__device__ __forceinline__ float2 byte_pair(uint32_t u, float bias) {
    const float a = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7440 | I)), b = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7440 | (I + 1)));
    float2 r;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %4};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a), "f"(b), "f"(-8388608.f - bias));
    return r;
}
__device__ __forceinline__ void fma_pair(float2& acc, float2 a, float bx, float by) {
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%0, %1};\n\t"
        "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "f"(a.x), "f"(a.y), "f"(bx), "f"(by));
}
// sum of the four bytes of u (less bias) times v
__device__ __forceinline__ float dot4(uint32_t u, float bias, const float4& v) {
    float2 s = make_float2(0.f, 0.f);
    fma_pair(s, byte_pair<0>(u, bias), v.x, v.y);
    fma_pair(s, byte_pair<2>(u, bias), v.z, v.w);
    return s.x + s.y;
}
__device__ __forceinline__ float sum4(const float4& v) { return (v.x + v.y) + (v.z + v.w); }
__device__ __forceinline__ float small_f(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.f; }  // v < 2^23

// What a lane loads of one row's step and how it multiplies it. kBytes: bytes of 256 columns; x_cols: where the lane's two
// runs of four columns begin (for the types of 32-column blocks both lie in one block).
template <uint32_t TYPE>
struct Lane;

template <>
struct Lane<T_Q8_0> {  // four lanes per 34-byte block, which is only 2-byte aligned
    static constexpr uint32_t kBytes = 272;
    uint32_t w[3], d;
    static __device__ __forceinline__ void x_cols(int l, uint32_t& a, uint32_t& b) {
        a = 8 * l;
        b = a + 4;
    }
    __device__ __forceinline__ void load(const uint8_t* p, int l) {
        const uint8_t* b = p + 34 * (l >> 2);
        const uintptr_t q = reinterpret_cast<uintptr_t>(b + 2 + 8 * (l & 3));
        const uint32_t* a = reinterpret_cast<const uint32_t*>(q & ~(uintptr_t)3);
        w[0] = __ldcs(a);
        w[1] = __ldcs(a + 1);
        w[2] = (q & 2) ? __ldcs(a + 2) : 0u;
        d = __ldcs(reinterpret_cast<const unsigned short*>(b));
    }
    __device__ __forceinline__ float dot(const uint8_t* p, int l, const float4& xa, const float4& xb, float, float) const {
        const uint32_t sh = (reinterpret_cast<uintptr_t>(p) + 34 * (l >> 2) + 2) & 2u ? 16u : 0u;
        const uint32_t lo = __funnelshift_r(w[0], w[1], sh) ^ 0x80808080u, hi = __funnelshift_r(w[1], w[2], sh) ^ 0x80808080u;
        return h2f(d) * (dot4(lo, 128.f, xa) + dot4(hi, 128.f, xb));
    }
};

template <bool kFive>
struct LaneK {  // Q4_K / Q5_K: word l of the block's nibble bytes: sub-blocks 2j (low) and 2j + 1 (high), j = l / 8
    static constexpr uint32_t kBytes = kFive ? 176 : 144;
    uint32_t w, h;
    uint4 hd;
    static __device__ __forceinline__ void x_cols(int l, uint32_t& a, uint32_t& b) {
        a = 64 * (l >> 3) + 4 * (l & 7);
        b = a + 32;
    }
    __device__ __forceinline__ void load(const uint8_t* p, int l) {
        hd = __ldcs(reinterpret_cast<const uint4*>(p));
        w = __ldcs(reinterpret_cast<const uint32_t*>(p + kBytes - 128) + l);
        if (kFive) h = __ldcs(reinterpret_cast<const uint32_t*>(p + 16) + (l & 7));
    }
    __device__ __forceinline__ float dot(const uint8_t*, int l, const float4& xa, const float4& xb, float sa, float sb) const {
        const int j = l >> 3;
        uint32_t lo = w & 0x0F0F0F0Fu, hi = (w >> 4) & 0x0F0F0F0Fu;
        if (kFive) {  // bits 2j and 2j + 1 of the qh bytes
            lo |= ((h >> (2 * j)) & 0x01010101u) << 4;
            hi |= ((h >> (2 * j + 1)) & 0x01010101u) << 4;
        }
        // getScaleMinK4 (src/compute/forward.zig:229-238), four sub-blocks as bytes
        uint32_t sc = j < 2 ? hd.y & 0x3F3F3F3Fu : (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u);
        uint32_t mn = j < 2 ? hd.z & 0x3F3F3F3Fu : ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u);
        sc >>= 16 * (j & 1);
        mn >>= 16 * (j & 1);
        const float q = small_f(sc & 0xFFu) * dot4(lo, 0.f, xa) + small_f((sc >> 8) & 0xFFu) * dot4(hi, 0.f, xb);
        const float m = small_f(mn & 0xFFu) * sa + small_f((mn >> 8) & 0xFFu) * sb;
        return h2f(hd.x) * q - h2f(hd.x >> 16) * m;
    }
};
template <>
struct Lane<T_Q4_K> : LaneK<false> {};
template <>
struct Lane<T_Q5_K> : LaneK<true> {};

template <>
struct Lane<T_Q6_K> {  // word l % 16 of half l / 16 of ql: columns 128 n + 4 (l % 16) (low) and 64 further on (high)
    static constexpr uint32_t kBytes = 210;
    uint32_t w[2], h[2], sc, d;
    static __device__ __forceinline__ void x_cols(int l, uint32_t& a, uint32_t& b) {
        a = 128 * (l >> 4) + 4 * (l & 15);
        b = a + 64;
    }
    __device__ __forceinline__ void load(const uint8_t* p, int l) {
        const int n = l >> 4, c = l & 15;
        const bool odd = reinterpret_cast<uintptr_t>(p) & 2;  // blocks are only 2-byte aligned
        const uint32_t* a = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3);
        w[0] = __ldcs(a + l);
        w[1] = odd ? __ldcs(a + l + 1) : 0u;
        h[0] = __ldcs(a + 32 + 8 * n + (c & 7));
        h[1] = odd ? __ldcs(a + 33 + 8 * n + (c & 7)) : 0u;
        // scales 8n + c / 4 (low) and 8n + 4 + c / 4 (high)
        sc = (uint32_t)__ldcs(p + 192 + 8 * n + (c >> 2)) | ((uint32_t)__ldcs(p + 196 + 8 * n + (c >> 2)) << 8);
        d = __ldcs(reinterpret_cast<const unsigned short*>(p + 208));
    }
    __device__ __forceinline__ float dot(const uint8_t* p, int l, const float4& xa, const float4& xb, float, float) const {
        const uint32_t sh = reinterpret_cast<uintptr_t>(p) & 2 ? 16u : 0u, up = ((l & 15) >> 3) * 2;
        const uint32_t q = __funnelshift_r(w[0], w[1], sh), t = __funnelshift_r(h[0], h[1], sh) >> up;
        const uint32_t lo = (q & 0x0F0F0F0Fu) | ((t & 0x03030303u) << 4), hi = ((q >> 4) & 0x0F0F0F0Fu) | (t & 0x30303030u);
        const float s0 = small_f((sc & 0xFFu) ^ 0x80u) - 128.f, s1 = small_f((sc >> 8) ^ 0x80u) - 128.f;
        return h2f(d) * (s0 * dot4(lo, 32.f, xa) + s1 * dot4(hi, 32.f, xb));
    }
};

template <>
struct Lane<T_MXFP4> {  // four lanes per 17-byte block: nibble bytes 4q .. : columns 4q (low) and 16 + 4q (high)
    static constexpr uint32_t kBytes = 136;
    uint32_t w[2], e;
    static __device__ __forceinline__ void x_cols(int l, uint32_t& a, uint32_t& b) {
        a = 32 * (l >> 2) + 4 * (l & 3);
        b = a + 16;
    }
    __device__ __forceinline__ void load(const uint8_t* p, int l) {
        const uint8_t* b = p + 17 * (l >> 2);
        const uintptr_t q = reinterpret_cast<uintptr_t>(b + 1 + 4 * (l & 3));
        const uint32_t* a = reinterpret_cast<const uint32_t*>(q & ~(uintptr_t)3);
        w[0] = __ldcs(a);
        w[1] = (q & 3) ? __ldcs(a + 1) : 0u;
        e = __ldcs(b);
    }
    // four nibbles, one per byte, times x
    static __device__ __forceinline__ float nib_dot(uint32_t nib, const float4& x) {
        const uint32_t sel = nib & 0x07070707u, s = (nib >> 3) & 0x01010101u;
        const uint32_t s4 = sel | (sel >> 4), packed = __byte_perm(s4, 0u, 0x4420);  // bytes 0 and 2: two selectors each
        // magnitudes 2 x {0, .5, 1, 1.5, 2, 3, 4, 6} by a byte table; 16 + mag or 16 - mag in every byte (mag <= 12, so
        // that nothing carries or borrows across bytes)
        const uint32_t mag = __byte_perm(0x03020100u, 0x0C080604u, packed);
        const uint32_t neg = mag & (s * 0xFFu);
        return dot4(0x10101010u + mag - 2u * neg, 16.f, x);
    }
    __device__ __forceinline__ float dot(const uint8_t* p, int l, const float4& xa, const float4& xb, float, float) const {
        const uint32_t sh = ((reinterpret_cast<uintptr_t>(p) + 17 * (l >> 2) + 1) & 3u) * 8u;
        const uint32_t q = __funnelshift_r(w[0], w[1], sh);
        return (0.5f * (nib_dot(q & 0x0F0F0F0Fu, xa) + nib_dot((q >> 4) & 0x0F0F0F0Fu, xb))) * e8m0_to_f32(e);
    }
};

template <uint32_t TYPE, int NR, int WK, int UN>
__global__ void __launch_bounds__(kRowWarps * 32) dmmv_row_kernel(const RowArgs a) {
    using L = Lane<TYPE>;
    constexpr int kGroups = kRowWarps / WK;  // row groups of a CTA
    constexpr bool kSums = TYPE == T_Q4_K || TYPE == T_Q5_K;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = warp / WK, wk = warp % WK;
    const uint64_t row_bytes = (uint64_t)(a.K / block_size(TYPE)) * bytes_per_block(TYPE);
    const uint32_t row0 = (blockIdx.x * kGroups + grp) * NR;
    const uint8_t* rows[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) rows[r] = a.A + (uint64_t)min(row0 + r, a.M - 1) * row_bytes;
    const uint32_t n_steps = (a.K + 255) >> 8;
    uint32_t ca, cb;
    L::x_cols(lane, ca, cb);
    L buf[UN][NR];
    auto live = [&](uint32_t s) { return s * 256 + (block_size(TYPE) == 256 ? 0u : ca) < a.K; };
    auto load = [&](uint32_t s0) {  // steps s0, s0 + WK, ...
#pragma unroll
        for (int u = 0; u < UN; ++u)
            if (live(s0 + u * WK)) {
#pragma unroll
                for (int r = 0; r < NR; ++r) buf[u][r].load(rows[r] + (uint64_t)(s0 + u * WK) * L::kBytes, lane);
            }
    };
    load(wk);
    chain_wait();
    chain_release();
    const float* x = a.x;
    float* y = a.y;
    after_wait(x);
    after_wait(y);
    float acc[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = 0.f;
    for (uint32_t s0 = wk; s0 < n_steps; s0 += UN * WK) {
        float4 xa[UN], xb[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u)
            if (live(s0 + u * WK)) {
                xa[u] = __ldg(reinterpret_cast<const float4*>(x + (s0 + u * WK) * 256 + ca));
                xb[u] = __ldg(reinterpret_cast<const float4*>(x + (s0 + u * WK) * 256 + cb));
            }
#pragma unroll
        for (int u = 0; u < UN; ++u)
            if (live(s0 + u * WK)) {
                const float sa = kSums ? sum4(xa[u]) : 0.f, sb = kSums ? sum4(xb[u]) : 0.f;
#pragma unroll
                for (int r = 0; r < NR; ++r)
                    acc[r] += buf[u][r].dot(rows[r] + (uint64_t)(s0 + u * WK) * L::kBytes, lane, xa[u], xb[u], sa, sb);
            }
        if (s0 + UN * WK < n_steps) load(s0 + UN * WK);
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = warp_sum(acc[r]);
    if constexpr (WK > 1) {
        __shared__ float part[kRowWarps][NR];
        if (lane == 0)
#pragma unroll
            for (int r = 0; r < NR; ++r) part[warp][r] = acc[r];
        __syncthreads();
        if (wk == 0 && lane < NR && row0 + lane < a.M) {
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < WK; ++i) s += part[warp + i][lane];
            y[row0 + lane] = a.acc_mode ? y[row0 + lane] + s : s;
        }
    } else if (lane == 0) {
#pragma unroll
        for (int r = 0; r < NR; ++r)
            if (row0 + r < a.M) y[row0 + r] = a.acc_mode ? y[row0 + r] + acc[r] : acc[r];
    }
}

template <uint32_t TYPE, int NR, int WK, int UN>
cudaError_t launch(const RowArgs& a, cudaStream_t s) {
    const uint32_t rows = kRowWarps / WK * NR;
    return launch_chained(dmmv_row_kernel<TYPE, NR, WK, UN>, dim3((a.M + rows - 1) / rows), dim3(kRowWarps * 32), 0, s, a);
}

template <uint32_t TYPE>
cudaError_t launch_type(const RowArgs& a, uint32_t sms, cudaStream_t s) {
    // Rows per warp: as many as leave every SM its 32 warps. Below that, warps per row: until there are 16 warps per SM
    // or a warp is left with one step.
    const uint32_t steps = (a.K + 255) >> 8;
    if (TYPE == T_Q8_0 || TYPE == T_Q5_K) {
        if (a.M >= sms * 32 * 4) return launch<TYPE, 4, 1, 1>(a, s);
        if (a.M >= sms * 32 * 2) return launch<TYPE, 2, 1, 2>(a, s);
    }
    if (a.M >= sms * 16 || steps < 2) return launch<TYPE, 1, 1, 4>(a, s);
    if (a.M >= sms * 8 || steps < 4) return launch<TYPE, 1, 2, 4>(a, s);
    if (a.M >= sms * 4 || steps < 8) return launch<TYPE, 1, 4, 4>(a, s);
    return launch<TYPE, 1, 8, 4>(a, s);
}

}  // namespace

bool row_dmmv_eligible(uint32_t type, const DmmvArgs& d) {
    if (d.push.world || d.merge.partial) return false;
    if (type == T_Q4_K || type == T_Q5_K) return (reinterpret_cast<uintptr_t>(d.A) & 15u) == 0;
    return type == T_Q8_0 || type == T_Q6_K || type == T_MXFP4;
}

cudaError_t launch_row_dmmv(uint32_t type, const DmmvArgs& d, cudaStream_t s) {
    const RowArgs a{d.A, d.x, d.y, d.M, d.K, d.acc_mode};
    const uint32_t sms = d.sm_count ? (uint32_t)d.sm_count : 148u;
    switch (type) {
        case T_Q4_K: return launch_type<T_Q4_K>(a, sms, s);
        case T_Q5_K: return launch_type<T_Q5_K>(a, sms, s);
        case T_Q6_K: return launch_type<T_Q6_K>(a, sms, s);
        case T_Q8_0: return launch_type<T_Q8_0>(a, sms, s);
        case T_MXFP4: return launch_type<T_MXFP4>(a, sms, s);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace zc
