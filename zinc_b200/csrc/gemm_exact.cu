// Preparation of the activations and dispatch of the f32-accurate prefill GEMM (gemm_exact.cuh).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "stream_common.cuh"

namespace zc {
namespace {

constexpr int kPrepMost = 1024;  // threads

struct PrepArgs {
    const void* X;
    __half* x;          // [terms][N][nblk * 256]
    __half* sums;       // [N][nblk * 64], Q4_K / Q5_K
    float* inv_scale;   // [N]
    float* D;           // zeroed where tiles lie on two CTA pairs
    uint32_t tokens, K, nblk, M, stride_b, stride_d;
    uint32_t sms;
    bool sums_on, zero, vec;
};

// Column of a 64-column group where the two runs of four of chunk c begin: the order in which the type's unpacking
// yields its weights (gemm_exact.cuh); within a run the order is 0, 2, 1, 3.
template <int ORDER>
__device__ __forceinline__ void chunk_columns(int c, uint32_t& a, uint32_t& b) {
    if (ORDER == 0) {         // Q4_K, Q5_K: low and high nibbles of a word
        a = 4 * c;
        b = 32 + 4 * c;
    } else if (ORDER == 1) {  // Q6_K, Q8_0: two words of a 32-column group
        a = 32 * (c >> 2) + 8 * (c & 3);
        b = a + 4;
    } else {                  // MXFP4: low and high nibbles of a 32-column block
        a = 32 * (c >> 2) + 4 * (c & 3);
        b = a + 16;
    }
}

// VEC: rows of whole, aligned groups of four (the code is fetched for one pass: without the general case there is less of it)
template <bool BF16, bool VEC>
__device__ __forceinline__ float4 load4(const void* row, uint32_t k, uint32_t K) {
    if (VEC) {
        if (k >= K) return make_float4(0.f, 0.f, 0.f, 0.f);
        if (!BF16) return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(row) + k));
        const uint2 t = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(row) + k));
        return make_float4(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xFFFF0000u), __uint_as_float(t.y << 16),
                           __uint_as_float(t.y & 0xFFFF0000u));
    }
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (BF16) v[i] = k + i < K ? __bfloat162float(static_cast<const __nv_bfloat16*>(row)[k + i]) : 0.f;
        else v[i] = k + i < K ? static_cast<const float*>(row)[k + i] : 0.f;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// what the fp16 rounding of (a, b) left over
__device__ __forceinline__ uint32_t pack_rest(float a, float b, uint32_t h) {
    const __half2 v = *reinterpret_cast<const __half2*>(&h);
    return pack_h2(a - __low2float(v), b - __high2float(v));
}

// One CTA per token: power-of-two scale from the largest element, fp16 terms in the order the GEMM consumes them,
// sums over 32-column sub-blocks, and (split tiles) the token's row of D set to zero. Bound: the bytes of X, D and
// the terms, 4 + 4 per element, and for few tokens the latency of one read behind the other: a thread's two chunks of a row of
// up to 16384 columns stay in its registers between the scale and the terms (read twice, four elements at a time: 4096 columns,
// 128 tokens
// 5.8 us, 658 tokens with D to zero 9.0; now 4.5 and 8.1, both with L2 cold).
template <int ORDER, bool BF16, bool VEC>
__global__ void __maxnreg__(40) exact_prep_kernel(const PrepArgs a) {
    chain_wait();
    chain_release();  // the GEMM's set-up and its first weight blocks overlap this kernel
    __shared__ float s_max[kPrepMost / 32];
    const uint32_t t = blockIdx.x, tid = threadIdx.x, threads = blockDim.x;
    const void* X = a.X;
    after_wait(X);
    const void* row = static_cast<const uint8_t*>(X) + (uint64_t)t * a.stride_b * (BF16 ? 2 : 4);
    const uint32_t chunks = a.nblk * 32;  // eight lanes per 64-column group, whole warps
    float4 va[2], vb[2];
    auto load = [&](uint32_t q0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t q = q0 + i * threads;
            uint32_t ka, kb;
            chunk_columns<ORDER>(q & 7, ka, kb);
            va[i] = vb[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q < chunks) {
                va[i] = load4<BF16, VEC>(row, (q >> 3) * 64 + ka, a.K);
                vb[i] = load4<BF16, VEC>(row, (q >> 3) * 64 + kb, a.K);
            }
        }
    };
    float mx = 0.f;
    for (uint32_t q0 = tid; q0 < chunks; q0 += 2 * threads) {
        load(q0);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(va[i].x), fabsf(va[i].y)), fmaxf(fabsf(va[i].z), fabsf(va[i].w))));
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(vb[i].x), fabsf(vb[i].y)), fmaxf(fabsf(vb[i].z), fabsf(vb[i].w))));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    if ((tid & 31) == 0) s_max[tid >> 5] = mx;
    if (a.zero) {
        float* d = a.D + (uint64_t)t * a.stride_d;
        if ((reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
            for (uint32_t m = tid * 4; m + 4 <= a.M; m += threads * 4) *reinterpret_cast<float4*>(d + m) = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tid < (a.M & 3u)) d[(a.M & ~3u) + tid] = 0.f;
        } else {
            for (uint32_t m = tid; m < a.M; m += threads) d[m] = 0.f;
        }
    }
    __syncthreads();
    mx = s_max[tid & 31 & (threads / 32 - 1)];  // the number of warps is a power of two
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    // Largest element to [2^14, 2^15), the top of fp16's range, so that an element keeps its 22 bits down to 2^-17 of the
    // largest; the inverse stays a normal number. Types with mins: their weights are 2^-10 of their value (gemm_exact.cuh),
    // and the sums are brought down to match, below 2^15 too.
    const uint32_t e = __float_as_uint(mx) >> 23;
    const uint32_t f = min(268u - e, 252u);
    const float scale = __uint_as_float(f << 23);
    if (tid == 0) a.inv_scale[t] = __uint_as_float((ORDER == 0 ? 264u - f : 254u - f) << 23);

    uint4* out = reinterpret_cast<uint4*>(a.x + (uint64_t)t * a.nblk * 256);
    const uint64_t low = (uint64_t)gridDim.x * a.nblk * 32;  // 16-byte chunks to the low term
    uint4* sums = reinterpret_cast<uint4*>(a.sums + (uint64_t)t * a.nblk * 64);
    const bool held = chunks <= 2 * threads;
    for (uint32_t q0 = tid; q0 < chunks; q0 += 2 * threads) {
        if (!held) load(q0);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t q = q0 + i * threads;
            if (q >= chunks) break;
            const uint32_t g = q >> 3;
            const int c = q & 7;
            const float4 xa = make_float4(va[i].x * scale, va[i].y * scale, va[i].z * scale, va[i].w * scale);
            const float4 xb = make_float4(vb[i].x * scale, vb[i].y * scale, vb[i].z * scale, vb[i].w * scale);
            uint4 hi;
            hi.x = pack_h2(xa.x, xa.z);
            hi.y = pack_h2(xa.y, xa.w);
            hi.z = pack_h2(xb.x, xb.z);
            hi.w = pack_h2(xb.y, xb.w);
            out[q] = hi;
            if (!BF16) {
                uint4 lo;
                lo.x = pack_rest(xa.x, xa.z, hi.x);
                lo.y = pack_rest(xa.y, xa.w, hi.y);
                lo.z = pack_rest(xb.x, xb.z, hi.z);
                lo.w = pack_rest(xb.y, xb.w, hi.w);
                out[low + q] = lo;
            }
            if (ORDER == 0 && a.sums_on) {
                float sa = (xa.x + xa.y) + (xa.z + xa.w), sb = (xb.x + xb.y) + (xb.z + xb.w);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) {
                    sa += __shfl_xor_sync(0xFFFFFFFFu, sa, o);
                    sb += __shfl_xor_sync(0xFFFFFFFFu, sb, o);
                }
                sa *= 1.f / 32.f;
                sb *= 1.f / 32.f;
                // a block's row: sub-block sums as [high 8][high 8][low 8][zeros 8], against the weights' min terms
                // [high][low][high][zeros]
                uint32_t* sp = reinterpret_cast<uint32_t*>(sums + (uint64_t)(g >> 2) * 8) + (g & 3);
                const uint32_t h = pack_h2(sa, sb);
                if (c == 0) sp[0] = h;
                if (c == 1) sp[4] = h;
                if (c == 2) sp[8] = pack_rest(sa, sb, h);
                if (c == 3) sp[12] = 0u;
            }
        }
    }
}

template <int ORDER, bool BF16>
cudaError_t launch_prep(const void* args, bool zero, cudaStream_t s) {
    PrepArgs a = *static_cast<const PrepArgs*>(args);
    a.zero = zero;
    // a whole row in the threads' registers where there are few tokens; beyond two CTAs to an SM the second read costs less than
    // the occupancy (Q5_K 407 x 10752, 1268 tokens: the whole product 61.6 us with 1024 threads, 49.2 with 256)
    uint32_t threads = 256;
    while (a.tokens <= 2 * a.sms && threads < kPrepMost && threads < a.nblk * 16) threads *= 2;
    return launch_chained(a.vec ? exact_prep_kernel<ORDER, BF16, true> : exact_prep_kernel<ORDER, BF16, false>, dim3(a.tokens), dim3(threads), 0, s, a);
}

// D = the sum of a tile's parts, in their order: [tile][part][token][rows]. One CTA: 1024 / rows tokens of a tile. Bound: the
// parts' bytes, which the kernel in front has left in L2, and the launch. It costs the smallest products 3 to 5 us over
// atomic adds in any order (Q4_K 512 x 2048, 16 tokens, call behind call 8.7 -> 11.9, 1024 x 4096, 64 tokens 11.3 -> 15.9) and
// 4096 x 4096, 64 tokens 1 (17.4 -> 18.5). Released early by the GEMM it was no sooner done. Slots that the last of a
// tile's warps adds up within the GEMM: 1024 x 4096 25.6 us where this takes 21.5 (with L2 cold), 256 tokens of 4096 x 4096
// 60 and 40.
// Four rows of one column a thread, four parts read at once: with two columns behind one another and an unrolled loop and its
// rest (code that is fetched for one pass) Q4_K f32 4096 x 4096, 32 tokens took 17.5 us, now 16.2, Q8_0 417 x 9248, 19 tokens
// 22.5 and 19.0.
template <uint32_t ROWS>
__global__ void __launch_bounds__(256)
add_parts_kernel(const float* parts, float* D, uint32_t M, uint32_t N, uint32_t row_tiles, uint32_t n_tile, uint32_t per, uint32_t stride_d) {
    chain_wait();
    chain_release();
    after_wait(parts);
    const uint32_t tile = blockIdx.x, r = threadIdx.x * 4 % ROWS, c = blockIdx.y * (1024 / ROWS) + threadIdx.x * 4 / ROWS;
    const uint32_t m = tile % row_tiles * ROWS + r, n = tile / row_tiles * n_tile + c;
    if (m < M && c < n_tile && n < N) {
        const float* p = parts + ((uint64_t)tile * per * n_tile + c) * ROWS + r;
        float4 s = make_float4(-0.f, -0.f, -0.f, -0.f);  // leaves what is added to it as it is
#pragma unroll 1
        for (uint32_t i = 0; i < per; i += 4) {
            float4 v[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (i + j < per) v[j] = __ldcg(reinterpret_cast<const float4*>(p + (uint64_t)(i + j) * n_tile * ROWS));
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (i + j < per) s = make_float4(s.x + v[j].x, s.y + v[j].y, s.z + v[j].z, s.w + v[j].w);
        }
        float* d = D + (uint64_t)n * stride_d + m;
        if (m + 4 <= M && (reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
            *reinterpret_cast<float4*>(d) = s;
        } else {
            d[0] = s.x;
            if (m + 1 < M) d[1] = s.y;
            if (m + 2 < M) d[2] = s.z;
            if (m + 3 < M) d[3] = s.w;
        }
    }
}

cudaError_t launch_type(const ExactGemm& p, const XPlan& plan, const ExactPrep& prep, cudaStream_t s) {
    switch (p.type) {
        case T_Q4_K: return launch_exact_q4k(p, plan, prep, s);
        case T_Q5_K: return launch_exact_q5k(p, plan, prep, s);
        case T_Q6_K: return launch_exact_q6k(p, plan, prep, s);
        case T_Q8_0: return launch_exact_q8(p, plan, prep, s);
        case T_MXFP4: return launch_exact_mxfp4(p, plan, prep, s);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace

cudaError_t launch_add_parts(const float* parts, float* D, uint32_t M, uint32_t N, uint32_t rows, uint32_t row_tiles, uint32_t n_tile,
                             uint32_t tiles, uint32_t per, uint32_t stride_d, cudaStream_t s) {
    return launch_chained(rows == 256 ? add_parts_kernel<256> : add_parts_kernel<128>, dim3(tiles, (n_tile * rows + 1023) / 1024), dim3(256), 0, s,
                          parts, D, M, N, row_tiles, n_tile, per, stride_d);
}

bool mul_mm_exact_eligible(uint32_t type, const uint8_t* A, uint32_t M, uint32_t N, uint32_t K) {
    if (type != T_Q4_K && type != T_Q5_K && type != T_Q6_K && type != T_Q8_0 && type != T_MXFP4) return false;
    if (reinterpret_cast<uintptr_t>(A) & 15u) return false;
    const uint64_t nblk = (K + 255) >> 8;
    // one token's terms must fit the scratch; unit counts stay in 32 bits
    return nblk * 256 * 8 < kExactTermBytes / 64 && ((uint64_t)(M + 255) / 256) * ((N + 31) / 32) * nblk < (1u << 31);
}

// equal tiles in steps of 16 tokens (the MMA's N over a CTA pair, eight-row swizzle groups)
static uint32_t equal_tiles(uint32_t N, uint32_t cols) { return ((N + cols - 1) / cols + 15) & ~15u; }

// Tokens of a tile, at most 256. Wide tiles unpack the weights fewer times, narrow ones waste fewer columns and leave no pairs
// idle; which of them wins depends on the shape, so every width's cost is estimated. 110 shapes (types, 96 to 2048 tokens, K to
// 11 Ki): the widths it picks take 1 % more than the best of each shape in the mean, the widest ones 5 %.
// 4096 x 4096, 512 tokens: 256 40.7 us, 176 42.7; 892 x 3072, 287 tokens: 96 17.2, 144 18.5.
static uint64_t width_cost(const ExactGemm& p, uint32_t w, uint32_t n_row_pairs, uint32_t nblk) {
    const uint32_t tiles = n_row_pairs * ((p.N + w - 1) / w), pairs = p.sms > 1 ? p.sms / 2 : 1;
    const XCost c = x_cost(p, p.type == T_Q6_K || p.type == T_Q8_0, w);
    const XDeal d = x_deal(tiles, w, nblk, pairs, c);
    const uint64_t blocks = ((uint64_t)tiles * nblk + d.pairs - 1) / d.pairs;
    uint64_t cost = blocks * c.block + c.epilogue;
    if (d.groups) cost += c.epilogue;
    else if (tiles >= pairs) cost += c.epilogue * tiles / pairs;
    if (tiles * nblk % d.pairs != 0 || d.groups || d.per == 2) cost += c.zero;
    return cost;
}
static uint32_t tile_width(const ExactGemm& p, uint32_t n_row_pairs, uint32_t nblk) {
    const uint32_t least = (p.N + 255) / 256;
    uint32_t best = 0;
    uint64_t best_cost = ~0ull;
    for (uint32_t cols = least; cols <= 2 * least + 4; ++cols) {
        const uint32_t w = equal_tiles(p.N, cols);
        if (best && w < 48) break;
        const uint64_t cost = width_cost(p, w, n_row_pairs, nblk);
        if (cost < best_cost) {
            best_cost = cost;
            best = w;
        }
    }
    return best;
}

cudaError_t launch_mul_mm_exact(const ExactGemm& whole, uint8_t* scratch, cudaStream_t s, uint64_t* launches) {
    const uint32_t nblk = (whole.K + 255) >> 8;
    const bool min_type = whole.type == T_Q4_K || whole.type == T_Q5_K;
    const size_t per_token = (size_t)nblk * 512 * (whole.bf16 ? 1 : 2) + (min_type ? (size_t)nblk * 128 : 0) + sizeof(float);
    const uint32_t most = (uint32_t)((kExactTermBytes - 4096) / per_token) & ~31u;
    for (uint32_t t0 = 0; t0 < whole.N; t0 += most) {
        ExactGemm p = whole;
        p.N = whole.N - t0 < most ? whole.N - t0 : most;
        p.B = static_cast<const uint8_t*>(whole.B) + (uint64_t)t0 * whole.stride_b * (whole.bf16 ? 2 : 4);
        p.D = whole.D + (uint64_t)t0 * whole.stride_d;
        XPlan plan{};
        plan.nblk = nblk;
        plan.n_row_pairs = (p.M + 255) / 256;
        // fine: the widest tiles there are (128 tokens, types of two fp16 terms 64)
        const uint32_t widest = p.type == T_Q6_K || p.type == T_Q8_0 ? 64 : 128;
        plan.n_tile = p.fine ? equal_tiles(p.N, (p.N + widest - 1) / widest) : tile_width(p, plan.n_row_pairs, nblk);
        plan.n_tiles = plan.n_row_pairs * ((p.N + plan.n_tile - 1) / plan.n_tile);
        uint8_t* q = scratch;
        plan.x = q;
        q += (size_t)p.N * nblk * 512 * (p.bf16 ? 1 : 2);
        plan.sums = q;
        if (min_type) q += (size_t)p.N * nblk * 128;
        plan.inv_scale = reinterpret_cast<float*>(q);
        plan.parts = reinterpret_cast<float*>(scratch + kExactTermBytes);
        plan.launches = launches;
        PrepArgs a{};
        a.X = p.B;
        a.x = static_cast<__half*>(plan.x);
        a.sums = static_cast<__half*>(plan.sums);
        a.inv_scale = plan.inv_scale;
        a.D = p.D;
        a.tokens = p.N;
        a.K = p.K;
        a.nblk = nblk;
        a.M = p.M;
        a.stride_b = p.stride_b;
        a.stride_d = p.stride_d;
        a.sms = p.sms;
        a.sums_on = min_type;
        a.vec = ((p.stride_b | p.K) & 3u) == 0 && (reinterpret_cast<uintptr_t>(p.B) & (p.bf16 ? 7u : 15u)) == 0;
        const int order = min_type ? 0 : p.type == T_MXFP4 ? 2 : 1;
        const ExactPrep prep{p.bf16 ? (order == 0 ? launch_prep<0, true> : order == 1 ? launch_prep<1, true> : launch_prep<2, true>)
                                    : (order == 0 ? launch_prep<0, false> : order == 1 ? launch_prep<1, false> : launch_prep<2, false>),
                             &a};
        if (cudaError_t e = launch_type(p, plan, prep, s); e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace zc
