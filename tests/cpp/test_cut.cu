// The GEMM that is cut along K, in every form that it has (CTAs a tile, clusters, tokens of a tile), whatever the rule would choose: the
// same bits every time, and the values of the uncut form; then with waits that run out: it reports, leaves by itself, writes nothing
// past D, and the next launch is sound. The kernel is compiled in, so that form and limit can be set.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

__device__ unsigned wait_limit = 1u << 22;
#define ZC_WAIT_LIMIT wait_limit

#include "../../zinc_b200/csrc/gemm_cut.cu"

using namespace zc;

#define CHECK(e)                                                         \
    do {                                                                 \
        const cudaError_t err_ = (e);                                    \
        if (err_ != cudaSuccess) {                                       \
            printf("line %d: %s\n", __LINE__, cudaGetErrorString(err_)); \
            exit(1);                                                     \
        }                                                                \
    } while (0)
#define EXPECT(c, ...)                      \
    do {                                    \
        if (!(c)) {                         \
            printf("line %d: ", __LINE__);  \
            printf(__VA_ARGS__);            \
            printf("\n");                   \
            exit(1);                        \
        }                                   \
    } while (0)

__global__ void fill(uint8_t* w, uint64_t n, uint32_t block, uint32_t scale) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t h = (uint32_t)i * 2654435761u + 12345u;
        h = (h ^ (h >> 15)) * 0x85EBCA6Bu;
        const uint32_t at = i % block;  // the high bytes of the f16 scales: 1e-3 .. 8e-3
        w[i] = at == scale + 1 || (block == 144 && at == 3) ? 0x14 + (h >> 30) : (uint8_t)(h >> 16);
    }
}
__global__ void fill_bf16(__nv_bfloat16* x, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[i] = __float2bfloat16((float)((i * 2654435761u) >> 16 & 1023u) / 512.f - 1.f);
}
__global__ void fill_f32(float* d, uint32_t n, float v) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) d[i] = v;
}

template <int TYPE>
void run(uint32_t M, uint32_t N, uint32_t K) {
    constexpr uint32_t block = TYPE == T_Q4_K ? 144 : 210;
    const uint64_t w_bytes = (uint64_t)M * (K / 256) * block;
    const uint32_t stride_d = M + 5, n_d = (N + 1) * stride_d;
    uint8_t* w;
    __nv_bfloat16* x;
    float* d;
    uint32_t* status;
    CHECK(cudaMalloc(&w, w_bytes));
    CHECK(cudaMalloc(&x, (uint64_t)N * K * 2));
    CHECK(cudaMalloc(&d, n_d * 4ull));
    CHECK(cudaMalloc(&status, 8));
    fill<<<512, 256>>>(w, w_bytes, block, TYPE == T_Q4_K ? 0 : 208);
    fill_bf16<<<512, 256>>>(x, N * K);
    cudaStream_t s;
    CHECK(cudaDeviceSynchronize());
    CHECK(cudaStreamCreate(&s));
    std::vector<float> now(n_d), first, whole;
    uint32_t st[2];
    auto launch = [&](const Cut& cut) {
        CHECK(cudaMemsetAsync(status, 0, 8, s));
        fill_f32<<<64, 256, 0, s>>>(d, n_d, 7.f);
        const cudaError_t e = launch_typed<TYPE>(w, x, d, M, N, K, K, stride_d, cut, status, s, nullptr);
        if (e == cudaErrorNotSupported) return false;  // two stages of so many tokens do not fit
        CHECK(e);
        CHECK(cudaMemcpyAsync(now.data(), d, n_d * 4ull, cudaMemcpyDeviceToHost, s));
        CHECK(cudaMemcpyAsync(st, status, 8, cudaMemcpyDeviceToHost, s));
        CHECK(cudaStreamSynchronize(s));
        for (uint32_t n = 0; n <= N; ++n)
            for (uint32_t m = n < N ? M : 0; m < stride_d; ++m) EXPECT(now[n * stride_d + m] == 7.f, "written past D, token %u row %u", n, m);
        return true;
    };
    int forms = 0, gave_up = 0;
    const int* held = most_clusters();
    for (uint32_t tiles : {1u, 2u, 3u, 7u}) {
        const uint32_t tn = ((N + tiles - 1) / tiles + 15u) & ~15u;
        if (tn > kCutMaxTokens) continue;
        for (uint32_t parts : {1u, 2u, 4u, 6u, 8u, 10u, 12u, 14u, 16u}) {
            const Cut cut{tn, parts, parts <= 2 ? 1 : parts / 2};
            if (parts > K / 256 || held[cut.cluster] < 1) continue;
            if (!launch(cut)) continue;
            first = now;
            ++forms;
            for (int i = 0; i < 4; ++i) {
                launch(cut);
                EXPECT(st[0] == 0, "tokens %u parts %u: wait %u gave up", tn, parts, st[1]);
                EXPECT(now == first, "tokens %u parts %u: not the same bits", tn, parts);
            }
            if (parts == 1 && whole.empty()) whole = first;
            // an accumulator loses up to 2^-23 of itself at each of its K / 16 instructions, however they are shared out
            double off = 0, all = 0;
            for (uint32_t n = 0; n < N; ++n)
                for (uint32_t m = 0; m < M; ++m) {
                    const double a = first[n * stride_d + m], b = whole[n * stride_d + m];
                    off += (a - b) * (a - b);
                    all += b * b;
                }
            EXPECT(all > 0 && std::sqrt(off / all) <= K / 16 * 1.2e-7, "tokens %u parts %u: %g off the uncut form", tn, parts, std::sqrt(off / all));
            for (unsigned limit : {0u, 1u, 3u, 20u}) {
                CHECK(cudaMemcpyToSymbol(wait_limit, &limit, sizeof limit));
                launch(cut);
                gave_up += st[0] == 1;
                EXPECT(st[0] == 1 || now == first, "limit %u: nothing gave up, and other bits", limit);
                limit = 1u << 22;
                CHECK(cudaMemcpyToSymbol(wait_limit, &limit, sizeof limit));
                launch(cut);
                EXPECT(st[0] == 0 && now == first, "tokens %u parts %u: not the same bits after a wait gave up", tn, parts);
            }
        }
    }
    EXPECT(forms >= (K >= 4096 ? 18 : 2) && gave_up >= forms, "%d forms, %d launches gave up", forms, gave_up);
    CHECK(cudaStreamDestroy(s));
    for (void* p : {(void*)w, (void*)x, (void*)d, (void*)status}) CHECK(cudaFree(p));
}

int main() {
    run<T_Q4_K>(263, 209, 4096);
    run<T_Q6_K>(263, 209, 4352);
    run<T_Q4_K>(129, 17, 512);
    run<T_Q6_K>(127, 33, 768);
    printf("ok\n");
    return 0;
}
