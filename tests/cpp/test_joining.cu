// What zc_end_record does with calls where a step of joining them is refused: the calls that it concerns stay launches.
// The entry points are compiled in with the refusals; the kernels of single calls come from the library.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../zinc_b200/csrc/program.cu"

enum Refuse { NOTHING, MEMORY, ATTRIBUTE };
static Refuse refuse = NOTHING;
static const void* indescribable = nullptr;  // a matrix whose description is made one that no tensor map takes
static bool hooked_program_op(uint32_t type, int mode, const zc::DmmvArgs& a, zc::ProgramOp& op) {
    if (!zc::program_op(type, mode, a, op)) return false;
    if (op.A[0] == indescribable) op.A[0] += 2;
    return true;
}
static bool armed = false;  // between zc_begin_record and the end of zc_end_record
#define program_op hooked_program_op
#define cudaMalloc(...) (armed && refuse == MEMORY ? cudaErrorMemoryAllocation : (cudaMalloc)(__VA_ARGS__))
#define cudaGraphKernelNodeSetAttribute(...) (refuse == ATTRIBUTE ? cudaErrorNotSupported : (cudaGraphKernelNodeSetAttribute)(__VA_ARGS__))
#include "../../zinc_b200/csrc/api.cu"
#undef cudaMalloc

#define EXPECT(c, ...)                 \
    do {                               \
        if (!(c)) {                    \
            printf("line %d: ", __LINE__); \
            printf(__VA_ARGS__);       \
            printf("\n");              \
            exit(1);                   \
        }                              \
    } while (0)
#define OK(call)                                                                          \
    do {                                                                                  \
        const int32_t rc_ = (call);                                                       \
        EXPECT(rc_ == ZC_OK, "%s: %s, %s", #call, zc_status_string(rc_), zc_last_error(ctx)); \
    } while (0)

int main() {
    constexpr uint32_t M = 12288, K = 4096, N = 5;  // two of these are worth being joined
    constexpr uint64_t kBytes = (uint64_t)M * (K / 256) * 210;
    zc_ctx* ctx = nullptr;
    EXPECT(zc_init(0, &ctx) == ZC_OK, "no context");
    std::vector<uint8_t> w(kBytes);
    std::vector<float> x(K), out(M);
    for (uint64_t i = 0; i < kBytes; ++i) w[i] = i % 210 == 209 ? 0x18 : (uint8_t)(i * 2654435761u >> 20);
    for (uint32_t i = 0; i < K; ++i) x[i] = (float)(i * 37 % 101) / 50.f - 1.f;
    void *W[N], *dx, *y;
    OK(zc_alloc(ctx, K * 4, &dx));
    OK(zc_alloc(ctx, (uint64_t)N * M * 4, &y));
    OK(zc_upload(ctx, dx, 0, x.data(), K * 4));
    OK(zc_submit_and_wait(ctx));
    for (uint32_t i = 0; i < N; ++i) {
        w[4 + i] ^= 0x55;
        OK(zc_alloc(ctx, kBytes, &W[i]));
        OK(zc_upload(ctx, W[i], 0, w.data(), kBytes));
        OK(zc_submit_and_wait(ctx));
    }
    auto calls = [&](uint32_t first, uint32_t n) {
        for (uint32_t i = first; i < first + n; ++i)
            OK(zc_dmmv(ctx, zc::T_Q6_K, W[i], kBytes, dx, K * 4, y, (uint64_t)N * M * 4, M, K, 0, 0, (uint64_t)i * M * 4, 0));
    };
    auto all_of = [&] {
        std::vector<float> v(N * M);
        OK(zc_download(ctx, v.data(), y, 0, (uint64_t)N * M * 4));
        OK(zc_submit_and_wait(ctx));
        OK(zc_memset(ctx, y, 0, 0, (uint64_t)N * M * 4));
        return v;
    };
    calls(0, N);
    const std::vector<float> want = all_of();
    auto recorded = [&](const char* what, Refuse r, int no_map, uint64_t launches) {
        refuse = r;
        indescribable = no_map < 0 ? nullptr : W[no_map];
        const uint64_t n0 = zc_launch_count(ctx);
        void* rec = nullptr;
        OK(zc_begin_record(ctx));
        armed = true;
        calls(0, N);
        OK(zc_end_record(ctx, &rec));
        armed = false;
        EXPECT(zc_launch_count(ctx) - n0 == launches, "%s: %d launches", what, (int)(zc_launch_count(ctx) - n0));
        for (int k = 0; k < 2; ++k) {
            OK(zc_replay(ctx, rec));
            const std::vector<float> got = all_of();
            double diff = 0, sum = 0;
            for (uint32_t i = 0; i < N * M; ++i) {
                diff += ((double)got[i] - want[i]) * ((double)got[i] - want[i]);
                sum += (double)want[i] * want[i];
            }
            EXPECT(sum > 0 && diff <= 1.5e-6 * 1.5e-6 * sum, "%s: %g of %g", what, diff, sum);
        }
        OK(zc_free_recording(ctx, rec));
    };
    recorded("nothing refused", NOTHING, -1, 1);
    recorded("no map for call 0", NOTHING, 0, 2);
    recorded("no map for call 1", NOTHING, 1, 3);   // 0 has no neighbour left
    recorded("no map for call 2", NOTHING, 2, 3);   // 0 and 1, 2, 3 and 4
    recorded("no map for call 4", NOTHING, 4, 2);
    recorded("no memory", MEMORY, -1, N);
    recorded("no attribute", ATTRIBUTE, -1, N);
    recorded("nothing refused", NOTHING, -1, 1);
    EXPECT(zc_destroy(ctx) == ZC_OK, "zc_destroy");
    printf("ok\n");
    return 0;
}
