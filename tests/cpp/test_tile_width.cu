// The tile width that the f32-accurate GEMM picks is the one its estimate is least for, on the SMs that the device has. On the host.
#include <cstdio>
#include <cstdlib>

#include "../../zinc_b200/csrc/gemm_exact.cu"

using namespace zc;

int main() {
    int differ = 0;
    for (uint32_t type : {T_Q4_K, T_Q5_K, T_Q6_K, T_Q8_0, T_MXFP4})
        for (uint32_t M : {256u, 892u, 4096u, 12288u})
            for (uint32_t N : {17u, 96u, 287u, 512u, 658u, 2048u}) {
                uint32_t widths[3], i = 0;
                for (uint32_t sms : {148u, 132u, 16u}) {
                    ExactGemm p{};
                    p.type = type;
                    p.M = M;
                    p.N = N;
                    p.K = 4096;
                    p.sms = sms;
                    const uint32_t pairs = (M + 255) / 256, nblk = 16, w = tile_width(p, pairs, nblk), least = (N + 255) / 256;
                    uint64_t best = ~0ull;
                    for (uint32_t cols = least; cols <= 2 * least + 4; ++cols) {
                        const uint32_t v = equal_tiles(N, cols);
                        if (cols == least || v >= 48) best = std::min(best, width_cost(p, v, pairs, nblk));
                    }
                    if (w == 0 || w > 256 || w % 16 || width_cost(p, w, pairs, nblk) != best) {
                        printf("type %u, %u rows, %u tokens, %u SMs: width %u\n", type, M, N, sms, w);
                        return 1;
                    }
                    widths[i++] = w;
                }
                differ += widths[0] != widths[2];
            }
    if (differ == 0) {
        printf("the SMs make no difference\n");
        return 1;
    }
    printf("ok %d\n", differ);
    return 0;
}
