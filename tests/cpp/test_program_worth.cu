// Which runs of recorded calls are worth being joined (program_plan, on the host): against what was measured on both sides.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../zinc_b200/csrc/common.cuh"
#include "../../zinc_b200/csrc/kernels.h"
#include "../../zinc_b200/csrc/program.h"

using namespace zc;

static uint32_t status;
static uintptr_t weights;
enum Mode { BESIDE, CHAIN, ADD, ADD_EVERY_SECOND };

static ProgramOp op(uint32_t type, int mode, uint32_t M, uint32_t K, uintptr_t x, uintptr_t y, uint32_t acc = 0) {
    DmmvArgs a;
    a.A = reinterpret_cast<const uint8_t*>(weights += 1u << 30);
    if (mode == MODE_GATE_UP_SWIGLU) a.A2 = reinterpret_cast<const uint8_t*>(weights += 1u << 30);
    a.a_end = reinterpret_cast<const uint8_t*>(weights + (1u << 30));
    a.x = reinterpret_cast<const float*>(x);
    a.y = reinterpret_cast<float*>(y);
    a.M = M;
    a.K = K;
    a.acc_mode = acc;
    a.status = &status;
    a.sm_count = 148;
    ProgramOp o;
    if (!program_op(type, mode, a, o)) {
        printf("%u x %u is not a call of a program\n", M, K);
        exit(1);
    }
    return o;
}
static uint32_t worth(const std::vector<ProgramOp>& ops) {
    std::vector<Program> p(1);
    float gain;
    return program_plan(ops.data(), (uint32_t)ops.size(), 148, p[0], &gain);
}
static uint32_t run(uint32_t type, uint32_t M, uint32_t K, uint32_t n, Mode mode) {
    std::vector<ProgramOp> ops;
    const uintptr_t x = 1u << 20, y = 1u << 24;
    for (uint32_t j = 0; j < n; ++j) {
        const uintptr_t own = y + j * (1u << 20);
        if (mode == CHAIN) ops.push_back(op(type, MODE_PLAIN, M, K, j ? own - (1u << 20) : x, own));
        else if (mode == ADD || (mode == ADD_EVERY_SECOND && j % 2)) ops.push_back(op(type, MODE_PLAIN, M, K, x, y, 1));
        else ops.push_back(op(type, MODE_PLAIN, M, K, x, own));
    }
    return worth(ops);
}
// a dense model's token; `reads`: every call reads what the one before wrote, else only the additions to one vector are ordered
static std::vector<ProgramOp> token(uint32_t hidden, uint32_t q, uint32_t ffn, uint32_t layers, bool reads) {
    const uintptr_t at = 1u << 24, h = at, qv = at + (1u << 20), act = at + (2u << 20), in1 = at + (3u << 20), in2 = at + (4u << 20), in3 = at + (5u << 20);
    std::vector<ProgramOp> ops;
    for (uint32_t l = 0; l < layers; ++l) {
        ops.push_back(op(T_Q4_K, MODE_PLAIN, q, hidden, reads ? h : in1, qv));
        ops.push_back(op(T_Q4_K, MODE_PLAIN, hidden, q, reads ? qv : in2, h, 1));
        ops.push_back(op(T_Q4_K, MODE_GATE_UP_SWIGLU, ffn, hidden, reads ? h : in1, act));
        ops.push_back(op(T_Q6_K, MODE_PLAIN, hidden, ffn, reads ? act : in3, h, 1));
    }
    return ops;
}
#define EXPECT(what, want)                                        \
    do {                                                          \
        const uint32_t got_ = (what);                             \
        if (got_ != (want)) {                                     \
            printf("%s is %u, not %u\n", #what, got_, (want));    \
            return 1;                                             \
        }                                                         \
    } while (0)

int main() {
    // measured, us joined and as launches
    EXPECT(run(T_Q4_K, 4096, 1024, 2, BESIDE), 0u);            // 10.2  8.1
    EXPECT(run(T_Q4_K, 4096, 1024, 4, BESIDE), 4u);            // 12.9 14.3
    EXPECT(run(T_Q4_K, 4096, 1024, 8, BESIDE), 8u);            // 18.4 26.6
    EXPECT(run(T_Q4_K, 4096, 4096, 2, BESIDE), 0u);            // 13.0 12.0
    EXPECT(run(T_Q4_K, 4096, 4096, 4, BESIDE), 4u);            // 16.7 21.7
    EXPECT(run(T_Q6_K, 12288, 4096, 2, BESIDE), 2u);           // 26.2 29.2
    EXPECT(run(T_Q4_K, 32768, 4096, 2, BESIDE), 0u);           // 36.4 34.4
    EXPECT(run(T_Q4_K, 32768, 4096, 8, BESIDE), 8u);           // 104.8 125.1
    EXPECT(run(T_Q6_K, 32768, 4096, 4, BESIDE), 4u);           // 84.8 99.4
    for (uint32_t n : {2u, 4u, 8u, 64u}) {
        EXPECT(run(T_Q4_K, 4096, 1024, n, CHAIN), 0u);         // 8 calls: 57.6 26.7
        EXPECT(run(T_Q4_K, 4096, 4096, n, CHAIN), 0u);         // 72.7 41.1
        EXPECT(run(T_Q6_K, 4096, 4096, n, CHAIN), 0u);         // 84.0 55.4
        EXPECT(run(T_Q6_K, 12288, 4096, n, CHAIN), 0u);        // 123.5 104.5
        EXPECT(run(T_Q6_K, 32768, 4096, n, CHAIN), 0u);        // 219.0 199.7
        EXPECT(run(T_Q4_K, 4096, 1024, n, ADD), 0u);           // 35.2 26.7
        EXPECT(run(T_Q4_K, 8192, 512, n, ADD), 0u);            // 2 calls: 13.7  7.5
    }
    EXPECT(run(T_Q6_K, 4096, 4096, 8, ADD), 8u);               // 47.3 55.6
    EXPECT(run(T_Q6_K, 12288, 4096, 8, ADD), 8u);              // 84.8 103.4
    EXPECT(run(T_Q4_K, 4096, 4096, 8, ADD_EVERY_SECOND), 8u);  // 31.3 41.0
    EXPECT(run(T_Q4_K, 8192, 512, 8, ADD_EVERY_SECOND), 0u);   // 29.5 23.0
    EXPECT(worth(token(4096, 6144 - 2048, 12288, 36, false)), 144u);  // 900 1557
    EXPECT(worth(token(2560, 2816, 7680, 16, false)), 64u);    // 222 488
    for (uint32_t from : {0u, 1u, 2u, 3u}) {                   // 1894 1527, 668 488
        for (const auto& t : {token(4096, 4096, 12288, 36, true), token(2560, 2816, 7680, 16, true)})
            EXPECT(worth(std::vector<ProgramOp>(t.begin() + from, t.end())), 0u);
    }
    // one call of many that reads a result: its wait is worth the rest
    auto ops = token(4096, 4096, 12288, 36, false);
    ops.push_back(op(T_Q6_K, MODE_PLAIN, 151936, 4096, 1u << 24, 1u << 28));
    EXPECT(worth(ops), 145u);
    // a chain behind calls that are worth it is left out
    ops.clear();
    for (uint32_t j = 0; j < 8; ++j) ops.push_back(op(T_Q4_K, MODE_PLAIN, 4096, 4096, 1u << 20, (1u << 24) + j * (1u << 20)));
    for (uint32_t j = 8; j < 40; ++j) ops.push_back(op(T_Q4_K, MODE_PLAIN, 4096, 4096, (1u << 24) + (j - 1) * (1u << 20), (1u << 24) + j * (1u << 20)));
    EXPECT(worth(ops), 8u);
    printf("ok\n");
    return 0;
}
