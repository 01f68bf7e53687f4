// reciprocal and quotient of csrc/dmmv_slice.cuh, and the limits that slice_plan takes reciprocals for.
#include <cstdio>
#include <cstdlib>

#include "../../zinc_b200/csrc/dmmv_slice.cuh"

using namespace zc;

constexpr uint64_t kAll = (uint64_t)1 << 32;

static void same(uint32_t n, uint32_t d, uint32_t mul, const char* what) {
    if (quotient(n, d, mul) == n / d) return;
    printf("%s: %u / %u by %u is %u\n", what, n, d, mul, quotient(n, d, mul));
    exit(1);
}
// all n of a short range; of a long one its ends, a sample, and both sides of multiples of d
static void check(uint32_t d, uint64_t limit, const char* what) {
    const uint32_t mul = reciprocal(d, limit);
    if (!mul && d > 1 && limit * d < kAll) {
        printf("%s: no reciprocal of %u below %llu\n", what, d, (unsigned long long)limit);
        exit(1);
    }
    const uint64_t step = limit / 20000 + 1;
    for (uint64_t n = 0; n < limit; n += step) {
        const uint64_t m = n / d * d;
        same((uint32_t)n, d, mul, what);
        if (m) same((uint32_t)(m - 1), d, mul, what);
        same((uint32_t)m, d, mul, what);
        if (m + d - 1 < limit) same((uint32_t)(m + d - 1), d, mul, what);
    }
    same((uint32_t)(limit - 1), d, mul, what);
}
template <uint32_t kMostWarps, uint32_t kColumns, uint32_t kTable>
struct Fmt {  // what slice_plan asks of a format
    static constexpr uint32_t kSlot = 2048, kMost = kMostWarps, kCols = kColumns, kDeepWarps = 32;
    static uint32_t table_bytes(uint32_t nblk) { return nblk * kTable + 128; }
};
template <typename F>
static int plans() {
    int n = 0;
    for (uint32_t M : {1u, 3u, 16u, 100u, 512u, 2048u, 2880u, 7001u, 16384u, 400000u})
        for (uint32_t K : {512u, 768u, 1024u, 2048u, 2880u, 4096u})
            for (uint32_t slots : {1u, 2u, 3u, 5u, 8u, 9u, 33u})
                for (int seg : {2, 3}) {
                    SliceArgs a = {};
                    a.M = M;
                    a.K = K;
                    a.nseg = slots;
                    uint32_t warps, grid, smem;
                    if (!slice_plan<F>(a, 1, seg, 148, warps, grid, smem)) continue;
                    ++n;
                    if (a.tpe != (M + a.h - 1) / a.h || a.bpe != (K + F::kCols - 1) / F::kCols) exit(2);
                    for (uint32_t T = 0; T < a.tiles; ++T) same(T, a.tpe, a.tpe_mul, "tile");
                    for (uint32_t b = 0; b < a.nblk; ++b) same(b, a.bpe, a.bpe_mul, "block");
                    if (a.tpe_mul != reciprocal(a.tpe, a.tiles) || a.bpe_mul != reciprocal(a.bpe, a.nblk)) exit(3);
                }
    return n;
}
int main() {
    for (uint32_t d : {1u, 2u, 3u, 5u, 6u, 32u, 147u, 180u, 205u, 4095u, 4096u, 16384u, 65535u, 0x80000001u})
        for (uint64_t limit : {(uint64_t)1, (uint64_t)d, (uint64_t)9 * d, (uint64_t)32 * d, (uint64_t)65536, kAll / d,
                               (kAll - 1) / d, kAll / d + 1, kAll})
            if (limit <= kAll) check(d, limit, "quotient");
    if (reciprocal(1, 10) || reciprocal(3, kAll / 2)) exit(4);
    const int n = plans<Fmt<16, 256, 868>>() + plans<Fmt<16, 512, 1608>>() + plans<Fmt<18, 512, 2056>>();
    if (n < 300) exit(5);
    printf("ok %d plans\n", n);
    return 0;
}
