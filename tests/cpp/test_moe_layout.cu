// How recorded MoE layers are laid out: every tile belongs to one CTA, every CTA has gate and up rows, the reciprocals are exact over
// their ranges and shared memory suffices. On the host.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../zinc_b200/csrc/moe_program.cu"

using namespace zc;

#define EXPECT(c, what)                                                                                                \
    do {                                                                                                               \
        if (!(c)) {                                                                                                    \
            printf("%s: mx %u H %u E %u k %u F %u, %d SMs\n", what, s.mx, s.H, s.E, s.k, s.F, sms);                     \
            exit(1);                                                                                                   \
        }                                                                                                              \
    } while (0)

static int laid_out = 0;
static MoeProgram p;

static void check(uint32_t mx, uint32_t H, uint32_t E, uint32_t k, uint32_t F, int sms, bool must) {
    MoeShape s = {};
    s.mx = mx;
    s.E = E;
    s.k = k;
    s.shared = !mx;
    s.slots = k + s.shared;
    s.H = H;
    s.F = F;
    if (!lay_out(s, sms, p)) {
        EXPECT(!must, "refused");
        return;
    }
    ++laid_out;
    EXPECT(p.smem <= 232448 && p.ring * p.place_bytes <= p.at_x && p.ring >= 8 && p.ring <= kMaxRing, "shared memory");
    EXPECT(p.grid % 2 == 0 && (int)p.grid <= sms && p.grid * p.router_rows >= E, "grid");
    std::vector<int> seen(p.gu_tiles);
    uint32_t most = 0, units_g = 0, units_d = 0;
    for (uint32_t c = 0; c < p.grid; ++c) {  // as Stage has it
        const uint32_t rest = p.gu_tiles - p.gu_even * p.grid;
        uint32_t n = p.gu_even;
        if (c < p.gu_takers && c < rest) n += (rest - c + p.gu_takers - 1) / p.gu_takers;
        EXPECT(n > 0, "a CTA without gate and up rows");
        for (uint32_t q = 0; q < n; ++q) {
            const uint32_t t = q < p.gu_even ? c + q * p.grid : p.gu_even * p.grid + c + (q - p.gu_even) * p.gu_takers;
            EXPECT(t < p.gu_tiles && !seen[t]++, "a tile of two CTAs");
        }
        const uint32_t d = p.grid - 1 - c < p.d_tiles ? (p.d_tiles - (p.grid - 1 - c) + p.grid - 1) / p.grid : 0;
        most = std::max(most, n);
        units_g = std::max(units_g, n * p.gu_units);
        units_d = std::max(units_d, d * p.d_units);
    }
    for (int v : seen) EXPECT(v == 1, "a tile of nobody");
    EXPECT(p.at_parts_d - p.at_parts_g >= units_g * 64 && p.at_sync - p.at_parts_d >= units_d * 64, "room for the parts");
    EXPECT(most * 16 <= kComputeThreads && (p.d_tiles + p.grid - 1) / p.grid * 64 <= kComputeThreads, "a thread a row");
    const uint32_t table = mx ? UnitOf<UNIT_MX>::table(F, s.slots) : UnitOf<UNIT_Q6K>::table(F, s.slots);
    EXPECT((p.act_step == 0 || p.act_step >= table) && p.at_zeros - p.at_act >= table + p.act_step, "room for the activations' tables");
    auto over_is_exact = [&](uint32_t limit, uint32_t d, uint32_t mul) {
        for (uint32_t n = 0; n < limit; ++n)
            if ((mul ? (uint32_t)(((uint64_t)n * mul) >> 32) : n) != n / d) return false;
        return true;
    };
    EXPECT(over_is_exact(kMoeMaxLayers * (units_g + units_d), p.ring, p.ring_mul), "ring");
    EXPECT(over_is_exact(units_g, p.gu_units, p.gu_units_mul) && over_is_exact(units_d, p.d_units, p.d_units_mul), "units");
    EXPECT(over_is_exact(p.gu_tiles, p.gu_tiles_slot, p.gu_tiles_slot_mul) && over_is_exact(units_d, p.d_units_slot, p.d_units_slot_mul), "slots");
    const uint32_t blocks = mx ? 2 * UnitOf<UNIT_MX>::units(F) : F / 256;
    EXPECT(over_is_exact(blocks * s.slots, blocks, p.blocks_slot_mul), "blocks");
}

int main() {
    for (int sms : {148, 132, 131, 16}) {
        const bool must = sms == 148;
        for (uint32_t h = 4; h <= 16; h += 3)
            for (uint32_t E : {64, 96, 128, 256})
                for (uint32_t k = 4; k <= 8; ++k)
                    for (uint32_t f = 2; f <= 4; ++f) check(0, 256 * h, E, k, 256 * f, sms, must && (k + 1) * 256 * f <= 12288);
        for (uint32_t h = 16; h <= 45; h += 2)
            for (uint32_t E : {16, 24, 32})
                for (uint32_t k = 2; k <= 4; ++k)
                    for (uint32_t f = 16; f <= 45; f += 3) check(1, 64 * h, E, k, 64 * f, sms, must);
        check(0, 256, 256, 1, 256, sms, false);
        check(1, 64, 1, 1, 64, sms, false);
        check(1, 6144, 128, 8, 3072, sms, false);
        check(0, 8192, 64, 31, 256, sms, false);
    }
    printf("ok %d\n", laid_out);
    return 0;
}
