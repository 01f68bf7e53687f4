// The kernel of recorded MoE layers when its waits run out: it reports, leaves by itself, writes nothing past its buffers and leaves its
// counters clean; the next launch is sound. And when one CTA falls some 40 us behind ahead of its down products, layer after layer: the
// same bits (the other CTA of its pair, which writes half of its table of activations, is a layer ahead by then). The kernel is compiled
// in, so that its limit can be set and a CTA be held up.
#include <cstdio>
#include <cstdlib>
#include <vector>

__device__ int late_cta = -1;
#define ZC_MOE_BEFORE_DOWN(layer)    \
    if ((int)blockIdx.x == late_cta) \
        for (int i_ = 0; i_ < 20; ++i_) __nanosleep(2000)

#include "../../zinc_b200/csrc/moe_program.cu"

using namespace zc;

#define CHECK(e)                                                                                      \
    do {                                                                                              \
        const cudaError_t err_ = (e);                                                                 \
        if (err_ != cudaSuccess) {                                                                    \
            printf("line %d: %s\n", __LINE__, cudaGetErrorString(err_));                              \
            exit(1);                                                                                  \
        }                                                                                             \
    } while (0)
#define EXPECT(c, ...)                                \
    do {                                              \
        if (!(c)) {                                   \
            printf("line %d: ", __LINE__);            \
            printf(__VA_ARGS__);                      \
            printf("\n");                             \
            exit(1);                                  \
        }                                             \
    } while (0)

__global__ void fill(uint8_t* w, uint64_t n, uint32_t seed, uint32_t block, uint32_t scale) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t h = (uint32_t)i * 2654435761u + seed;
        h = (h ^ (h >> 15)) * 0x85EBCA6Bu;
        // the high byte of an f16 scale 1e-3 .. 8e-3 (Q4_K d and dmin at 0, Q6_K d at 208), an E8M0 exponent of 2^-9 .. 2^-6 (MXFP4)
        const uint32_t at = i % block;
        w[i] = block == 17 ? (at == 0 ? 118 + (h >> 30) : (uint8_t)(h >> 16))
                           : at == scale + 1 || (block == 144 && at == 3) ? 0x14 + (h >> 30) : (uint8_t)(h >> 16);
    }
}
__global__ void fill_f32(float* x, uint32_t n, float scale) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[i] = ((float)((i * 2654435761u) >> 16 & 1023u) / 512.f - 1.f) * scale;
}

static void run(bool mx, int sms, uint32_t H, uint32_t F, uint32_t E, bool one_table) {
    constexpr uint32_t k = 4, L = 3;
    const uint32_t shared = mx ? 0 : 1, slots = k + shared, gb = mx ? 17 : 144, db = mx ? 17 : 210, ge = mx ? 32 : 256;
    const uint64_t gs = (uint64_t)F * (H / ge) * gb, ds = (uint64_t)H * (F / ge) * db;
    uint8_t *wg, *wu, *wd, *sg, *su, *sd;
    uint8_t** stacks[] = {&wg, &wu, &wd, &sg, &su, &sd};
    for (int i = 0; i < 6; ++i) {
        const uint64_t n = (i % 3 == 2 ? ds : gs) * (i < 3 ? E : 1);
        CHECK(cudaMalloc(stacks[i], n));
        fill<<<512, 256>>>(*stacks[i], n, 77u * i, i % 3 == 2 ? db : gb, i % 3 == 2 && !mx ? 208 : 0);
    }
    float *x, *router, *out;  // out: logits, activations, hidden, routing
    const uint32_t n_out = E + slots * F + H + 2 * slots;
    CHECK(cudaMalloc(&x, H * 4));
    CHECK(cudaMalloc(&router, (uint64_t)L * E * H * 4));
    CHECK(cudaMalloc(&out, n_out * 4));
    fill_f32<<<64, 256>>>(x, H, 1.f);
    fill_f32<<<64, 256>>>(router, L * E * H, 0.1f);
    uint32_t* status;
    CHECK(cudaMalloc(&status, 8));
    std::vector<MoeCalls> calls(L);
    for (uint32_t l = 0; l < L; ++l) {
        MoeCalls& c = calls[l];
        c.router = {x, nullptr, router + (uint64_t)l * E * H, nullptr, out, reinterpret_cast<uint32_t*>(out + E + slots * F + H), nullptr, E, H, k, mx ? 1u : 0u, shared};
        c.gate_up_type = mx ? T_MXFP4 : T_Q4_K;
        c.down_type = mx ? T_MXFP4 : T_Q6_K;
        DmmvArgs g;
        g.A = wg;
        g.A2 = wu;
        g.x = x;
        g.y = out + E;
        g.act = mx ? 2 : 1;
        g.routing = c.router.routing;
        g.M = F;
        g.K = H;
        g.expert_stride = gs;
        g.n_used = slots;
        g.n_experts_max = E;
        g.status = status;
        if (shared) {
            g.A_sh = sg;
            g.A2_sh = su;
        }
        c.gate_up = g;
        DmmvArgs d;
        d.A = wd;
        d.x = out + E;
        d.y = out + E + slots * F;
        d.routing = c.router.routing;
        d.M = H;
        d.K = F;
        d.expert_stride = ds;
        d.n_used = slots;
        d.x_expert_stride = F;
        d.n_experts_max = E;
        d.status = status;
        if (shared) d.A_sh = sd;
        c.down = d;
    }
    std::vector<MoeProgram> storage(1);
    MoeProgram& p = storage[0];
    EXPECT(moe_plan(calls.data(), L, sms, p) == L, "not one program");
    EXPECT((p.act_step == 0) == one_table, "%u x %u: not the tables that were to be tested", H, F);
    std::vector<CUtensorMap> maps((size_t)L * p.n_maps);
    EXPECT(moe_maps(calls.data(), p, maps.data()), "tensor maps");
    constexpr uint32_t kGuard = 4096;
    const uint64_t map_bytes = maps.size() * sizeof(CUtensorMap), own = moe_exchange_bytes(p), total = map_bytes + kGuard + own + kGuard;
    uint8_t* mem;
    CHECK(cudaMalloc(&mem, total));
    CHECK(cudaMemset(mem, 0xA5, total));
    CHECK(cudaMemcpy(mem, maps.data(), map_bytes, cudaMemcpyHostToDevice));
    uint8_t* words = mem + map_bytes + kGuard;
    CHECK(cudaMemset(words, 0, own));
    p.maps = mem;
    p.words = reinterpret_cast<uint32_t*>(words);
    p.logits_x = reinterpret_cast<uint64_t*>(words + 256);
    p.act_x = p.logits_x + 2 * E;
    p.status = status;
    void* func = nullptr;
    uint32_t threads = 0, st[2], tags = 0;
    CHECK(moe_program_kernel(mx, sms, p, &func, threads));

    std::vector<uint32_t> first(n_out), now(n_out);
    std::vector<uint8_t> back(total);
    auto launch = [&](uint32_t limit, uint32_t x_waits) {
        std::vector<MoeProgram> copy(1, p);
        copy[0].spin_limit = limit;
        for (uint32_t l = 1; l < L; ++l) copy[0].layers[l].x_waits = x_waits;
        CHECK(cudaMemset(status, 0, 8));
        CHECK(cudaMemset(out, 0, n_out * 4));
        void* args[] = {&copy[0]};
        CHECK(cudaLaunchCooperativeKernel(func, dim3(p.grid), dim3(threads), args, p.smem, nullptr));
        CHECK(cudaDeviceSynchronize());
        tags += L;
        CHECK(cudaMemcpy(st, status, 8, cudaMemcpyDeviceToHost));
        CHECK(cudaMemcpy(now.data(), out, n_out * 4, cudaMemcpyDeviceToHost));
        CHECK(cudaMemcpy(back.data(), mem, total, cudaMemcpyDeviceToHost));
        const uint32_t* w = reinterpret_cast<const uint32_t*>(back.data() + map_bytes + kGuard);
        EXPECT(w[0] == tags && w[1] == 0 && w[2] == 0, "words %u %u %u after a launch", w[0], w[1], w[2]);
        for (uint32_t i = 0; i < kGuard; ++i) EXPECT(back[map_bytes + i] == 0xA5 && back[total - kGuard + i] == 0xA5, "guard byte %u", i);
    };
    launch(1u << 24, 0);
    EXPECT(st[0] == 0, "wait %u gave up", st[1]);
    first = now;
    double sum = 0;
    for (uint32_t i = E + slots * F; i < E + slots * F + H; ++i) {
        float v;
        memcpy(&v, &first[i], 4);
        EXPECT(v == v && v - v == 0.f, "hidden %u is not a number", i);
        sum += (double)v * v;
    }
    EXPECT(sum > 0, "hidden is zero");
    for (int cta : {0, 1, 2, 37, 74, 75, (int)p.grid - 2, (int)p.grid - 1, -1}) {
        CHECK(cudaMemcpyToSymbol(late_cta, &cta, sizeof cta));
        for (int round = 0; round < 3; ++round) {
            launch(1u << 24, 0);
            EXPECT(st[0] == 0, "CTA %d late: wait %u gave up", cta, st[1]);
            EXPECT(now == first, "CTA %d late: not the same bits", cta);
        }
    }
    int gave_up = 0;
    for (int round = 0; round < 30; ++round) {
        for (uint32_t limit : {0u, 1u, 3u, 10u}) {
            for (uint32_t x_waits : {0u, 1u}) {
                launch(limit, x_waits);
                gave_up += st[0] == 1;
                EXPECT(st[0] == 1 || now == first, "limit %u: nothing gave up, and other bits", limit);
                launch(1u << 24, x_waits);
                EXPECT(st[0] == 0, "after limit %u: wait %u gave up", limit, st[1]);
                EXPECT(now == first, "after limit %u: not the same bits", limit);
            }
        }
    }
    EXPECT(gave_up >= 30, "%d launches gave up", gave_up);
    for (uint8_t** s : stacks) CHECK(cudaFree(*s));
    for (void* m : {(void*)mem, (void*)x, (void*)router, (void*)out, (void*)status}) CHECK(cudaFree(m));
}

int main() {
    cudaDeviceProp prop;
    CHECK(cudaGetDeviceProperties(&prop, 0));
    for (bool mx : {false, true}) {
        run(mx, prop.multiProcessorCount, 1024, 768, 64, false);
        run(mx, prop.multiProcessorCount, mx ? 2880 : 1024, mx ? 2880 : 2304, 16, true);
    }
    printf("ok\n");
    return 0;
}
