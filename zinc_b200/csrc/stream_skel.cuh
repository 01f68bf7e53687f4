// Primitives of the streaming matvec kernels: programmatic dependent launch, asynchronous copies, shared-memory loads,
// tensor-core instructions and the receiving half of the fused exchange.
#pragma once

#include "common.cuh"
#include "stream_common.cuh"

namespace zc {
namespace {

// Programmatic dependent launch: let the next kernel of the stream start its prologue while this
// one runs, and wait for the previous kernel's results before touching anything it may have
// written. Both are no-ops for kernels launched without the attribute.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Start of a streaming kernel: release the next kernel of the stream at once, unless this launch was told that
// its predecessor did the same while the routing buffer was still being written. Then the dependency wait comes
// first, so that whatever starts behind this kernel finds every older kernel complete.
// In two steps, as there is set-up work that touches nothing another kernel writes: pdl_begin at the start, pdl_late
// before the first read of the routing buffer (or of anything else a predecessor writes).
__device__ __forceinline__ void pdl_begin(uint32_t late) {
    if (!late) pdl_launch_dependents();
}
__device__ __forceinline__ void pdl_late(uint32_t late) {
    if (late) {
        pdl_wait();
        pdl_launch_dependents();
    }
}

// The activation a fused gate + up launch applies (src/shaders/swiglu.comp:25-33, swiglu_oai.comp:24-34).
__device__ __forceinline__ float gate_up_act(uint32_t act, float gate, float up) {
    if (act == 2) {
        const float g = fminf(gate, 7.0f);
        const float u = fmaxf(-7.0f, fminf(up, 7.0f));
        return (g / (1.0f + expf(1.702f * (-g)))) * (u + 1.0f);
    }
    return (gate / (1.0f + expf(-gate))) * up;
}

// Loads through the shared window (32-bit addresses from smem_u32): the pointers of the carved shared
// memory go through integer arithmetic, after which the compiler can no longer prove the address space
// and would fall back to generic loads.
__device__ __forceinline__ uint4 lds_v4(uint32_t saddr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr));
    return v;
}
__device__ __forceinline__ float2 lds_f2(uint32_t saddr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(saddr));
    return v;
}
__device__ __forceinline__ float lds_f1(uint32_t saddr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(saddr));
    return v;
}

// Stores to the cluster's shared window
__device__ __forceinline__ void st_cluster(uint32_t a, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void st_cluster(uint32_t a, const uint4& v) {
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void st_cluster_u8(uint32_t a, int v) { asm volatile("st.shared::cluster.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// D(16x8,f32) += A(16x16,f16,row) * B(16x8,f16,col)
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// D(16x8,s32) += A(16x32,u8,row) * B(32x8,s8,col)
__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint2 ld_volatile_u2(const uint2* p) {
    uint2 v;
    asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}

// n / d by the high word of a product, where 2^32 / d + 1 is exact for every n < limit; 0: it is not (quotient divides).
inline uint32_t reciprocal(uint32_t d, uint64_t limit) { return d > 1 && limit * d < (1ull << 32) ? (uint32_t)((1ull << 32) / d) + 1 : 0; }
__host__ __device__ __forceinline__ uint32_t quotient(uint32_t n, uint32_t d, uint32_t mul) {
    return mul ? (uint32_t)(((uint64_t)n * mul) >> 32) : n / d;
}

// The consumer half of the fused exchange, spread over the grid: element i belongs to thread i / n_ctas of CTA
// i % n_ctas. Waits (bounded) for the tagged value of every rank, adds them in rank order and clears the tags.
__device__ __forceinline__ void consume_pushed(const ConsumeArgs& c, uint32_t cta, uint32_t n_ctas, uint32_t tid,
                                               uint32_t n_threads) {
    for (uint32_t i = tid * n_ctas + cta; i < c.n; i += n_threads * n_ctas) {
        float s = c.acc ? c.dst[i] : 0.f;
        for (uint32_t r = 0; r < c.world; ++r) {
            uint2* p = c.slots + (size_t)r * kPushMaxFloats + i;
            uint2 q = ld_volatile_u2(p);
            uint32_t spins = 0;
            while (q.y == 0u) {
                if (++spins > c.spin_limit) {
                    c.status[0] = 1;
                    c.status[1] = 400u + r;
                    break;
                }
                q = ld_volatile_u2(p);
            }
            s += __uint_as_float(q.x);
            *p = make_uint2(0u, 0u);
        }
        c.dst[i] = s;
    }
}

enum { EPI_PLAIN = 0, EPI_GATE_UP = 1, EPI_SIGMOID_ACC = 2, EPI_PAIR = 3, EPI_ACC = 4 };

}  // namespace
}  // namespace zc
