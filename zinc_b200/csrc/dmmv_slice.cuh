// Skeleton of the streaming matvec kernels: rows are dealt to CTAs, K to the warps of a CTA.
//
// Every CTA owns a contiguous run of row tiles (at most 16 rows each, the height chosen so that the SMs get equal numbers
// of rows); inside it, warp (wr, wk) works through the tiles wr, wr + n_wr, ... and owns the blocks (512 columns, Q6_K 256) wk, wk + n_wk,
// ... of every one of them. So
//   * x is converted once per CTA, a block or a few per warp, and every row of the CTA uses it;
//   * a row's partial sums meet in shared memory: one barrier per few tiles, no hand-off between CTAs, results
//     that do not depend on timing;
//   * the warps of a CTA read adjacent blocks of the same rows at about the same time: whole DRAM pages.
// (Units dealt to all warps of the GPU in one contiguous range each had every CTA convert all of x and a tile's sums travel
// through L2: Q/K/V 6144 x 4096 Q4_K 7.2 us, down 4096 x 12288 Q6_K 15.8 us.)
//
// A format F supplies: the copies of one unit (16 rows x one block) into a ring slot, the conversion of x, and the
// unit's dot products. Copies are 16-byte cp.async; a warp keeps `depth` units in flight, requested before the dependency
// wait: weights depend on no kernel.
// Bound: HBM for large matrices; a few MB are bound by launch, x and write-back latency.
#pragma once

#include "kernels.h"
#include "stream_skel.cuh"

namespace zc {
namespace {


struct SliceArgs {
    const uint8_t* A[2];
    const uint8_t* a_end[2];   // first byte past the buffers (formats that fetch aligned supersets)
    const float* x;
    float* y;
    float* y2;
    const float* gate;
    uint32_t M, K, acc_mode;
    uint32_t* status;
    // kSeg 1: matrices that share x; kSeg 2: expert slots, one output block each; kSeg 3: expert slots side by side along K
    uint32_t nseg;
    uint32_t seg_end[3];       // last tile + 1 of matrix i
    const uint8_t* segA[3];
    float* segY[3];
    uint32_t segM[3];
    const uint32_t* routing;
    uint64_t expert_stride;
    uint32_t n_experts_max;
    uint32_t x_slot_stride;    // kSeg 3: elements between the slots' activation vectors
    PushArgs push;
    ConsumeArgs consume;
    uint32_t act;
    const uint8_t* A_sh[2];
    const uint8_t* A_sh_end[2];
    const float* bias[2];
    uint32_t late;
    // how the work is cut
    uint32_t h, tiles, tpe, tpc;   // rows per tile, tiles, tiles per expert slot, tiles per CTA
    uint32_t n_wk, n_wr, depth;
    uint32_t round;                // tiles between two meetings of a CTA's warps, a multiple of n_wr
    uint32_t nblk, bpe;            // blocks of a (concatenated) row; of one matrix's row
    uint32_t tpe_mul, bpe_mul;     // reciprocals of tpe and bpe (quotient)
};

inline SliceArgs slice_args(const DmmvArgs& a) {
    SliceArgs s = {};
    s.A[0] = a.A;
    s.A[1] = a.A2 ? a.A2 : a.A;
    s.a_end[0] = a.a_end;
    s.a_end[1] = a.A2 ? a.a2_end : a.a_end;
    s.x = a.x;
    s.y = a.y;
    s.y2 = a.y2;
    s.gate = a.gate;
    s.M = a.M;
    s.K = a.K;
    s.acc_mode = a.acc_mode;
    s.status = a.status;
    s.nseg = 1;
    s.routing = a.routing;
    s.expert_stride = a.expert_stride;
    s.n_experts_max = a.n_experts_max;
    s.x_slot_stride = a.x_expert_stride;
    s.push = a.push;
    s.consume = a.consume;
    s.act = a.act;
    s.A_sh[0] = a.A_sh;
    s.A_sh[1] = a.A2_sh ? a.A2_sh : a.A_sh;
    s.A_sh_end[0] = a.a_sh_end;
    s.A_sh_end[1] = a.A2_sh ? a.a2_sh_end : a.a_sh_end;
    s.bias[0] = a.bias;
    s.bias[1] = a.bias2;
    s.late = a.late ? 1u : 0u;
    return s;
}

// One block of up to 16 rows.
struct Unit {
    const uint8_t* mat;  // the matrix's first byte; nullptr: a slot without an expert on this rank (contributes zeros)
    const uint8_t* end;
    uint32_t row0, rows;  // first row, valid rows of the tile
    uint32_t lb, kb;     // block within the matrix's row, within the concatenated row
};

// The matrices of the expert slots: lane s holds slot s's, found once (a look-up through the routing buffer per unit would
// put a chain of dependent loads in front of every request). More than 32 slots: looked up each time.
template <int NS, int kSeg>
struct Slots {
    const uint8_t* mat[NS];
    __device__ __forceinline__ static const uint8_t* find(const SliceArgs& a, uint32_t slot, int strm) {
        const uint32_t e = __ldg(a.routing + slot);
        return e == kSkipExpert ? nullptr : expert_matrix(a.A[strm], a.A_sh[strm], e, a.expert_stride, a.n_experts_max, a.status);
    }
    __device__ __forceinline__ void init(const SliceArgs& a, int lane) {
        if constexpr (kSeg >= 2) {
#pragma unroll
            for (int i = 0; i < NS; ++i) mat[i] = (uint32_t)lane < a.nseg ? find(a, lane, i) : nullptr;
        }
    }
    __device__ __forceinline__ const uint8_t* get(const SliceArgs& a, uint32_t slot, uint32_t strm) const {
        if (a.nseg > 32) return find(a, slot, (int)strm);
        const uint64_t m = reinterpret_cast<uint64_t>(NS == 2 && strm ? mat[NS - 1] : mat[0]);
        return reinterpret_cast<const uint8_t*>(__shfl_sync(0xFFFFFFFFu, m, slot));
    }
};

template <int NS, int kSeg>
__device__ __forceinline__ Unit find_unit(const SliceArgs& a, const Slots<NS, kSeg>& slots, uint32_t T, uint32_t strm, uint32_t kb) {
    Unit u;
    u.kb = u.lb = kb;
    uint32_t M = a.M;
    if constexpr (kSeg == 1) {
        const uint32_t sg = (T >= a.seg_end[0] ? 1u : 0u) + (T >= a.seg_end[1] ? 1u : 0u);
        const uint32_t t0 = sg == 0 ? 0u : sg == 1 ? a.seg_end[0] : a.seg_end[1];
        u.mat = sg == 0 ? a.segA[0] : sg == 1 ? a.segA[1] : a.segA[2];
        M = sg == 0 ? a.segM[0] : sg == 1 ? a.segM[1] : a.segM[2];
        u.end = nullptr;
        u.row0 = (T - t0) * a.h;
    } else if constexpr (kSeg == 2 || kSeg == 3) {
        const uint32_t slot = kSeg == 2 ? quotient(T, a.tpe, a.tpe_mul) : quotient(kb, a.bpe, a.bpe_mul);
        u.row0 = (kSeg == 2 ? T - slot * a.tpe : T) * a.h;
        if (kSeg == 3) u.lb = kb - slot * a.bpe;
        u.mat = slots.get(a, slot, strm);
        u.end = u.mat && u.mat == a.A_sh[strm] ? a.A_sh_end[strm] : a.a_end[strm];
    } else {
        u.mat = a.A[strm];
        u.end = a.a_end[strm];
        u.row0 = T * a.h;
    }
    u.rows = min(a.h, M - u.row0);
    return u;
}

// The output row a thread finishes, and what its epilogue reads besides the sums: requested ahead of the barrier.
struct OutRow {
    float *y, *y2;
    uint32_t row;
    bool ok;
    float yold, b0, b1;
};

template <int EPI, int kSeg>
__device__ __forceinline__ OutRow out_row(const SliceArgs& a, uint32_t T, uint32_t rr, bool live) {
    OutRow o{nullptr, nullptr, 0u, false, 0.f, 0.f, 0.f};
    if (!live || rr >= a.h) return o;
    uint32_t Mrows = a.M, slot = 0;
    o.y = a.y;
    o.y2 = a.y2;
    if constexpr (kSeg == 1) {
        const uint32_t sg = (T >= a.seg_end[0] ? 1u : 0u) + (T >= a.seg_end[1] ? 1u : 0u);
        o.row = (T - (sg == 0 ? 0u : sg == 1 ? a.seg_end[0] : a.seg_end[1])) * a.h + rr;
        Mrows = sg == 0 ? a.segM[0] : sg == 1 ? a.segM[1] : a.segM[2];
        o.y = sg == 0 ? a.segY[0] : sg == 1 ? a.segY[1] : a.segY[2];
    } else if constexpr (kSeg == 2) {
        slot = quotient(T, a.tpe, a.tpe_mul);
        o.row = (T - slot * a.tpe) * a.h + rr;
        o.y += (size_t)slot * a.M;
        if (o.y2) o.y2 += (size_t)slot * a.M;
    } else {
        o.row = T * a.h + rr;
    }
    o.ok = o.row < Mrows;
    if (!o.ok) return o;
    const bool adds = EPI == EPI_ACC || EPI == EPI_SIGMOID_ACC || (EPI == EPI_PLAIN && a.acc_mode != 0 && a.push.world == 0);
    if (adds) o.yold = o.y[o.row];
    if constexpr (EPI == EPI_SIGMOID_ACC) o.b0 = __ldg(a.gate);
    if constexpr (EPI == EPI_PAIR) {  // the slot's expert's biases (none for a shared or absent expert)
        if (a.bias[0]) {
            const uint32_t e = __ldg(a.routing + slot);
            if (e < a.n_experts_max) {
                o.b0 = __ldg(a.bias[0] + (size_t)e * a.M + o.row);
                if (a.bias[1]) o.b1 = __ldg(a.bias[1] + (size_t)e * a.M + o.row);
            }
        }
    }
    if constexpr (EPI == EPI_ACC) {  // the selected experts' biases, weighted like their products
        if (a.bias[0]) {
#pragma unroll 4
            for (uint32_t s = 0; s < a.nseg; ++s) {
                const uint32_t e = __ldg(a.routing + s);
                if (e < a.n_experts_max)
                    o.b0 = fmaf(__uint_as_float(__ldg(a.routing + a.nseg + s)), __ldg(a.bias[0] + (size_t)e * a.M + o.row), o.b0);
            }
        }
    }
    return o;
}

template <int NS, int EPI>
__device__ __forceinline__ void write_out(const SliceArgs& a, const OutRow& o, const float (&v)[NS]) {
    if (!o.ok) return;
    if constexpr (EPI == EPI_GATE_UP) {
        o.y[o.row] = (v[0] / (1.0f + expf(-v[0]))) * v[NS - 1];
    } else if constexpr (EPI == EPI_ACC) {
        o.y[o.row] = o.yold + (v[0] + o.b0);
    } else if constexpr (EPI == EPI_PAIR) {
        const float vg = v[0] + o.b0, vu = v[NS - 1] + o.b1;
        if (a.act) {
            o.y[o.row] = gate_up_act(a.act, vg, vu);
        } else {
            o.y[o.row] = vg;
            o.y2[o.row] = vu;
        }
    } else if constexpr (EPI == EPI_SIGMOID_ACC) {
        o.y[o.row] = o.yold + (1.0f / (1.0f + expf(-o.b0))) * v[0];
    } else if (a.push.world) {
        const uint2 pv = make_uint2(__float_as_uint(v[0]), 1u);
        for (uint32_t r = 0; r < a.push.world; ++r) a.push.peers[r][o.row] = pv;
    } else {
        o.y[o.row] = a.acc_mode ? o.yold + v[0] : v[0];
    }
}

// F: format; Extra: what its activation loader takes besides the arguments (nothing, or the attention partials).
// One loop requests a unit ahead and works off the oldest one. The request, the dot products and the meeting of the
// warps each stand in the code once: with several copies (unrolled streams, a prologue of its own) the few units of a
// launch ran through 20 KB of cold instructions, and "no instruction" was the largest stall.
template <typename F, int NS, int EPI, int kSeg, typename Extra>
__device__ __forceinline__ void slice_body(const SliceArgs& a, const Extra& extra) {
    extern __shared__ uint8_t smem_raw[];
    pdl_begin(a.late);
    uint8_t* base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    const uint32_t n_warps = blockDim.x >> 5;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t* ring = base + (size_t)warp * a.depth * F::kSlot;
    float* spart = reinterpret_cast<float*>(base + (size_t)n_warps * a.depth * F::kSlot);  // [2][round][n_wk][NS * 16]
    const uint32_t part_tile = a.n_wk * NS * 16;
    const typename F::Tab tab = F::carve(reinterpret_cast<uint8_t*>(spart + 2 * a.round * part_tile), a.nblk);
    const uint32_t wk = (uint32_t)warp % a.n_wk, wr = (uint32_t)warp / a.n_wk;
    const uint32_t ct0 = blockIdx.x * a.tpc, nt = min(a.tpc, a.tiles - ct0);

    typename F::Copier copier;
    copier.init(a, lane);
    typename F::Lane ln;
    ln.init(a, tab, lane);
    pdl_late(a.late);
    Slots<NS, kSeg> slots;
    slots.init(a, lane);

    uint32_t p_tl = wr, p_strm = 0, p_kb = wk;  // the unit to request next: tile, stream, block
    uint32_t tl = wr, strm = 0, kb = wk;        // the unit to work off next
    uint32_t r0 = 0;                            // first tile of the round the warps meet for next
    const uint32_t n_prep = F::prep_count(a), x_at = a.late ? 0u : a.depth - 1;
    typename F::X x;
    typename F::Acc acc;
    acc.clear();
    uint32_t p_slot = 0, slot = 0;
    for (uint32_t it = 0;; ++it) {
        if (p_tl < nt) {
            const Unit u = find_unit<NS, kSeg>(a, slots, ct0 + p_tl, p_strm, p_kb);
            if (u.mat) copier.copy(a, u, ring + p_slot * F::kSlot, lane);
            p_kb += a.n_wk;
            if (p_kb >= a.nblk) {
                p_kb = wk;
                if (++p_strm == NS) {
                    p_strm = 0;
                    p_tl += a.n_wr;
                }
            }
        }
        cp_async_commit();
        if (++p_slot == a.depth) p_slot = 0;
        if (it == x_at) {
            if (!a.late) pdl_wait();
            if ((uint32_t)warp < n_prep) F::template load_x<kSeg>(x, a, extra, warp, lane);
        }
        if (it + 1 < a.depth) continue;
        if (it + 1 == a.depth) {  // ---- the activation, once the ring is full ----
            if (a.consume.n) consume_pushed(a.consume, blockIdx.x, gridDim.x, tid, blockDim.x);
            F::clear(tab, tid);
            for (uint32_t b = warp; b < n_prep; b += n_warps) {
                typename F::X next;
                if (b + n_warps < n_prep) F::template load_x<kSeg>(next, a, extra, b + n_warps, lane);
                F::prep(tab, x, a, b, lane);
                x = next;
            }
            __syncthreads();
        }
        bool meet = true;
        if (tl < nt) {
            if (a.depth == 2) cp_async_wait<1>();
            else if (a.depth == 3) cp_async_wait<2>();
            else cp_async_wait<3>();
            __syncwarp();
            const Unit u = find_unit<NS, kSeg>(a, slots, ct0 + tl, strm, kb);
            if (u.mat) ln.dot(a, u, smem_u32(ring) + slot * F::kSlot, acc);
            __syncwarp();
            if (++slot == a.depth) slot = 0;
            kb += a.n_wk;
            meet = false;
            if (kb >= a.nblk) {  // the warp's share of a tile's stream is complete
                float* part = spart + (((tl / a.round) & 1) * a.round + tl % a.round) * part_tile + wk * (NS * 16) + strm * 16;
                float v0, v1;
                ln.finish(acc, v0, v1);  // rows g and g + 8, this lane's share
                acc.clear();
                v0 += __shfl_xor_sync(0xFFFFFFFFu, v0, 1);
                v1 += __shfl_xor_sync(0xFFFFFFFFu, v1, 1);
                v0 += __shfl_xor_sync(0xFFFFFFFFu, v0, 2);
                v1 += __shfl_xor_sync(0xFFFFFFFFu, v1, 2);
                if ((lane & 3) == 0) {
                    part[lane >> 2] = v0;
                    part[(lane >> 2) + 8] = v1;
                }
                kb = wk;
                if (++strm == NS) {
                    strm = 0;
                    tl += a.n_wr;
                    meet = tl >= r0 + a.round || tl >= nt;
                }
            }
        }
        if (meet) {
            // ---- the warps meet: four lanes per row add the warps' shares, in a fixed order ----
            const uint32_t buf = (r0 / a.round) & 1, n_red = min(a.round, nt - r0) * 64;
            OutRow o{};
            if ((uint32_t)tid < n_red) o = out_row<EPI, kSeg>(a, ct0 + r0 + (tid >> 6), (tid >> 2) & 15u, (tid & 3u) == 0);
            __syncthreads();
            for (uint32_t i = tid; i < n_red; i += blockDim.x) {
                if (i != (uint32_t)tid) o = out_row<EPI, kSeg>(a, ct0 + r0 + (i >> 6), (i >> 2) & 15u, (i & 3u) == 0);
                const float* p = spart + (buf * a.round + (i >> 6)) * part_tile + ((i >> 2) & 15u);
                float v[NS];
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    float w = 0.f;
#pragma unroll 4
                    for (uint32_t k = i & 3u; k < a.n_wk; k += 4) w += p[k * (NS * 16) + s * 16];
                    w += __shfl_xor_sync(0xFFFFFFFFu, w, 1);
                    w += __shfl_xor_sync(0xFFFFFFFFu, w, 2);
                    v[s] = w;
                }
                write_out<NS, EPI>(a, o, v);
            }
            r0 += a.round;
            if (r0 >= nt) break;
        }
    }
}

struct NoExtra {};

// The form for many tiles per CTA, of one matrix (or pair): the CTA's units (16 rows x one block, tile by tile) are dealt to
// its warps in equal contiguous ranges. A warp writes the tiles it has to itself; of the at most two it shares with its
// neighbours, the parts meet in shared memory once, at the end, and are added in the order of the warps. No warp waits for
// another on the way, and none has more than one unit more to do than the next. A unit is requested into the slot that has
// just been read, so that the whole ring is in flight while a unit's sums are finished.
// (The tiles of a CTA shared by all its warps with a meeting every few of them, as above: LM head Q6_K 151936 x 4096 109.9
// us, here 99.4; Q4_K 40000 x 2816 16.6 and 14.3.)
template <typename F, int NS, int EPI>
__device__ __forceinline__ void flow_body(const SliceArgs& a) {
    extern __shared__ uint8_t smem_raw[];
    pdl_begin(a.late);
    uint8_t* base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    const uint32_t n_warps = blockDim.x >> 5;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t* ring = base + (size_t)warp * a.depth * F::kSlot;
    float* spart = reinterpret_cast<float*>(base + (size_t)n_warps * a.depth * F::kSlot);  // [warp][first, last range][NS * 16]
    const typename F::Tab tab = F::carve(reinterpret_cast<uint8_t*>(spart + n_warps * 2 * NS * 16), a.nblk);
    const uint32_t ct0 = (uint32_t)part_begin(blockIdx.x, a.tiles, gridDim.x);
    const uint32_t U = ((uint32_t)part_begin(blockIdx.x + 1, a.tiles, gridDim.x) - ct0) * a.nblk;
    auto begin_of = [&](uint32_t w) { return w * U / n_warps; };
    const uint32_t u0 = begin_of(warp), u1 = begin_of(warp + 1);

    typename F::Copier copier;
    copier.init(a, lane);
    typename F::Lane ln;
    ln.init(a, tab, lane);
    pdl_late(a.late);
    auto unit = [&](uint32_t tl, uint32_t strm, uint32_t kb) {
        Unit u;
        u.mat = a.A[NS == 2 ? strm : 0];
        u.end = a.a_end[NS == 2 ? strm : 0];
        u.row0 = (ct0 + tl) * 16;
        u.rows = min(16u, a.M - u.row0);
        u.lb = u.kb = kb;
        return u;
    };
    uint32_t p_u = u0, p_tl = u0 / a.nblk, p_kb = u0 - p_tl * a.nblk, p_strm = 0;  // the unit to request next
    uint32_t u = u0, tl = p_tl, kb = p_kb, strm = 0;                               // the unit to work off next
    uint32_t kb0 = kb, seg = 0;                                                    // the range: where it began, its number
    auto request = [&](uint32_t slot) {
        if (p_u < u1) {
            copier.copy(a, unit(p_tl, p_strm, p_kb), ring + slot * F::kSlot, lane);
            if (NS == 1 || ++p_strm == NS) {
                p_strm = 0;
                ++p_u;
                if (++p_kb == a.nblk) {
                    p_kb = 0;
                    ++p_tl;
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll 1
    for (uint32_t i = 0; i < a.depth; ++i) request(i);
    if (!a.late) pdl_wait();
    // ---- the activation ----
    const uint32_t n_prep = F::prep_count(a);
    typename F::X x;
    if ((uint32_t)warp < n_prep) F::template load_x<0>(x, a, NoExtra(), warp, lane);
    if (a.consume.n) consume_pushed(a.consume, blockIdx.x, gridDim.x, tid, blockDim.x);
    F::clear(tab, tid);
    for (uint32_t b = warp; b < n_prep; b += n_warps) {
        typename F::X next;
        if (b + n_warps < n_prep) F::template load_x<0>(next, a, NoExtra(), b + n_warps, lane);
        F::prep(tab, x, a, b, lane);
        x = next;
    }
    __syncthreads();

    typename F::Acc acc, other;  // of the stream at hand, of the other one
    acc.clear();
    other.clear();
    for (uint32_t slot = 0; u < u1;) {
        if (a.depth == 2) cp_async_wait<1>();
        else if (a.depth == 3) cp_async_wait<2>();
        else cp_async_wait<3>();
        __syncwarp();
        ln.dot(a, unit(tl, strm, kb), smem_u32(ring) + slot * F::kSlot, acc);
        __syncwarp();
        request(slot);  // into the slot just read
        if (++slot == a.depth) slot = 0;
        if (NS == 2) {
            const typename F::Acc t = acc;
            acc = other;
            other = t;
            if (++strm < NS) continue;
            strm = 0;
        }
        ++u;
        if (++kb < a.nblk && u < u1) continue;
        // ---- the warp's part of a tile is complete ----
        float v[NS][2];
        ln.finish(acc, v[0][0], v[0][1]);
        if (NS == 2) ln.finish(other, v[NS - 1][0], v[NS - 1][1]);
        acc.clear();
        other.clear();
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int i = 0; i < 2; ++i) {  // rows g and g + 8, the four lanes' shares
                v[s][i] += __shfl_xor_sync(0xFFFFFFFFu, v[s][i], 1);
                v[s][i] += __shfl_xor_sync(0xFFFFFFFFu, v[s][i], 2);
            }
        const uint32_t half = lane & 3, rr = (lane >> 2) + 8 * (half & 1);  // lanes 0 and 1 of a row's four: rows g and g + 8
        float r[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) r[s] = half ? v[s][1] : v[s][0];
        if (kb0 == 0 && kb == a.nblk) {
            write_out<NS, EPI>(a, out_row<EPI, 0>(a, ct0 + tl, rr, half < 2), r);
        } else if (half < 2) {
#pragma unroll
            for (int s = 0; s < NS; ++s) spart[((warp * 2 + (seg ? 1 : 0)) * NS + s) * 16 + rr] = r[s];
        }
        ++seg;
        kb0 = 0;
        if (kb == a.nblk) {
            kb = 0;
            ++tl;
        }
    }
    // ---- the shared tiles: 16 threads for each, at the first border between warps that lies inside it ----
    const uint32_t b = (uint32_t)(tid >> 4) + 1, ub = begin_of(b), t0 = ub / a.nblk * a.nblk;  // b, its unit, its tile's first
    const bool mine = b < n_warps && ub != t0 && begin_of(b - 1) <= t0;
    const OutRow o = out_row<EPI, 0>(a, ct0 + t0 / a.nblk, tid & 15u, mine);
    __syncthreads();
    if (!mine) return;
    float sum[NS];
    const float* p = spart + ((b - 1) * 2 + (begin_of(b - 1) == t0 ? 0 : 1)) * NS * 16 + (tid & 15u);
#pragma unroll
    for (int s = 0; s < NS; ++s) sum[s] = p[s * 16];
    for (uint32_t w = b; w < n_warps && begin_of(w) < t0 + a.nblk; ++w) {
        if (begin_of(w) == begin_of(w + 1)) continue;  // fewer units than warps
        p = spart + w * 2 * NS * 16 + (tid & 15u);
#pragma unroll
        for (int s = 0; s < NS; ++s) sum[s] += p[s * 16];
    }
    write_out<NS, EPI>(a, o, sum);
}
template <typename F, int NS, int EPI, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, kWarps == 8 ? 2 : 1) dmmv_flow_kernel(const SliceArgs a) {
    flow_body<F, NS, EPI>(a);
}

template <typename F, int NS, int EPI, int kSeg, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, kWarps == 8 ? 2 : 1) dmmv_slice_kernel(const SliceArgs a) {
    slice_body<F, NS, EPI, kSeg>(a, NoExtra());
}
template <typename F, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, kWarps == 8 ? 2 : 1) dmmv_slice_merge_kernel(const SliceArgs a, const MergeArgs m) {
    slice_body<F, 1, EPI_PLAIN, 0>(a, m);
}

constexpr uint32_t kSliceSmem1 = 232448u, kSliceSmem2 = 113u * 1024u;  // one, two CTAs per SM

// Units a warp keeps in flight: four at most; two where there are more than `deep` warps. (Q6_K in sixteen warps, as many as fit and
// two: 8192 x 12288 23.2 and 22.6 us, 5120 x 8192 13.4 and 12.9, 28672 x 12288 66.3 and 65.8, 40000 x 10240 71.9 and 71.8.)
inline uint32_t most_depth(uint32_t depth, uint32_t warps, uint32_t deep) {
    const uint32_t most = warps > deep ? 2u : 4u;
    return depth < most ? depth : most;
}

// Cuts the work. `rows(i)`: the row counts of the matrices (kSeg 1) or of one expert slot. False: x does not fit.
template <typename F>
bool slice_plan(SliceArgs& a, int NS, int kSeg, int sm_count, uint32_t& warps, uint32_t& grid, uint32_t& smem) {
    a.bpe = (a.K + F::kCols - 1) / F::kCols;
    a.nblk = a.bpe * (kSeg == 3 ? a.nseg : 1u);
    const uint32_t sms = sm_count > 0 ? (uint32_t)sm_count : 148u;
    // Up to K = 4096: eight warps and two CTAs per SM, so that the next kernel's CTAs find room early; else one CTA with as
    // many warps as the registers allow. A format whose units are bound by latency (kMost > 16) always takes the latter
    // (MXFP4 gate + up 20.1 -> 17.9 us with 18 warps instead of 12); along slots K is long enough for twelve to sixteen.
    // Warps along K: as few as leave the longest share unchanged; the rest along the rows.
    const bool pair = F::kMost <= 16 && a.nblk * F::kCols <= 4096;
    const uint32_t most = pair ? 8u : kSeg == 3 ? 16u : F::kMost;
    const uint32_t per_sm = pair ? 2u : 1u, room = pair ? kSliceSmem2 : kSliceSmem1;
    uint32_t per = (a.nblk + most - 1) / most;
    auto cut = [&](uint32_t p, uint32_t wr, uint32_t round) {  // false: two units per warp do not fit beside x
        a.n_wk = (a.nblk + p - 1) / p;
        a.n_wr = wr;
        a.round = round;
        warps = a.n_wk * wr;
        const uint32_t fixed = 128u + 2u * round * a.n_wk * (uint32_t)NS * 16u * 4u + F::table_bytes(a.nblk);
        if (fixed + warps * 2u * F::kSlot > room) return false;
        a.depth = (room - fixed) / (warps * F::kSlot);
        a.depth = most_depth(a.depth, warps, F::kDeepWarps);
        smem = fixed + warps * a.depth * F::kSlot;
        return true;
    };
    // Four tiles per CTA and more: the cut whose busiest warp has least to do, tiles of a CTA dealt to n_wr rows of warps, a
    // longer share of K for each where more rows of warps fit; meetings every eight tiles, nine with three rows of warps (a
    // multiple of the rows, so that none idles before one; below, with one to three tiles per CTA, four and six). (Q4_K 8192 x 12288 16.3 ->
    // 14.6 us, 11008 x 5120 12.2 -> 10.1, 65536 x 8192 53.8 -> 52.1 against the cut below.)
    const uint32_t tpc16 = ((a.M + 15) / 16 + sms * per_sm - 1) / (sms * per_sm);
    uint32_t tall_per = 0, tall_wr = 0;
    if (kSeg == 0 && tpc16 >= 4) {
        uint32_t least = 0xFFFFFFFFu;
        for (uint32_t p = a.nblk < per * 4 ? a.nblk : per * 4; p >= per; --p) {
            const uint32_t wk = (a.nblk + p - 1) / p;
            for (uint32_t wr = 1; wr <= 4 && wr * wk <= most; ++wr) {
                // by 5 % at least: between equals the longer share (Q6_K 151936 x 4096: 109 us, 112 with all warps along K)
                if ((uint64_t)((tpc16 + wr - 1) / wr * p) * 20 < (uint64_t)least * 19 && cut(p, wr, wr == 3 ? 9 : 8)) {
                    least = (tpc16 + wr - 1) / wr * p;
                    tall_per = p;
                    tall_wr = wr;
                }
            }
        }
    }
    if (tall_per) {
        cut(tall_per, tall_wr, tall_wr == 3 ? 9 : 8);
    } else {
        const uint32_t wk = (a.nblk + per - 1) / per, wr = most / wk > 4 ? 4 : most / wk;
        if (!cut(per, wr, wr == 3 ? 6 : 4)) return false;
    }
    // Tile height: the one that gives the busiest CTA the least to do (an MMA costs the same for fewer rows: 0.3 per row)
    uint32_t best = 0xFFFFFFFFu;
    for (uint32_t h = 16; h >= 4; --h) {
        uint32_t tiles = 0;
        if (kSeg == 1) for (uint32_t i = 0; i < a.nseg; ++i) tiles += (a.segM[i] + h - 1) / h;
        else tiles = ((a.M + h - 1) / h) * (kSeg == 2 ? a.nseg : 1u);
        const uint32_t tpc = (tiles + sms * per_sm - 1) / (sms * per_sm);
        const uint32_t cost = tpc * (10 * h + 3 * (16 - h));
        if (cost < best) {
            best = cost;
            a.h = h;
            a.tiles = tiles;
            a.tpc = tpc;
        }
    }
    a.tpe = (a.M + a.h - 1) / a.h;
    a.tpe_mul = reciprocal(a.tpe, a.tiles);
    a.bpe_mul = reciprocal(a.bpe, a.nblk);
    if (kSeg == 1) {
        uint32_t t = 0;
        for (uint32_t i = 0; i < 3; ++i) {
            if (i < a.nseg) t += (a.segM[i] + a.h - 1) / a.h;
            a.seg_end[i] = i < a.nseg ? t : 0xFFFFFFFFu;
        }
    }
    grid = (a.tiles + a.tpc - 1) / a.tpc;
    return true;
}

// The cut of the other form (flow_body), where it is the faster one: many tiles per SM.
// F::flow_pair(K): whether eight warps on each of two CTAs are tried, F::flow_tiles(K): from how many tiles per two SMs (both
// streams counted) they are ahead. In tiles per SM, measured over 250 shapes, this form against the one above:
//   Q4_K   K <= 512 always (65536 rows 6.2 and 9.2 us: most warps had no block); K <= 4096 from 8 (K = 4096, 16500 rows 10.4
//          and 10.2, 20000 rows 11.7 and 12.7, 28672 rows 14.9 and 16.6), beyond from 3 (5120 x 5120 7.5 and 7.7, 14336 x
//          5120 11.3 and 12.9)
//   Q6_K   K <= 7424 from 2 (5120 x 2816 8.3 and 9.0, 8192 x 4608 13.3 and 13.8, 21669 x 4608 27.3 and 31.4, 65536 x 6144 67.2 and
//          73.0, 128256 x 3072 85.8 and 101.6, 151936 x 4096 99.1 and 108.6; the other way 20000 x 5120 29.2 and 27.7); K = 8192 (rows
//          on 16-byte boundaries) from 4.5 (28672 rows 44.2, one CTA 47.7, the form above 45.9; 12000 rows 22.6, 24.5, 22.2; below,
//          8192 rows 17.0 and 16.2)
//   MXFP4  K <= 1024 always (20000 x 512 4.1 and 7.8), beyond from 10 (20000 x 2880 14.4 and 13.8, 28672 x 2880 19.3 and 20.4)
// Beyond, Q6_K takes one CTA of sixteen warps from 4.5 tiles per SM (11008 x 12288 27.9 us in both forms, 28672 rows 65.8 and 69.0,
// 30000 x 12032 75.9 and 84.2; two CTAs of eight 32.4, 64.7, 85.1, 12000 x 7936 28.8 for 27.6, 40000 x 10240 69.3 for 71.8); the others
// stay above (Q4_K 65536 x 12288 76 and 74).
template <typename F>
bool flow_plan(SliceArgs& a, int NS, int sm_count, uint32_t& warps, uint32_t& grid, uint32_t& smem) {
    a.nblk = a.bpe = (a.K + F::kCols - 1) / F::kCols;
    a.tiles = (a.M + 15) / 16;
    a.h = 16;
    const uint32_t sms = sm_count > 0 ? (uint32_t)sm_count : 148u;
    auto cut = [&](uint32_t n, uint32_t room) {
        warps = n;
        const uint32_t fixed = 128u + warps * 2u * (uint32_t)NS * 16u * 4u + F::table_bytes(a.nblk);
        if (fixed + warps * 2u * F::kSlot > room) return false;
        a.depth = (room - fixed) / (warps * F::kSlot);
        a.depth = most_depth(a.depth, warps, F::kDeepWarps);
        smem = fixed + warps * a.depth * F::kSlot;
        return true;
    };
    uint32_t ctas = 2 * sms;
    if (F::flow_pair(a.K) && cut(8, kSliceSmem2)) {
        if (a.tiles * (uint32_t)NS * 2 < F::flow_tiles(a.K) * sms) return false;
    } else {
        ctas = sms;
        if (!F::kFlowOne || a.tiles * 2 < 9 * sms || !cut(16, kSliceSmem1)) return false;
    }
    const uint32_t busy = (uint32_t)(((uint64_t)a.tiles * a.nblk + warps - 1) / warps);  // CTAs with a unit for every warp
    grid = ctas < busy ? ctas : busy;
    return true;
}

template <typename F, int NS, int EPI, int kSeg>
cudaError_t slice_launch(SliceArgs a, int sm_count, cudaStream_t s) {
    uint32_t warps, grid, smem;
    if constexpr (kSeg == 0) {
        if (flow_plan<F>(a, NS, sm_count, warps, grid, smem)) {
            static std::atomic<uint64_t> flow8{0}, flow16{0};
            if (warps == 8) {
                auto kern = dmmv_flow_kernel<F, NS, EPI, 8>;
                if (cudaError_t e = ensure_dynamic_smem(kern, kSliceSmem1, flow8); e != cudaSuccess) return e;
                return launch_chained(kern, dim3(grid), dim3(warps * 32), smem, s, a);
            }
            if constexpr (F::kFlowOne) {
                auto kern = dmmv_flow_kernel<F, NS, EPI, 16>;
                if (cudaError_t e = ensure_dynamic_smem(kern, kSliceSmem1, flow16); e != cudaSuccess) return e;
                return launch_chained(kern, dim3(grid), dim3(warps * 32), smem, s, a);
            }
        }
    }
    if (!slice_plan<F>(a, NS, kSeg, sm_count, warps, grid, smem)) return cudaErrorInvalidConfiguration;
    static std::atomic<uint64_t> attr8{0}, attr16{0};
    if (warps <= 8) {
        auto kern = dmmv_slice_kernel<F, NS, EPI, kSeg, 8>;
        if (cudaError_t e = ensure_dynamic_smem(kern, kSliceSmem1, attr8); e != cudaSuccess) return e;
        return launch_chained(kern, dim3(grid), dim3(warps * 32), smem, s, a);
    }
    auto kern = dmmv_slice_kernel<F, NS, EPI, kSeg, kSeg == 3 ? 16 : (int)F::kMost>;
    if (cudaError_t e = ensure_dynamic_smem(kern, kSliceSmem1, attr16); e != cudaSuccess) return e;
    return launch_chained(kern, dim3(grid), dim3(warps * 32), smem, s, a);
}

// How far the formats reach whose x is 21-bit fixed point per 256 elements (Q4_K, Q6_K; relative L2 error 1.1e-6, f32 sums
// 1.2e-7): the longest (concatenated) x, and the fewest units of 16 rows x 512 columns. Beyond, the row kernels' f32.
constexpr uint32_t kFixedPointMaxK = 12288, kFixedPointMinUnits = 16;

// Does the activation of a launch fit beside two units per warp?
template <typename F>
bool slice_fits(uint32_t K, uint32_t slots, int NS) {
    SliceArgs a = {};
    a.M = 16;
    a.K = K;
    a.nseg = slots;
    uint32_t w, g, m;
    return slice_plan<F>(a, NS, slots > 1 ? 3 : 0, 148, w, g, m);
}

}  // namespace
}  // namespace zc
