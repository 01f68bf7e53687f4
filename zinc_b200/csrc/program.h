// Recorded sequences of matvecs as one kernel: what a call contributes, and how a run of calls is cut.
#pragma once

#include <cuda.h>

#include "kernels.h"

namespace zc {

constexpr uint32_t kProgMaxOps = 220;   // with which a program fits the 32,764 bytes of kernel parameters
constexpr uint32_t kProgMaxDeps = 512;

// The third: rows that do not start on 16-byte boundaries. Eight rows together do, so a tile is the rows c, c + 8, .. c + 120
// of 128: within groups of eight they lie at one place, and one tensor copy fetches them.
enum : uint8_t { PROG_Q4K = 0, PROG_Q6K = 1, PROG_Q6K_APART = 2 };
enum : uint8_t { PROG_PLAIN = 0, PROG_GATE_UP = 1, PROG_SIGMOID_ACC = 2 };

// One recorded call. Tiles are 16 rows of one matrix (of both matrices for gate + up); tile t belongs to CTA (first + t) % grid.
struct alignas(16) ProgramOp {
    const uint8_t* A[3];
    float* y[3];
    const float* x;
    const float* gate;
    uint32_t M[3];
    uint32_t tile_end[2];     // of matrices 0 and 1 (up to three matrices on one x)
    uint32_t tiles;
    uint32_t K;
    uint32_t x_table;         // where converted x lies, in 16 bytes of Program::tables
    uint16_t units;           // of a tile: 16 rows x two blocks, both streams
    uint16_t map;             // the first matrix's tensor map
    uint16_t first;
    uint16_t table;           // where x goes in shared memory, in 16 bytes
    uint16_t wait_warps;      // the compute warps must all have reached this op before the table is replaced
    uint16_t x_first;         // block b of x is converted by CTA (x_first + b) % grid
    uint16_t dep0, deps_x, deps_y;  // ops that must be complete before this one reads x, writes y: Program::deps[dep0 ..]
    uint8_t kind, epi, acc, streams, awaited;
};

struct Program {
    uint32_t n_ops, grid;
    uint32_t* done;           // finished tiles of every op; these counters are zero between launches
    uint32_t* converted;      // converted blocks of x of every op
    uint32_t* left;           // CTAs that have left
    uint8_t* tables;          // table_bytes of memory for converted x
    const uint8_t* maps;      // n_maps tensor maps of the weights
    uint32_t table_bytes, n_maps;
    uint32_t spin_limit;      // polls after which a wait gives up; program_plan sets it
    uint32_t* status;
    uint16_t deps[kProgMaxDeps];
    ProgramOp ops[kProgMaxOps];
};
static_assert(sizeof(Program) <= 32764, "kernel parameters");

// The call that `mode` and the arguments describe, as an op; false: it takes another kernel than the streaming matvecs of
// Q4_K and Q6_K, or carries something they alone carry.
bool program_op(uint32_t type, int mode, const DmmvArgs& a, ProgramOp& op);
bool program_op_multi(uint32_t type, uint32_t n, const uint8_t* const* A, float* const* y, const uint32_t* M, const DmmvArgs& common,
                      ProgramOp& op);
// Orders the first ops of `list` as a program; returns how many it took (at least two, or none). With `gain`: as many as are worth
// being joined, and what that is to gain in us; else as many as there can be.
uint32_t program_plan(const ProgramOp* list, uint32_t n, int sm_count, Program& p, float* gain);
// Fills the program's n_maps tensor maps; returns how many ops it described: fewer than n_ops where a matrix cannot be.
uint32_t program_maps(const Program& p, CUtensorMap* maps);
// The kernel for a graph node: its function, block size and shared memory; cudaErrorNotSupported where it does not fit the device.
cudaError_t program_kernel(int sm_count, void** func, uint32_t& threads, uint32_t& smem);

}  // namespace zc
