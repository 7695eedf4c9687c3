// resident.cuh — launch interface of the block-resident persistent iteration
// (resident.cu) for graphs of up to kResMaxArcs arcs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "graph.cuh"

namespace prg {

constexpr uint32_t kResL1Hot = 8192;
constexpr uint64_t kResMaxArcs = 10u << 20;  // see resident.cu
constexpr unsigned kResBlocks = 160;         // most blocks of a launch

enum ResKind : int {
    RES_POWER = 0,  // damped FP64 power iteration (uniform or personalised teleport)
    RES_EIG = 1,    // max-normalised iteration x' = (shift I + A) x / max
};

// Read once, by whichever thread comes first.
struct DeviceLimits {
    int sms = 0, smem_optin = 0;
};
const DeviceLimits &device_limits();

struct ResPlan {
    unsigned grid = 0;   // 0: the graph does not fit, use the other kernels
    size_t smem = 0;     // dynamic shared memory per block
    bool stream = false; // column indices and weights are read from memory every iteration, not kept in shared memory
    uint32_t alpha = 0;  // a row weighs as much as alpha arcs in the split over the blocks
};

struct ResArgs {
    const uint32_t *row_ptr;
    const uint32_t *col;
    const double *w64;    // null: unweighted
    const double *dval;   // RES_POWER
    const double *t64;    // RES_POWER: teleport vector (null: uniform)
    const double *start;  // RES_POWER: start vector (null = the teleport vector)
    double *x_out;        // the last iterate; RES_EIG: in, the start vector
    double *xt[2];        // RES_POWER: gathered vectors, rewritten in turn
    double2 *rec;         // 2 x grid records
    uint32_t *bar;        // arrival counter, zero at launch
    Ctl *ctl;             // out: iters, diff, done, status; RES_EIG: dsum = (x.Ax, x.x)
    uint64_t total;       // arcs + alpha n
    // a plan made without the rows' lengths: the longest row on the device and
    // the shared memory given; where a block's share may exceed it, every block
    // returns with Ctl::status = 1 (null: the plan is known to fit).  With
    // `longest`, a nonzero status at launch makes the kernel return at once.
    const uint32_t *longest;
    uint32_t smem;
    uint32_t n, alpha, max_iter;
    uint32_t bar_extra;   // test hook: arrivals every barrier waits for beyond the grid's
    uint32_t l1hot;       // sources at or above this id are gathered without L1 allocation
    double damping, thr, shift;
};

// Launch shape for graph g, or grid = 0 where it does not apply (reads the
// rows' split back from the device when the sizes alone do not decide).
ResPlan res_plan(const DeviceGraph &g, int kind, cudaStream_t s);
// Whether a graph of these sizes can have a plan at all, whatever its rows.
bool res_sizes_fit(uint32_t n, uint64_t arcs, bool weighted, int kind);
// No plan holds a longer row.
uint32_t res_longest_row(uint32_t n, uint64_t arcs);
// The plan before the graph is built, for graphs whose indices surely stay in
// shared memory as long as no row is long (ResArgs::longest checks that).
ResPlan res_plan_blind(uint32_t n, uint64_t arcs, bool weighted, int kind);
// Bytes of scratch the launch needs (records and arrival counter).
size_t res_scratch_bytes(unsigned grid);
// Iterates until the stop rule holds or max_iter iterations ran; false when
// the device cannot hold the grid at once (nothing was launched).
bool launch_resident(int kind, const ResPlan &p, const ResArgs &a, cudaStream_t s);

}  // namespace prg
