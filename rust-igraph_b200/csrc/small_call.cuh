// small_call.cuh — one-call drop-ins on small graphs as two launches: a
// cooperative CSR build (small_call.cu) and the block-resident iteration
// (resident.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "resident.cuh"

namespace prg {

struct SmallCall {
    uint32_t n = 0;
    uint64_t m = 0;
    const uint32_t *from = nullptr, *to = nullptr;  // host
    const double *w = nullptr;                      // host weights or null
    bool directed = true;
    int kind = RES_POWER;
    const double *reset = nullptr;  // RES_POWER: normalised teleport vector (host) or null
    double damping = 0.85, thr = 0, shift = 0;
    uint32_t max_iter = 0;
    bool check_weights = false;     // refuse NaN, infinite and negative weights
    bool strength_seed = false;     // RES_EIG: start from the row sums over their maximum (else from ones)
};

// An uploaded edge list (one allocation).
struct SmallEdges {
    unsigned char *block = nullptr;  // null: nothing is held
    const uint32_t *from = nullptr, *to = nullptr;
    const double *w = nullptr;
};

struct SmallResult {
    uint32_t iterations = 0, max_endpoint = 0, bad_edge = 0;
    double eigenvalue = 0;
    SmallEdges edges;  // SMALL_NOT_HERE after the upload: for the general path, the caller's to free
};

enum SmallStatus : int32_t {
    SMALL_DONE = 0,
    SMALL_NOT_HERE = 1,      // take the general path (nothing written to out)
    SMALL_OUT_OF_RANGE = 2,  // an endpoint is >= n: SmallResult::max_endpoint
    SMALL_BAD_WEIGHT = 3,    // check_weights: SmallResult::bad_edge is the first such edge
    SMALL_LONG_ROW = 4,      // (device) a row no plan holds
};

// Solves into out (host double[n]).  Sizes, tuning and the rows' lengths
// decide whether the call runs here.
SmallStatus small_call(const SmallCall &c, double *out, SmallResult &r, cudaStream_t s);

}  // namespace prg
