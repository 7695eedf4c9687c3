// pool.cuh — per-call host resources that are expensive to create: pinned
// control-block slabs and non-blocking streams.
//
// A one-call drop-in creates a handle, solves and destroys it.  On a B200
// host, cudaMallocHost takes 1.3-7 ms and cudaFreeHost 0.2-2 ms whatever the
// size (page pinning and a device synchronisation), and creating and
// destroying a stream 0.2 ms, while the device work of a small graph is below
// 0.5 ms: G(1000, 25 000) took 4-14 ms per call, of which these were over
// 80 %.  Released slabs and streams are therefore kept for the next call.
//
// The pool is bounded (kPoolSlabs x kSlabBytes pinned bytes and kPoolStreams
// streams; what exceeds that is given back to CUDA at once), guarded by a
// mutex, and keyed by the CUDA context: entries of a context that is gone
// (another device, or the process reset it) are never handed out.  What is
// still pooled when the process ends goes with its context.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace prg {

constexpr size_t kSlabBytes = 1024;
constexpr size_t kPoolSlabs = 64;
constexpr size_t kPoolStreams = 16;

// A pinned host slab of kSlabBytes, its contents unspecified.  Release it
// only when no copy into or out of it is in flight.
void *pinned_acquire();
void pinned_release(void *p);

// A non-blocking stream of the current device with no work in flight.
// Releasing synchronises it; a stream whose work failed is destroyed.
cudaStream_t stream_acquire();
void stream_release(cudaStream_t s);

}  // namespace prg
