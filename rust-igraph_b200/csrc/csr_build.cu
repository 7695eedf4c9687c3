// csr_build.cu — device construction of the in-arc CSR (the transpose the
// power iteration pulls over), out-degree / out-strength and the row-block
// work list of the SpMV.
//
// Semantics follow rust-igraph exactly:
//   * arcs: directed edge u->v gives in_adj[v] += u; an undirected edge
//     {u,v} gives in_adj[u] += v then in_adj[v] += u, a self-loop gives
//     in_adj[v] += v twice (pagerank.rs:76-101, pagerank_weighted.rs:103-124,
//     personalized_pagerank.rs:125-143);
//   * rows keep edge-id order: the arcs are produced in edge order and
//     sorted by destination with a STABLE radix sort, so row v lists its
//     in-neighbours in the same order as the reference's Vec<Vec<u32>>;
//   * out-degree = neighbors_iter(v).len(): out-edges for directed graphs,
//     all incident edge ends (self-loop twice) for undirected ones
//     (graph.rs:877-900, pagerank.rs:69-72);
//   * out-strength accumulates w per arc end (self-loop adds 2w,
//     pagerank_weighted.rs:81-101); a vertex is dangling iff its divisor is 0.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <exception>
#include <vector>

#include "graph.cuh"
#include "pool.cuh"
#include "prims.cuh"

namespace prg {

static inline unsigned grid_for(uint64_t n, unsigned per_block, unsigned cap = 148u * 64u) {
    uint64_t g = (n + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

// What the build running on this thread holds: an exception (out of device
// memory) frees it.
struct Scratch {
    cudaStream_t s;
    std::vector<void *> held;
    Scratch *outer;
    int unwinding = std::uncaught_exceptions();
    static thread_local Scratch *top;
    explicit Scratch(cudaStream_t stream) : s(stream), outer(top) { top = this; }
    Scratch(const Scratch &) = delete;
    ~Scratch() {
        top = outer;
        if (std::uncaught_exceptions() == unwinding) return;
        for (void *p : held) cudaFreeAsync(p, s);
    }
    // p is freed, or the graph's from here on
    static void forget(void *p) {
        if (!top) return;
        auto &h = top->held;
        h.erase(std::remove(h.begin(), h.end(), p), h.end());
    }
};
thread_local Scratch *Scratch::top = nullptr;

template <class T>
static T *dalloc(uint64_t count, cudaStream_t s) {
    void *p = nullptr;
    PRG_CUDA(cudaMallocAsync(&p, std::max<uint64_t>(count, 1) * sizeof(T), s));
    if (Scratch::top) Scratch::top->held.push_back(p);
    return (T *)p;
}
template <class T>
static void dfree(T *&p, cudaStream_t s) {
    if (!p) return;
    Scratch::forget((void *)p);
    cudaFreeAsync((void *)p, s);
    p = nullptr;
}

// ------------------------------------------------------------------ scan

constexpr int kScanItems = 16;
constexpr int kScanTile = kThreads * kScanItems;

__global__ void __launch_bounds__(kThreads) scan_tile_sums(const uint32_t *in, uint64_t n, uint32_t *bsum) {
    __shared__ uint32_t sh[32];
    uint64_t base = (uint64_t)blockIdx.x * kScanTile;
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        uint64_t idx = base + (uint64_t)i * kThreads + threadIdx.x;
        if (idx < n) acc += in[idx];
    }
    uint32_t t = block_sum<uint32_t>(acc, sh);
    if (threadIdx.x == 0) bsum[blockIdx.x] = t;
}

// Single-block exclusive scan of a (moderate) array in place; writes total.
__global__ void __launch_bounds__(1024) scan_single_block(uint32_t *a, uint64_t n, uint32_t *total) {
    __shared__ uint32_t sh[33];
    uint64_t per = (n + blockDim.x - 1) / blockDim.x;
    uint64_t lo = per * threadIdx.x, hi = lo + per < n ? lo + per : n;
    uint32_t s = 0;
    for (uint64_t i = lo; i < hi; i++) s += a[i];
    uint32_t tot;
    uint32_t pre = block_excl_scan(s, sh, &tot);
    for (uint64_t i = lo; i < hi; i++) {
        uint32_t v = a[i];
        a[i] = pre;
        pre += v;
    }
    if (threadIdx.x == 0 && total) *total = tot;
}

__global__ void __launch_bounds__(kThreads) scan_tiles_apply(const uint32_t *in, uint32_t *out, uint64_t n,
                                                             const uint32_t *boff) {
    __shared__ uint32_t sh[33];
    __shared__ uint32_t tile[kScanTile];
    uint64_t base = (uint64_t)blockIdx.x * kScanTile;
    // coalesced load into shared, then each thread scans a contiguous run
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        uint64_t idx = base + (uint64_t)i * kThreads + threadIdx.x;
        tile[i * kThreads + threadIdx.x] = idx < n ? in[idx] : 0u;
    }
    __syncthreads();
    uint32_t run[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        run[i] = tile[threadIdx.x * kScanItems + i];
        s += run[i];
    }
    uint32_t tot;
    uint32_t pre = block_excl_scan(s, sh, &tot) + boff[blockIdx.x];
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        tile[threadIdx.x * kScanItems + i] = pre;
        pre += run[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        uint64_t idx = base + (uint64_t)i * kThreads + threadIdx.x;
        if (idx < n) out[idx] = tile[i * kThreads + threadIdx.x];
    }
}

void exclusive_scan_u32(const uint32_t *in, uint32_t *out, uint64_t n, cudaStream_t s) {
    uint64_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 0) nb = 1;
    uint32_t *bsum = dalloc<uint32_t>(nb + 1, s);
    scan_tile_sums<<<(unsigned)nb, kThreads, 0, s>>>(in, n, bsum);
    scan_single_block<<<1, 1024, 0, s>>>(bsum, nb, out + n);
    scan_tiles_apply<<<(unsigned)nb, kThreads, 0, s>>>(in, out, n, bsum);
    PRG_CUDA(cudaGetLastError());
    dfree(bsum, s);
}

// ------------------------------------------------------------------ radix sort

constexpr int kRsThreads = 512;
constexpr int kRsItems = 8;
constexpr int kRsTile = kRsThreads * kRsItems;  // 4096 pairs
constexpr int kRsWarps = kRsThreads / 32;

__global__ void __launch_bounds__(kThreads) rs_upsweep(const uint32_t *keys, uint64_t N, uint64_t chunk, int shift,
                                                       int bits, uint32_t *counts, uint32_t G) {
    __shared__ uint32_t h[kThreads / 32][256];
    for (int i = threadIdx.x; i < kThreads * 8; i += kThreads) (&h[0][0])[i] = 0;
    __syncthreads();
    const uint32_t mask = (1u << bits) - 1u;
    uint64_t begin = (uint64_t)blockIdx.x * chunk;
    uint64_t end = begin + chunk < N ? begin + chunk : N;
    int w = threadIdx.x >> 5;
    for (uint64_t i = begin + threadIdx.x; i < end; i += kThreads) {
        uint32_t d = (keys[i] >> shift) & mask;
        atomicAdd(&h[w][d], 1u);
    }
    __syncthreads();
    uint32_t t = threadIdx.x;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kThreads / 32; k++) s += h[k][t];
    if (t <= mask) counts[(uint64_t)t * G + blockIdx.x] = s;
}

// Stable scatter: each chunk is processed tile by tile; within a tile keys
// are ranked per warp in position order, then ordered by digit in shared
// memory and written out in digit runs (coalesced).  Bound by the instructions
// and shared-memory accesses of the ranking, not by memory (67 M pairs: 1.07 GB,
// 0.16 ms at the copy rate).  So the lanes with equal digits are found by
// ballots over the digit's bits, for all of a lane's keys before the first
// count is read (match.any: 0.49 ms against 0.39), key and value move through
// shared memory as one word, a digit's place in the tile is folded into the
// warps' counts, and two blocks of 64 registers a thread, which spill nothing,
// share an SM (three of 40: 0.45; 16 keys per lane 0.55).  67 M pairs, R-MAT
// scale 22 heads, passes of 8, 7 and 7 bits: 0.58 + 0.51 + 0.51 ms (8 bits each,
// tiles of 2048, match.any) before, 0.49 + 0.36 + 0.36 now.
template <int BITS>
struct RsShared {
    uint2 pairs[kRsTile];
    uint32_t at[kRsWarps][1 << BITS];  // a warp's count of each digit, then the place of its first in the tile
    uint32_t base[1 << BITS];          // of the digit's run in the output, less its start in the tile
    uint32_t scan[33];
};
template <int BITS>
__global__ void __launch_bounds__(kRsThreads, 2) rs_downsweep(const uint32_t *kin, const uint32_t *vin,
                                                              uint32_t *kout, uint32_t *vout, uint64_t N,
                                                              uint64_t chunk, int shift, int bits,
                                                              const uint32_t *offsets, uint32_t G) {
    extern __shared__ __align__(16) unsigned char s_rs[];
    RsShared<BITS> &sh = *reinterpret_cast<RsShared<BITS> *>(s_rs);
    constexpr int kDigits = 1 << BITS;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const uint32_t mask = (1u << bits) - 1u;
    uint64_t begin = (uint64_t)blockIdx.x * chunk;
    uint64_t end = begin + chunk < N ? begin + chunk : N;
    uint32_t off = (uint32_t)tid <= mask ? offsets[(uint64_t)tid * G + blockIdx.x] : 0u;
    const uint32_t ltmask = lanemask_lt();
    const uint32_t first = w * (32 * kRsItems) + lane;  // this lane's first key of a tile

    for (uint64_t tb = begin; tb < end; tb += kRsTile) {
        uint32_t key[kRsItems], val[kRsItems], peers[kRsItems];
        const uint32_t nvalid = (uint32_t)min((uint64_t)kRsTile, end - tb);
        const uint32_t *kt = kin + tb + first, *vt = vin + tb + first;
#pragma unroll
        for (int i = 0; i < kRsItems; i++) key[i] = first + 32 * i < nvalid ? __ldcs(kt + 32 * i) : 0u;
#pragma unroll
        for (int i = 0; i < kRsItems; i++) val[i] = first + 32 * i < nvalid ? __ldcs(vt + 32 * i) : 0u;
        for (int i = lane; i < kDigits; i += 32) sh.at[w][i] = 0;
#pragma unroll
        for (int i = 0; i < kRsItems; i++) {
            const uint32_t d = key[i] >> shift;
            uint32_t p = __ballot_sync(0xffffffffu, first + 32 * i < nvalid);
#pragma unroll
            for (int b = 0; b < BITS; b++) {
                const uint32_t one = (uint32_t)((int32_t)((d & mask) << (31 - b)) >> 31);  // the bit, 32 times
                p &= ~(__ballot_sync(0xffffffffu, one) ^ one);
            }
            peers[i] = p;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kRsItems; i++) {
            const uint32_t before = sh.at[w][key[i] >> shift & mask], rank = __popc(peers[i] & ltmask);
            __syncwarp();
            if (first + 32 * i < nvalid && rank == 0u) sh.at[w][key[i] >> shift & mask] = before + __popc(peers[i]);
            __syncwarp();
            peers[i] = before + rank;  // the key's place among the warp's keys of its digit
        }
        __syncthreads();
        uint32_t cnt = 0, tot;
        if (tid < kDigits) {
#pragma unroll
            for (int k = 0; k < kRsWarps; k++) cnt += sh.at[k][tid];
        }
        uint32_t ds = block_excl_scan(cnt, sh.scan, &tot);
        if (tid < kDigits) {
            sh.base[tid] = off - ds;
            off += cnt;
#pragma unroll
            for (int k = 0; k < kRsWarps; k++) {
                const uint32_t c = sh.at[k][tid];
                sh.at[k][tid] = ds;
                ds += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kRsItems; i++)
            if (first + 32 * i < nvalid)
                sh.pairs[sh.at[w][key[i] >> shift & mask] + peers[i]] = make_uint2(key[i], val[i]);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kRsItems; i++) {
            const uint32_t j = tid + i * kRsThreads;
            if (j < nvalid) {
                const uint2 p = sh.pairs[j];
                const uint32_t gpos = sh.base[p.x >> shift & mask] + j;
                kout[gpos] = p.x;
                vout[gpos] = p.y;
            }
        }
        __syncthreads();
    }
}

template <int BITS>
static void launch_downsweep(uint64_t G, const uint32_t *keys, const uint32_t *vals, uint32_t *kout, uint32_t *vout,
                             uint64_t N, uint64_t chunk, int shift, int bits, const uint32_t *counts, cudaStream_t s) {
    constexpr int smem = (int)sizeof(RsShared<BITS>);
    PRG_CUDA(cudaFuncSetAttribute(rs_downsweep<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    rs_downsweep<BITS><<<(unsigned)G, kRsThreads, smem, s>>>(keys, vals, kout, vout, N, chunk, shift, bits, counts,
                                                             (uint32_t)G);
}

// Stable passes over the key's bits from first_shift up to key_bits, in as few
// digits of at most 8 bits as it takes, the bits spread evenly (fewer digits:
// longer runs to write).  The first pass reads (keys, vals), which stay as they are, and
// writes (k[0], v[0]); later ones go back and forth between k[0], v[0] and
// k[1], v[1] (k[1], v[1] may be the source itself, which is then lost).  The
// result is in *keys / *vals, the source when there is nothing to sort.
static int radix_pass_count(uint64_t N, int first_shift, int key_bits) {
    return N <= 1 || key_bits <= first_shift ? 0 : (key_bits - first_shift + 7) / 8;
}
static void radix_passes(const uint32_t **keys, const uint32_t **vals, uint32_t *const k[2], uint32_t *const v[2],
                         uint64_t N, int first_shift, int key_bits, cudaStream_t s) {
    if (radix_pass_count(N, first_shift, key_bits) == 0) return;
    uint64_t tiles = (N + kRsTile - 1) / kRsTile;
    uint64_t G = std::min<uint64_t>(tiles, 148u * 8u);
    uint64_t chunk_tiles = (tiles + G - 1) / G;
    uint64_t chunk = chunk_tiles * kRsTile;
    G = (N + chunk - 1) / chunk;
    uint32_t *counts = dalloc<uint32_t>(256 * G + 1, s);  // + the scan's total
    int to = 0, left = radix_pass_count(N, first_shift, key_bits);
    for (int shift = first_shift, bits; shift < key_bits; shift += bits, to ^= 1, left--) {
        bits = (key_bits - shift + left - 1) / left;
        rs_upsweep<<<(unsigned)G, kThreads, 0, s>>>(*keys, N, chunk, shift, bits, counts, (uint32_t)G);
        exclusive_scan_u32(counts, counts, G << bits, s);  // in place: each tile is loaded before it is written
        (bits > 7 ? launch_downsweep<8> : launch_downsweep<7>)(G, *keys, *vals, k[to], v[to], N, chunk, shift, bits,
                                                               counts, s);
        PRG_CUDA(cudaGetLastError());
        *keys = k[to];
        *vals = v[to];
    }
    dfree(counts, s);
}

void radix_sort_pairs(uint32_t **keys, uint32_t **vals, uint32_t **keys_alt, uint32_t **vals_alt, uint64_t N,
                      int key_bits, cudaStream_t s) {
    uint32_t *const k[2] = {*keys_alt, *keys}, *const v[2] = {*vals_alt, *vals};
    const uint32_t *ks = *keys, *vs = *vals;
    radix_passes(&ks, &vs, k, v, N, 0, key_bits, s);
    if (ks != *keys) {
        std::swap(*keys, *keys_alt);
        std::swap(*vals, *vals_alt);
    }
}

// One stable pass on the 8-bit digit at `shift`: (keys, vals) -> (keys_out,
// vals_out).
static void radix_pass_pairs(uint32_t *keys, uint32_t *vals, uint32_t *keys_out, uint32_t *vals_out, uint64_t N,
                             int shift, cudaStream_t s) {
    if (N <= 1) {
        if (N == 1) {
            PRG_CUDA(cudaMemcpyAsync(keys_out, keys, 4, cudaMemcpyDeviceToDevice, s));
            PRG_CUDA(cudaMemcpyAsync(vals_out, vals, 4, cudaMemcpyDeviceToDevice, s));
        }
        return;
    }
    uint32_t *const k[2] = {keys_out, keys}, *const v[2] = {vals_out, vals};
    const uint32_t *ks = keys, *vs = vals;
    radix_passes(&ks, &vs, k, v, N, shift, shift + 8, s);
}

// ------------------------------------------------------------------ CSR

Tuning &tuning() {
    static Tuning t;
    return t;
}

__global__ void gather_f64_kernel(double *dst, const double *src, const uint32_t *idx, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[idx[i]];
}

void gather_f64(double *dst, const double *src, const uint32_t *idx, uint32_t n, cudaStream_t s) {
    gather_f64_kernel<<<grid_for(n, kThreads), kThreads, 0, s>>>(dst, src, idx, n);
    PRG_CUDA(cudaGetLastError());
}

void preload_gather_f64() {
    cudaFuncAttributes fa;
    PRG_CUDA(cudaFuncGetAttributes(&fa, gather_f64_kernel));
}

// ---- degree-sorted relabelling.  On skewed (power-law) graphs the vertices
// that are gathered most often are those with the largest out-degree; giving
// them the smallest internal ids packs the hot part of the rank vector into a
// few cache lines (L1/L2 hits instead of one sector per arc).  The order is
// out-degree descending, then caller id (stable sort); on directed graphs the
// vertices without in-arcs come after all others.  That puts the rows with
// arcs at ids 0 .. k-1, so a pass that walks arcs finds the row of its i-th
// row end at id i without an index, and a pass over the rows without arcs
// reads one contiguous range.  On power-law graphs it costs the hot prefix
// nothing: a vertex without in-arcs rarely has a large out-degree (none with
// out-degree >= 16 among the 2.2 M of R-MAT scale 22).

// One atomic per block: an atomic per warp to one word took 50 us at 4 M
// entries, ten times the read.
template <int THREADS>
__device__ __forceinline__ void block_atomic_max(uint32_t mx, uint32_t *out) {
    __shared__ uint32_t sh[THREADS / 32];
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < THREADS / 32; w++) mx = max(mx, sh[w]);
        atomicMax(out, mx);
    }
}

__global__ void __launch_bounds__(kThreads) max_u32_kernel(const uint32_t *a, uint32_t n, uint32_t *out) {
    uint32_t mx = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) mx = max(mx, a[v]);
    block_atomic_max<kThreads>(mx, out);
}

// noin: 1 for a vertex without in-arcs (null: out-degree alone); it is the
// key's most significant bit
__global__ void relabel_keys(const uint32_t *deg, const uint8_t *noin, uint32_t n, uint32_t maxdeg, int bits,
                             uint32_t *key, uint32_t *val) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        key[v] = noin ? (uint32_t)noin[v] << bits | (maxdeg - deg[v]) : maxdeg - deg[v];
        val[v] = v;
    }
}

__global__ void mark_empty_rows(const uint32_t *cnt, uint32_t n, uint8_t *noin) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        noin[v] = cnt[v] == 0u ? 1 : 0;
}

__global__ void relabel_finish(const uint32_t *perm, const uint32_t *deg_old, uint32_t n, uint32_t *iperm,
                               uint32_t *deg_new) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t o = perm[i];
        iperm[o] = i;
        deg_new[i] = deg_old[o];
    }
}

// Arc a of the in-CSR before sorting: key = destination row, value = source
// (unweighted) or arc id (weighted, to fetch the edge weight after the sort).
__global__ void make_arcs(const uint32_t *from, const uint32_t *to, uint64_t m, bool directed, bool carry_id,
                          uint32_t *key, uint32_t *val) {
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t u = from[e], v = to[e];
        if (directed) {
            key[e] = v;
            val[e] = carry_id ? (uint32_t)e : u;
        } else {
            // arc 2e: in_adj[u] += v ; arc 2e+1: in_adj[v] += u (self-loop: both v)
            key[2 * e] = u;
            val[2 * e] = carry_id ? (uint32_t)(2 * e) : v;
            key[2 * e + 1] = v;
            val[2 * e + 1] = carry_id ? (uint32_t)(2 * e + 1) : u;
        }
    }
}

// Out-degree by atomics.  Degree-heavy vertices usually have small ids (the
// generators, and any degree-sorted numbering, put them there); their counts
// are first gathered in a per-block shared-memory histogram so thousands of
// updates to one hub do not serialise on a single L2 address.
constexpr uint32_t kDegBins = 12224;  // 47.75 KB, the rest of 48 for the block maximum
constexpr int kDegThreads = 1024;

// The same pass finds the largest endpoint.
constexpr int kDegItems = 4;  // edges of a thread, loaded before any is used

__global__ void __launch_bounds__(kDegThreads) out_degree_kernel(const uint32_t *from, const uint32_t *to, uint64_t m,
                                                                 bool directed, uint32_t n, uint32_t *deg,
                                                                 uint32_t *max_endpoint) {
    __shared__ uint32_t bins[kDegBins];
    for (uint32_t i = threadIdx.x; i < kDegBins; i += kDegThreads) bins[i] = 0u;
    __syncthreads();
    uint32_t mx = 0u;
    auto add = [&](uint32_t v) {
        if (v >= n) return;  // out-of-range ids are reported through max_endpoint
        if (v < kDegBins) atomicAdd_block(&bins[v], 1u);
        else atomicAdd(&deg[v], 1u);
    };
    const uint64_t step = (uint64_t)gridDim.x * kDegThreads * kDegItems;
    for (uint64_t b = (uint64_t)blockIdx.x * kDegThreads * kDegItems + threadIdx.x; b < m; b += step) {
        uint32_t f[kDegItems], t[kDegItems];
#pragma unroll
        for (int j = 0; j < kDegItems; j++) {
            const uint64_t e = b + (uint64_t)j * kDegThreads;
            f[j] = e < m ? __ldcs(from + e) : 0u;
            t[j] = e < m ? __ldcs(to + e) : 0u;
        }
#pragma unroll
        for (int j = 0; j < kDegItems; j++) {
            mx = max(mx, max(f[j], t[j]));
            if (b + (uint64_t)j * kDegThreads < m) {
                add(f[j]);
                if (!directed) add(t[j]);
            }
        }
    }
    block_atomic_max<kDegThreads>(mx, max_endpoint);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kDegBins && i < n; i += kDegThreads)
        if (bins[i]) atomicAdd(&deg[i], bins[i]);
}

// Arcs per row of a CSR from its sorted row keys (cnt zeroed before): the
// first arc i of a row takes i off its count, the row's last arc adds i + 1.
// Work is one thread per arc however long the runs of rows without arcs are.
constexpr int kRunItems = 4;  // keys of a lane, loaded before any is used
__global__ void __launch_bounds__(kThreads) row_counts(const uint32_t *key, uint64_t N, uint32_t *cnt) {
    const uint64_t step = (uint64_t)gridDim.x * kThreads * kRunItems;
    const int lane = threadIdx.x & 31;
    // a warp's 128 keys; every lane of the warp takes the loop or none does
    for (uint64_t b = ((uint64_t)blockIdx.x * kThreads + (threadIdx.x & ~31u)) * kRunItems; b < N; b += step) {
        uint32_t k[kRunItems], before = 0u, after = 0u;
#pragma unroll
        for (int j = 0; j < kRunItems; j++) {
            const uint64_t i = b + 32 * j + lane;
            k[j] = i < N ? __ldg(key + i) : 0u;
        }
        if (lane == 0 && b > 0) before = __ldg(key + b - 1);
        if (lane == 31 && b + 32 * kRunItems < N) after = __ldg(key + b + 32 * kRunItems);
#pragma unroll
        for (int j = 0; j < kRunItems; j++) {
            const uint64_t i = b + 32 * j + lane;
            uint32_t prev = __shfl_up_sync(0xffffffffu, k[j], 1), next = __shfl_down_sync(0xffffffffu, k[j], 1);
            const uint32_t last = j > 0 ? __shfl_sync(0xffffffffu, k[j > 0 ? j - 1 : 0], 31) : before;
            const uint32_t first = j + 1 < kRunItems ? __shfl_sync(0xffffffffu, k[j + 1 < kRunItems ? j + 1 : 0], 0) : after;
            if (lane == 0) prev = last;
            if (lane == 31) next = first;
            if (i >= N) continue;
            const bool head = i == 0 || prev != k[j], tail = i + 1 == N || next != k[j];
            if (head || tail) atomicAdd(cnt + k[j], (tail ? (uint32_t)(i + 1) : 0u) - (head ? (uint32_t)i : 0u));
        }
    }
}
static void count_rows(const uint32_t *key, uint64_t N, uint32_t n, uint32_t *cnt, cudaStream_t s) {
    PRG_CUDA(cudaMemsetAsync(cnt, 0, std::max<uint64_t>(n, 1) * 4, s));
    if (N) row_counts<<<grid_for(N, kThreads * kRunItems), kThreads, 0, s>>>(key, N, cnt);
}

__global__ void gather_u32_kernel(uint32_t *dst, const uint32_t *src, const uint32_t *idx, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[idx[i]];
}

// How far a row's arcs move when the rows take their internal order (mod 2^32).
__global__ void row_shifts(const uint32_t *old_ptr, const uint32_t *row_ptr, const uint32_t *iperm, uint32_t n,
                           uint32_t *shift) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        shift[v] = row_ptr[iperm[v]] - old_ptr[v];
}

// The sorted arcs (row keys and sources, or arc ids for weighted graphs) to
// their places in the CSR: arc i of caller row k goes to i + shift[k], its
// source becomes an internal id (iperm null: neither changes).  One gather of
// iperm per arc bounds it.
template <bool WEIGHTED>
__global__ void __launch_bounds__(kThreads) place_rows(const uint32_t *key, const uint32_t *val, uint64_t arcs,
                                                       const uint32_t *shift, const uint32_t *iperm,
                                                       const uint32_t *from, const uint32_t *to, const double *w,
                                                       bool directed, uint32_t *col, double *w64, float *w32) {
    const uint64_t step = (uint64_t)gridDim.x * kThreads * kRunItems;
    for (uint64_t b = (uint64_t)blockIdx.x * kThreads * kRunItems + threadIdx.x; b < arcs; b += step) {
        uint32_t src[kRunItems], dst[kRunItems];
        double we[kRunItems];
#pragma unroll
        for (int j = 0; j < kRunItems; j++) {
            const uint64_t i = b + (uint64_t)j * kThreads;
            src[j] = dst[j] = 0u;
            if (i < arcs) {
                src[j] = __ldg(val + i);
                dst[j] = iperm ? __ldg(key + i) : 0u;
            }
        }
#pragma unroll
        for (int j = 0; j < kRunItems; j++) {
            const uint64_t i = b + (uint64_t)j * kThreads;
            if (i < arcs) {
                if (WEIGHTED) {
                    const uint32_t a = src[j];
                    const uint64_t e = directed ? a : a >> 1;
                    src[j] = directed || (a & 1u) ? __ldg(from + e) : __ldg(to + e);
                    we[j] = __ldg(w + e);
                }
                if (iperm) dst[j] = __ldg(shift + dst[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < kRunItems; j++)
            if (iperm && b + (uint64_t)j * kThreads < arcs) src[j] = __ldg(iperm + src[j]);
#pragma unroll
        for (int j = 0; j < kRunItems; j++) {
            const uint64_t i = b + (uint64_t)j * kThreads;
            if (i >= arcs) continue;
            const uint32_t p = (uint32_t)i + dst[j];
            col[p] = src[j];
            if (WEIGHTED) {
                w64[p] = we[j];
                w32[p] = (float)we[j];
            }
        }
    }
}

// Segmented row sums of per-arc weights (one warp per row, fixed tree); row r
// goes to out[at[r]] (at null: out[r]).
__global__ void row_weight_sums(const uint32_t *ptr, const double *wv, const uint32_t *perm, uint32_t nrows,
                                const uint32_t *at, double *outsum) {
    uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t lane = threadIdx.x & 31;
    uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = warp; r < nrows; r += nw) {
        double acc = 0.0;
        for (uint32_t p = ptr[r] + lane; p < ptr[r + 1]; p += 32) acc += perm ? wv[perm[p]] : wv[p];
        acc = warp_sum(acc);
        if (lane == 0) outsum[at ? at[r] : r] = acc;
    }
}

__global__ void finish_degrees(uint32_t n, const uint32_t *deg, double *strength_io, bool weighted, double *dval,
                               float *inv32, uint32_t *n_dangling) {
    uint32_t cnt = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        double d = weighted ? strength_io[v] : (double)deg[v];
        dval[v] = d;
        inv32[v] = d > 0.0 ? (float)(1.0 / d) : 0.0f;
        cnt += d == 0.0 ? 1u : 0u;
    }
    __shared__ uint32_t sh[32];
    cnt = block_sum<uint32_t>(cnt, sh);
    if (threadIdx.x == 0 && cnt) atomicAdd(n_dangling, cnt);
}

__global__ void __launch_bounds__(kThreads) max_degree_kernel(const uint32_t *row_ptr, uint32_t n, uint32_t *out) {
    uint32_t mx = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        mx = max(mx, row_ptr[v + 1] - row_ptr[v]);
    block_atomic_max<kThreads>(mx, out);
}

// ------------------------------------------------------------------ row-blocks
//
// Row-blocks are the work units of one warp of the iteration kernel.  A row
// is "short" (deg <= shortmax), "long" (shortmax < deg <= split: one warp
// streams it) or a hub (deg > split: ceil(deg/split) chunk row-blocks whose
// partial sums are combined by the last chunk to finish).  A run of short
// rows forms a stream row-block; a new one starts at row r when r is a
// multiple of 32, when the previous row was not short, or when row r's first
// arc crosses a multiple of capw.  A stream block therefore holds <= 32 rows
// (32-row aligned, so its epilogue stores are coalesced) and
// < capw + shortmax <= kWarpBuf arcs; the kernel sums each of its rows with a
// power-of-two group of lanes sized to the row count.

__global__ void rb_count(const uint32_t *rp, uint32_t n, uint32_t capw, uint32_t shortmax, uint32_t split,
                         uint32_t *cnt, uint32_t *hubflag) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t deg = rp[r + 1] - rp[r];
        uint32_t c, h = 0;
        if (deg > split) {
            c = (deg + split - 1) / split;
            h = 1;
        } else if (deg > shortmax) {
            c = 1;
        } else {
            bool start = (r % kRowCap == 0);
            if (!start) {
                const uint32_t pdeg = rp[r] - rp[r - 1];
                start = (pdeg > shortmax) || (rp[r] / capw != rp[r - 1] / capw);
            }
            c = start ? 1u : 0u;
        }
        cnt[r] = c;
        hubflag[r] = h;
    }
}

__global__ void rb_fill(const uint32_t *rp, uint32_t n, uint32_t shortmax, uint32_t split, const uint32_t *off,
                        const uint32_t *hoff, uint4 *rb, Hub *hubs) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t k = off[r], c = off[r + 1] - k;
        if (c == 0) continue;
        const uint32_t p0 = rp[r], p1 = rp[r + 1], deg = p1 - p0;
        if (deg > split) {
            const uint32_t h = hoff[r];
            hubs[h] = Hub{r, c, k, 0};
            for (uint32_t j = 0; j < c; j++) {
                const uint32_t lo = p0 + j * split, hi = min(p1, lo + split);
                rb[k + j] = make_uint4(r, kChunkFlag | h, lo, hi);
            }
        } else if (deg > shortmax) {
            rb[k] = make_uint4(r, r + 1, p0, p1);
        } else {
            rb[k] = make_uint4(r, 0, p0, 0);  // end filled by rb_fix
        }
    }
}

__global__ void rb_fix(const uint32_t *rp, uint4 *rb, uint32_t nrb, uint32_t n) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nrb; k += gridDim.x * blockDim.x) {
        uint4 d = rb[k];
        if (d.y == 0u) {  // stream row-block: runs to the next row-block's first row
            d.y = (k + 1 < nrb) ? rb[k + 1].x : n;
            d.w = rp[d.y];
            rb[k] = d;
        }
    }
}

void build_row_blocks(DeviceGraph &g, uint32_t capw, uint32_t shortmax, uint32_t split, cudaStream_t s) {
    // a stream row-block holds < capw + shortmax arcs, which must fit the warp buffer
    shortmax = std::max<uint32_t>(1u, std::min<uint32_t>(shortmax, kWarpBuf / 2));
    capw = std::max<uint32_t>(32u, std::min<uint32_t>(capw, kWarpBuf - shortmax));
    split = std::max<uint32_t>(split, std::max<uint32_t>(shortmax, 256u));
    const uint32_t n = g.n;
    if (g.rb) cudaFreeAsync(g.rb, s);
    if (g.hubs) cudaFreeAsync(g.hubs, s);
    g.rb = nullptr;
    g.hubs = nullptr;
    uint32_t *cnt = dalloc<uint32_t>(n + 1, s), *off = dalloc<uint32_t>(n + 1, s);
    uint32_t *hf = dalloc<uint32_t>(n + 1, s), *hoff = dalloc<uint32_t>(n + 1, s);
    const unsigned gb = grid_for(n, kThreads);
    rb_count<<<gb, kThreads, 0, s>>>(g.row_ptr, n, capw, shortmax, split, cnt, hf);
    exclusive_scan_u32(cnt, off, n, s);
    exclusive_scan_u32(hf, hoff, n, s);
    uint32_t hv[2];
    PRG_CUDA(cudaMemcpyAsync(&hv[0], off + n, 4, cudaMemcpyDeviceToHost, s));
    PRG_CUDA(cudaMemcpyAsync(&hv[1], hoff + n, 4, cudaMemcpyDeviceToHost, s));
    PRG_CUDA(cudaStreamSynchronize(s));
    g.nrb = hv[0];
    g.nhub = hv[1];
    g.rb = dalloc<uint4>(g.nrb, s);
    Scratch::forget(g.rb);
    g.hubs = dalloc<Hub>(g.nhub, s);
    Scratch::forget(g.hubs);
    rb_fill<<<gb, kThreads, 0, s>>>(g.row_ptr, n, shortmax, split, off, hoff, g.rb, g.hubs);
    rb_fix<<<grid_for(g.nrb, kThreads), kThreads, 0, s>>>(g.row_ptr, g.rb, g.nrb, n);
    PRG_CUDA(cudaGetLastError());
    dfree(cnt, s);
    dfree(off, s);
    dfree(hf, s);
    dfree(hoff, s);
    g.capw = capw;
    g.shortmax = shortmax;
    g.split = split;
}

static int bits_for(uint32_t maxkey) {
    int b = 0;
    while (b < 32 && (maxkey >> b) != 0) b++;
    return b;
}

// Divisors, dangling count, maximum in-degree and row-blocks of a graph whose
// row_ptr / col (/ weights) and deg are built; strength (weighted graphs, n
// entries, freed here) holds the out-strengths.
static void finish_graph(DeviceGraph &g, double *&strength, cudaStream_t s) {
    const uint32_t n = g.n;
    const unsigned gr = grid_for(n, kThreads, 148u * 8u);  // one atomic per block
    PRG_CUDA(cudaMallocAsync((void **)&g.dval, std::max<uint64_t>(n, 1) * 8, s));
    PRG_CUDA(cudaMallocAsync((void **)&g.inv32, std::max<uint64_t>(n, 1) * 4, s));
    uint32_t *d_nd = dalloc<uint32_t>(2, s);
    PRG_CUDA(cudaMemsetAsync(d_nd, 0, 8, s));
    finish_degrees<<<gr, kThreads, 0, s>>>(n, g.deg, strength, g.weighted, g.dval, g.inv32, d_nd);
    max_degree_kernel<<<gr, kThreads, 0, s>>>(g.row_ptr, n, d_nd + 1);
    PRG_CUDA(cudaGetLastError());
    uint32_t hnd[2];
    PRG_CUDA(cudaMemcpyAsync(hnd, d_nd, 8, cudaMemcpyDeviceToHost, s));
    dfree(strength, s);
    dfree(d_nd, s);
    PRG_CUDA(cudaStreamSynchronize(s));
    g.n_dangling = hnd[0];
    g.max_in_degree = hnd[1];
    build_row_blocks(g, g.capw, g.shortmax, g.split, s);
}

// Degree-sorted relabelling of the vertices when g.relabel asks for it (1) or
// the degree distribution is skewed (2: max degree >= 32 x mean, n >= 4096):
// g.perm (new -> old), g.iperm (old -> new) and g.deg in new ids.  Needs
// g.deg (out-degree), g.arcs and the in-degrees in caller ids (in_cnt).
// Returns whether it relabelled.
static bool relabel_vertices(DeviceGraph &g, cudaStream_t s, const uint32_t *in_cnt) {
    const uint32_t n = g.n;
    if (n < 2 || g.relabel == 0) return false;
    const unsigned gn = grid_for(n, kThreads);
    uint32_t *d_mx = dalloc<uint32_t>(1, s), maxdeg = 0;
    PRG_CUDA(cudaMemsetAsync(d_mx, 0, 4, s));
    max_u32_kernel<<<std::min(gn, 148u * 8u), kThreads, 0, s>>>(g.deg, n, d_mx);
    PRG_CUDA(cudaMemcpyAsync(&maxdeg, d_mx, 4, cudaMemcpyDeviceToHost, s));
    PRG_CUDA(cudaStreamSynchronize(s));
    dfree(d_mx, s);
    const double mean = (double)g.arcs / (double)n;
    const bool skewed = n >= 4096 && (double)maxdeg >= 32.0 * (mean > 1.0 ? mean : 1.0);
    if (g.relabel != 1 && !skewed) return false;
    uint32_t *pk = dalloc<uint32_t>(n, s), *pv = dalloc<uint32_t>(n, s);
    uint32_t *pk1 = dalloc<uint32_t>(n, s), *pv1 = dalloc<uint32_t>(n, s);
    // the no-in-arc bit: directed graphs whose key still fits 32 bits with it
    uint8_t *noin = nullptr;
    if (g.directed && bits_for(maxdeg) < 32) {
        noin = dalloc<uint8_t>(n, s);
        mark_empty_rows<<<gn, kThreads, 0, s>>>(in_cnt, n, noin);
    }
    relabel_keys<<<gn, kThreads, 0, s>>>(g.deg, noin, n, maxdeg, bits_for(maxdeg), pk, pv);
    radix_sort_pairs(&pk, &pv, &pk1, &pv1, n, bits_for(maxdeg) + (noin ? 1 : 0), s);
    dfree(noin, s);
    PRG_CUDA(cudaMallocAsync((void **)&g.perm, (uint64_t)n * 4, s));
    PRG_CUDA(cudaMallocAsync((void **)&g.iperm, (uint64_t)n * 4, s));
    PRG_CUDA(cudaMemcpyAsync(g.perm, pv, (uint64_t)n * 4, cudaMemcpyDeviceToDevice, s));
    uint32_t *deg_new = dalloc<uint32_t>(n, s);
    relabel_finish<<<gn, kThreads, 0, s>>>(g.perm, g.deg, n, g.iperm, deg_new);
    cudaFreeAsync(g.deg, s);
    g.deg = deg_new;
    Scratch::forget(g.deg);
    dfree(pk, s);
    dfree(pv, s);
    dfree(pk1, s);
    dfree(pv1, s);
    return true;
}

bool build_graph(DeviceGraph &g, const uint32_t *d_from, const uint32_t *d_to, const double *d_w, cudaStream_t s,
                 uint32_t *max_endpoint) {
    Scratch scratch(s);
    cudaEvent_t e0, e1;
    PRG_CUDA(cudaEventCreate(&e0));
    PRG_CUDA(cudaEventCreate(&e1));
    PRG_CUDA(cudaEventRecord(e0, s));
    const uint32_t n = g.n;
    const uint64_t m = g.m;
    const bool directed = g.directed, weighted = d_w != nullptr;
    g.weighted = weighted;
    const uint64_t arcs = directed ? m : 2 * m;
    g.arcs = arcs;
    const unsigned ge = grid_for(m, kThreads), gn = grid_for(n, kThreads);
    const int key_bits = bits_for(n ? n - 1 : 0);
    const uint64_t padded = arcs + kColPad;

    // out-degree (unweighted divisor; also kept for weighted graphs)
    PRG_CUDA(cudaMallocAsync((void **)&g.deg, std::max<uint64_t>(n, 1) * 4, s));
    PRG_CUDA(cudaMemsetAsync(g.deg, 0, std::max<uint64_t>(n, 1) * 4, s));
    *max_endpoint = 0;
    if (m) {
        uint32_t *d_mx = dalloc<uint32_t>(1, s);
        PRG_CUDA(cudaMemsetAsync(d_mx, 0, 4, s));
        out_degree_kernel<<<148 * 2, kDegThreads, 0, s>>>(d_from, d_to, m, directed, n, g.deg, d_mx);
        PRG_CUDA(cudaGetLastError());
        PRG_CUDA(cudaMemcpyAsync(max_endpoint, d_mx, 4, cudaMemcpyDeviceToHost, s));
        dfree(d_mx, s);
        PRG_CUDA(cudaStreamSynchronize(s));
        if (*max_endpoint >= n) {  // nothing below runs on ids out of range
            dfree(g.deg, s);
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return false;
        }
    }

    // Arcs in edge order, stably sorted by destination, in caller ids: a
    // directed unweighted edge list is sorted as it is.  Relabelling afterwards
    // (rows moved as runs, one gather of the new source id per arc) costs half
    // the gathers that relabelled edges would, and the row lengths tell which
    // vertices have no in-arcs.  R-MAT scale 22 (4 M vertices, 67 M arcs): edges
    // relabelled first, heads flagged, arcs and row ends from them 1.50 ms;
    // sorted first, rows counted and moved 0.41 ms.
    const bool as_is = directed && !weighted;
    const int passes = radix_pass_count(arcs, 0, key_bits);
    uint32_t *k[2] = {nullptr, nullptr}, *v[2] = {nullptr, nullptr};
    for (int i = 0; i < 2; i++) {
        if (i == 1 && as_is && passes < 2) break;
        k[i] = dalloc<uint32_t>(arcs, s);
        v[i] = dalloc<uint32_t>(padded, s);
    }
    const uint32_t *ks = d_to, *vs = d_from;
    if (!as_is) {
        if (m) make_arcs<<<ge, kThreads, 0, s>>>(d_from, d_to, m, directed, weighted, k[1], v[1]);
        ks = k[1];
        vs = v[1];
    }
    radix_passes(&ks, &vs, k, v, arcs, 0, key_bits, s);

    uint32_t *cnt = dalloc<uint32_t>(n, s);
    count_rows(ks, arcs, n, cnt, s);
    PRG_CUDA(cudaGetLastError());

    // optional degree-sorted relabelling (internal ids)
    PRG_CUDA(cudaMallocAsync((void **)&g.row_ptr, (uint64_t)(n + 1) * 4, s));
    const bool relabelled = relabel_vertices(g, s, cnt);
    uint32_t *shift = nullptr;
    if (relabelled) {
        uint32_t *rows = dalloc<uint32_t>(n + 1, s);
        shift = dalloc<uint32_t>(n, s);
        gather_u32_kernel<<<gn, kThreads, 0, s>>>(rows, cnt, g.perm, n);
        exclusive_scan_u32(rows, g.row_ptr, n, s);
        exclusive_scan_u32(cnt, rows, n, s);  // the rows' places in caller order
        row_shifts<<<gn, kThreads, 0, s>>>(rows, g.row_ptr, g.iperm, n, shift);
        dfree(rows, s);
    } else {
        exclusive_scan_u32(cnt, g.row_ptr, n, s);
    }
    dfree(cnt, s);

    double *strength = nullptr;
    if (!weighted && !relabelled && vs != d_from) {
        g.col = v[vs == v[1]];  // in place
        Scratch::forget(g.col);
        v[vs == v[1]] = nullptr;
    } else {
        PRG_CUDA(cudaMallocAsync((void **)&g.col, padded * 4, s));
        if (weighted) {
            PRG_CUDA(cudaMallocAsync((void **)&g.w64, padded * 8, s));
            PRG_CUDA(cudaMallocAsync((void **)&g.w32, padded * 4, s));
            PRG_CUDA(cudaMemsetAsync(g.w64 + arcs, 0, kColPad * 8, s));
            PRG_CUDA(cudaMemsetAsync(g.w32 + arcs, 0, kColPad * 4, s));
        }
        const unsigned gp = grid_for(arcs, kThreads * kRunItems);
        if (arcs && weighted)
            place_rows<true><<<gp, kThreads, 0, s>>>(ks, vs, arcs, shift, g.iperm, d_from, d_to, d_w, directed, g.col,
                                                     g.w64, g.w32);
        else if (arcs)
            place_rows<false><<<gp, kThreads, 0, s>>>(ks, vs, arcs, shift, g.iperm, d_from, d_to, d_w, directed, g.col,
                                                      nullptr, nullptr);
    }
    PRG_CUDA(cudaMemsetAsync(g.col + arcs, 0, kColPad * 4, s));
    PRG_CUDA(cudaGetLastError());
    if (weighted) {
        strength = dalloc<double>(n, s);
        if (!directed) {
            // undirected: arcs out of u are exactly the arcs into u (same weights)
            row_weight_sums<<<grid_for((uint64_t)n * 32, kThreads), kThreads, 0, s>>>(g.row_ptr, g.w64, nullptr, n,
                                                                                   nullptr, strength);
        } else {
            // directed: group edge ids by source with a second stable sort
            uint32_t *ocnt = dalloc<uint32_t>(n, s), *optr = dalloc<uint32_t>(n + 1, s);
            if (m) make_arcs<<<ge, kThreads, 0, s>>>(d_to, d_from, m, true, true, k[1], v[1]);  // (source, edge id)
            const uint32_t *sk = k[1], *sv = v[1];
            radix_passes(&sk, &sv, k, v, m, 0, key_bits, s);
            count_rows(sk, m, n, ocnt, s);
            exclusive_scan_u32(ocnt, optr, n, s);
            row_weight_sums<<<grid_for((uint64_t)n * 32, kThreads), kThreads, 0, s>>>(optr, d_w, sv, n, g.iperm,
                                                                                   strength);
            dfree(ocnt, s);
            dfree(optr, s);
        }
    }
    dfree(shift, s);
    for (int i = 0; i < 2; i++) {
        dfree(k[i], s);
        dfree(v[i], s);
    }

    finish_graph(g, strength, s);
    PRG_CUDA(cudaEventRecord(e1, s));
    PRG_CUDA(cudaEventSynchronize(e1));
    PRG_CUDA(cudaEventElapsedTime(&g.build_ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return true;
}

// ------------------------------------------------------------------ streamed build from host edges
//
// The edge list arrives in chunks (host -> device copies on a side stream);
// each chunk is processed while the next one is in flight.  An arc's final
// CSR position is
//     row_ptr[dst] + (arcs into dst in earlier chunks) + (rank among the
//                                                          chunk's arcs into dst)
// and only row_ptr needs the whole list.  So every chunk is stably sorted by
// destination on arrival, its ranks are added to the running per-destination
// counts (off[arc], cnt[dst]), and after the last chunk one scan of the
// counts and one scatter place every arc.  Within a row the arcs keep their
// arc order, exactly as the sort of the whole list in build_graph leaves
// them, so both builds produce the same CSR.

// Start of each destination's run in the sorted chunk: base = cnt - i.
__global__ void chunk_ranks_begin(const uint32_t *keys, uint64_t N, uint32_t n, const uint32_t *cnt, uint32_t *base) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t k = keys[i];
        if (k < n && (i == 0 || keys[i - 1] != k)) base[k] = cnt[k] - (uint32_t)i;
    }
}

// off[arc] = arcs into its destination before it; the run's last arc
// advances cnt.  (u32 arithmetic: base + i is the true count.)
__global__ void chunk_ranks_end(const uint32_t *keys, const uint32_t *vals, uint64_t N, uint32_t n,
                                const uint32_t *base, uint32_t *cnt, uint32_t *off) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t k = keys[i];
        if (k >= n) continue;
        const uint32_t b = base[k];
        off[vals[i]] = b + (uint32_t)i;
        if (i + 1 == N || keys[i + 1] != k) cnt[k] = b + (uint32_t)i + 1u;
    }
}

// The arcs' final positions, row_ptr[dst] + off[arc], are a permutation of
// [0, arcs).  Writing each arc straight to its position would be one random
// 4-byte HBM write per arc.  Instead: (1) arc_positions writes (position,
// value) pairs in arc order; (2) one stable radix pass on the position's top
// 8 bits groups them into 256 windows of consecutive positions; (3)
// place_arcs writes each window while its slice of col sits in L2.
// value = the relabelled source (unweighted) or the arc id (weighted: the
// source and the edge weight are fetched when placing).
__global__ void arc_positions(const uint32_t *from, const uint32_t *to, uint64_t arcs, bool directed, bool weighted,
                              const uint32_t *iperm, const uint32_t *row_ptr, const uint32_t *off, uint32_t *pos,
                              uint32_t *val) {
    for (uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; a < arcs;
         a += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t e = directed ? a : (a >> 1);
        uint32_t dst = to[e], src = from[e];
        if (!directed && (a & 1u) == 0u) {
            dst = from[e];
            src = to[e];
        }
        if (iperm) {
            dst = iperm[dst];
            src = iperm[src];
        }
        pos[a] = row_ptr[dst] + off[a];
        val[a] = weighted ? (uint32_t)a : src;
    }
}

__global__ void place_arcs(const uint32_t *pos, const uint32_t *val, uint64_t arcs, bool directed,
                           const uint32_t *from, const uint32_t *to, const double *w, const uint32_t *iperm,
                           uint32_t *col, double *w64, float *w32) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < arcs; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t p = pos[i];
        if (p >= arcs) continue;  // never for a consistent build
        if (!w) {
            col[p] = val[i];
            continue;
        }
        const uint32_t a = val[i];
        const uint64_t e = directed ? a : (a >> 1);
        uint32_t src = (directed || (a & 1u)) ? from[e] : to[e];
        if (iperm) src = iperm[src];
        col[p] = src;
        const double we = w[e];
        w64[p] = we;
        w32[p] = (float)we;
    }
}

bool build_graph_host(DeviceGraph &g, const uint32_t *h_from, const uint32_t *h_to, const double *h_w, cudaStream_t s,
                      uint32_t *max_endpoint, DeviceEdges *keep) {
    Scratch scratch(s);
    cudaEvent_t e0, e1;
    PRG_CUDA(cudaEventCreate(&e0));
    PRG_CUDA(cudaEventCreate(&e1));
    PRG_CUDA(cudaEventRecord(e0, s));
    const uint32_t n = g.n;
    const uint64_t m = g.m;
    const bool directed = g.directed, weighted = h_w != nullptr;
    g.weighted = weighted;
    const uint64_t arcs = directed ? m : 2 * m;
    g.arcs = arcs;
    const uint64_t chunk = std::max<uint64_t>(kStreamChunkMin, (m + kStreamChunks - 1) / kStreamChunks);
    const uint64_t nchunks = (m + chunk - 1) / chunk;
    const uint64_t chunk_arcs = directed ? chunk : 2 * chunk;
    const int key_bits = bits_for(n ? n - 1 : 0);

    uint32_t *d_from = dalloc<uint32_t>(m, s), *d_to = dalloc<uint32_t>(m, s);
    double *d_w = weighted ? dalloc<double>(m, s) : nullptr;
    PRG_CUDA(cudaMallocAsync((void **)&g.deg, std::max<uint64_t>(n, 1) * 4, s));
    PRG_CUDA(cudaMemsetAsync(g.deg, 0, std::max<uint64_t>(n, 1) * 4, s));
    uint32_t *cnt = dalloc<uint32_t>(n, s), *base = dalloc<uint32_t>(n, s), *off = dalloc<uint32_t>(arcs, s);
    PRG_CUDA(cudaMemsetAsync(cnt, 0, std::max<uint64_t>(n, 1) * 4, s));
    uint32_t *d_mx = dalloc<uint32_t>(1, s);
    PRG_CUDA(cudaMemsetAsync(d_mx, 0, 4, s));
    uint32_t *ka = dalloc<uint32_t>(chunk_arcs, s), *va = dalloc<uint32_t>(chunk_arcs, s);
    uint32_t *kb = dalloc<uint32_t>(chunk_arcs, s), *vb = dalloc<uint32_t>(chunk_arcs, s);

    struct CopyStream {
        cudaStream_t s = stream_acquire();
        ~CopyStream() { release(); }
        void release() {  // waits for the copies
            if (s) stream_release(s);
            s = nullptr;
        }
    } copies;
    const cudaStream_t cs = copies.s;
    std::vector<cudaEvent_t> ev(nchunks + 1);
    for (cudaEvent_t &e : ev) PRG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    // the copy stream starts once the allocations above are usable
    PRG_CUDA(cudaEventRecord(ev[nchunks], s));
    PRG_CUDA(cudaStreamWaitEvent(cs, ev[nchunks], 0));
    for (uint64_t c = 0; c < nchunks; c++) {
        const uint64_t b = c * chunk, len = std::min(chunk, m - b);
        const uint64_t a0 = directed ? b : 2 * b, la = directed ? len : 2 * len;
        PRG_CUDA(cudaMemcpyAsync(d_from + b, h_from + b, len * 4, cudaMemcpyHostToDevice, cs));
        PRG_CUDA(cudaMemcpyAsync(d_to + b, h_to + b, len * 4, cudaMemcpyHostToDevice, cs));
        if (weighted) PRG_CUDA(cudaMemcpyAsync(d_w + b, h_w + b, len * 8, cudaMemcpyHostToDevice, cs));
        PRG_CUDA(cudaEventRecord(ev[c], cs));
        PRG_CUDA(cudaStreamWaitEvent(s, ev[c], 0));
        const unsigned gl = grid_for(len, kThreads), gla = grid_for(la, kThreads);
        out_degree_kernel<<<148 * 2, kDegThreads, 0, s>>>(d_from + b, d_to + b, len, directed, n, g.deg, d_mx);
        make_arcs<<<gl, kThreads, 0, s>>>(d_from + b, d_to + b, len, directed, true, ka, va);
        uint32_t *k0 = ka, *v0 = va, *k1 = kb, *v1 = vb;
        radix_sort_pairs(&k0, &v0, &k1, &v1, la, key_bits, s);
        chunk_ranks_begin<<<gla, kThreads, 0, s>>>(k0, la, n, cnt, base);
        chunk_ranks_end<<<gla, kThreads, 0, s>>>(k0, v0, la, n, base, cnt, off + a0);
        PRG_CUDA(cudaGetLastError());
    }
    const bool trace = std::getenv("PRG_TRACE") != nullptr;
    cudaEvent_t t_copy = nullptr, t_loop = nullptr, t_tail[4] = {};
    if (trace) {
        PRG_CUDA(cudaEventCreate(&t_copy));
        PRG_CUDA(cudaEventCreate(&t_loop));
        for (cudaEvent_t &e : t_tail) PRG_CUDA(cudaEventCreate(&e));
        PRG_CUDA(cudaEventRecord(t_copy, cs));
        PRG_CUDA(cudaEventRecord(t_loop, s));
    }
    uint32_t mx = 0;
    PRG_CUDA(cudaMemcpyAsync(&mx, d_mx, 4, cudaMemcpyDeviceToHost, s));
    PRG_CUDA(cudaStreamSynchronize(s));
    for (cudaEvent_t &e : ev) cudaEventDestroy(e);
    copies.release();
    dfree(ka, s);
    dfree(va, s);
    dfree(kb, s);
    dfree(vb, s);
    dfree(d_mx, s);
    *max_endpoint = mx;
    if (m > 0 && mx >= n) {
        dfree(d_from, s);
        dfree(d_to, s);
        dfree(d_w, s);
        dfree(cnt, s);
        dfree(base, s);
        dfree(off, s);
        if (trace) {
            cudaEventDestroy(t_copy);
            cudaEventDestroy(t_loop);
            for (cudaEvent_t &e : t_tail) cudaEventDestroy(e);
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        return false;
    }

    const unsigned gn = grid_for(n, kThreads), ga = grid_for(arcs, kThreads);
    const bool relabelled = relabel_vertices(g, s, cnt);
    if (trace) PRG_CUDA(cudaEventRecord(t_tail[0], s));
    uint32_t *rows = cnt;
    if (relabelled) {
        gather_u32_kernel<<<gn, kThreads, 0, s>>>(base, cnt, g.perm, n);  // base is free now
        rows = base;
    }
    PRG_CUDA(cudaMallocAsync((void **)&g.row_ptr, (uint64_t)(n + 1) * 4, s));
    exclusive_scan_u32(rows, g.row_ptr, n, s);
    const uint64_t padded = arcs + kColPad;
    PRG_CUDA(cudaMallocAsync((void **)&g.col, padded * 4, s));
    PRG_CUDA(cudaMemsetAsync(g.col, 0, padded * 4, s));
    if (weighted) {
        PRG_CUDA(cudaMallocAsync((void **)&g.w64, padded * 8, s));
        PRG_CUDA(cudaMallocAsync((void **)&g.w32, padded * 4, s));
        PRG_CUDA(cudaMemsetAsync(g.w64, 0, padded * 8, s));
        PRG_CUDA(cudaMemsetAsync(g.w32, 0, padded * 4, s));
    }
    if (trace) PRG_CUDA(cudaEventRecord(t_tail[1], s));
    if (arcs) {
        const uint32_t *ip = relabelled ? g.iperm : nullptr;
        uint32_t *pk = dalloc<uint32_t>(arcs, s), *pv = dalloc<uint32_t>(arcs, s);
        uint32_t *pk1 = dalloc<uint32_t>(arcs, s), *pv1 = dalloc<uint32_t>(arcs, s);
        arc_positions<<<ga, kThreads, 0, s>>>(d_from, d_to, arcs, directed, weighted, ip, g.row_ptr, off, pk, pv);
        const int pbits = bits_for((uint32_t)(arcs - 1));
        radix_pass_pairs(pk, pv, pk1, pv1, arcs, std::max(0, pbits - 8), s);
        place_arcs<<<ga, kThreads, 0, s>>>(pk1, pv1, arcs, directed, d_from, d_to, d_w, ip, g.col, g.w64, g.w32);
        dfree(pk, s);
        dfree(pv, s);
        dfree(pk1, s);
        dfree(pv1, s);
    }
    PRG_CUDA(cudaGetLastError());
    if (trace) PRG_CUDA(cudaEventRecord(t_tail[2], s));
    double *strength = nullptr;
    if (weighted) {
        // undirected only: arcs out of u are exactly the arcs into u (same weights)
        strength = dalloc<double>(n, s);
        row_weight_sums<<<grid_for((uint64_t)n * 32, kThreads), kThreads, 0, s>>>(g.row_ptr, g.w64, nullptr, n,
                                                                               nullptr, strength);
    }
    if (keep) {
        *keep = DeviceEdges{d_from, d_to};
        Scratch::forget(d_from);
        Scratch::forget(d_to);
    } else {
        dfree(d_from, s);
        dfree(d_to, s);
    }
    dfree(d_w, s);
    dfree(cnt, s);
    dfree(base, s);
    dfree(off, s);
    finish_graph(g, strength, s);
    PRG_CUDA(cudaEventRecord(e1, s));
    PRG_CUDA(cudaEventSynchronize(e1));
    PRG_CUDA(cudaEventElapsedTime(&g.build_ms, e0, e1));
    if (trace) {
        float c = 0, l = 0, r = 0, sc = 0, sca = 0;
        cudaEventElapsedTime(&c, e0, t_copy);
        cudaEventElapsedTime(&l, e0, t_loop);
        cudaEventElapsedTime(&r, t_loop, t_tail[0]);
        cudaEventElapsedTime(&sc, t_tail[0], t_tail[1]);
        cudaEventElapsedTime(&sca, t_tail[1], t_tail[2]);
        std::fprintf(stderr,
                     "[prg] streamed build: %llu chunks, copies done %.2f ms, chunk work done %.2f ms, relabel %.2f, "
                     "scan+alloc %.2f, scatter %.2f, finish %.2f, total %.2f ms\n",
                     (unsigned long long)nchunks, c, l, r, sc, sca, g.build_ms - l - r - sc - sca, g.build_ms);
        cudaEventDestroy(t_copy);
        cudaEventDestroy(t_loop);
        for (cudaEvent_t &e : t_tail) cudaEventDestroy(e);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return true;
}

void free_graph(DeviceGraph &g) {
    cudaFree(g.row_ptr);
    cudaFree(g.col);
    cudaFree(g.w64);
    cudaFree(g.w32);
    cudaFree(g.deg);
    cudaFree(g.dval);
    cudaFree(g.inv32);
    cudaFree(g.rb);
    cudaFree(g.hubs);
    cudaFree(g.perm);
    cudaFree(g.iperm);
    g = DeviceGraph{};
}

// ------------------------------------------------------------------ R-MAT

// Counter-based R-MAT: edge e draws `scale` uniforms from its own SplitMix64
// stream seeded with seed ^ (e * 0xD1B54A32D192ED03).  Bit-identical to the
// CPU generator used by the tests (same integer mixing, same double compare).
__global__ void rmat_kernel(uint32_t scale, uint64_t m, double t1, double t2, double t3, uint64_t seed,
                            uint32_t *from, uint32_t *to) {
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t st = seed ^ (e * 0xD1B54A32D192ED03ULL);
        uint32_t u = 0, v = 0;
        for (uint32_t l = 0; l < scale; l++) {
            st += 0x9E3779B97F4A7C15ULL;
            uint64_t z = st;
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
            z ^= z >> 31;
            double x = (double)(z >> 11) * (1.0 / 9007199254740992.0);
            uint32_t rb, cb;
            if (x < t1) { rb = 0; cb = 0; }
            else if (x < t2) { rb = 0; cb = 1; }
            else if (x < t3) { rb = 1; cb = 0; }
            else { rb = 1; cb = 1; }
            u = (u << 1) | rb;
            v = (v << 1) | cb;
        }
        from[e] = u;
        to[e] = v;
    }
}

void rmat_generate(uint32_t scale, uint64_t m, double a, double b, double c, uint64_t seed, uint32_t *d_from,
                   uint32_t *d_to, cudaStream_t s) {
    double t1 = a, t2 = a + b, t3 = a + b + c;
    rmat_kernel<<<grid_for(m, kThreads, 148u * 32u), kThreads, 0, s>>>(scale, m, t1, t2, t3, seed, d_from, d_to);
    PRG_CUDA(cudaGetLastError());
}

}  // namespace prg

namespace prg {

// ---- further seeded generators (training graphs for the warm start) ------
// Counter-based like the R-MAT generator: edge e draws from its own
// SplitMix64 stream seeded with seed ^ (e * 0xD1B54A32D192ED03).

__device__ __forceinline__ double sm_unit(uint64_t &st) {
    st += 0x9E3779B97F4A7C15ULL;
    uint64_t z = st;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// Chung-Lu power law: both endpoints drawn with probability proportional to
// (i + i0)^(-alpha) by inverting the continuous cumulative weight; alpha =
// 1/(gamma - 1) (gamma = 3 gives the degree law of preferential attachment).
__global__ void chung_lu_kernel(uint32_t n, uint64_t m, double alpha, double i0, uint64_t seed, uint32_t *from,
                                uint32_t *to) {
    const double b = 1.0 - alpha;
    const double lo = pow(i0, b), hi = pow((double)n + i0, b);
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t st = seed ^ (e * 0xD1B54A32D192ED03ULL);
        uint32_t ends[2];
        for (int k = 0; k < 2; k++) {
            const double u = sm_unit(st);
            double x = pow(lo + u * (hi - lo), 1.0 / b) - i0;
            uint32_t v = x < 0.0 ? 0u : (uint32_t)x;
            ends[k] = v >= n ? n - 1 : v;
        }
        from[e] = ends[0];
        to[e] = ends[1];
    }
}

// Block model with a fixed edge count: block of the edge uniform among
// `blocks` equal blocks; with probability p_in both ends in that block,
// otherwise the target in another uniformly chosen block.
__global__ void sbm_edges_kernel(uint32_t n, uint64_t m, uint32_t blocks, double p_in, uint64_t seed, uint32_t *from,
                                 uint32_t *to) {
    const uint32_t bs = n / blocks;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t st = seed ^ (e * 0xD1B54A32D192ED03ULL);
        const uint32_t b0 = min((uint32_t)(sm_unit(st) * blocks), blocks - 1);
        uint32_t b1 = b0;
        if (sm_unit(st) >= p_in && blocks > 1) {
            b1 = min((uint32_t)(sm_unit(st) * (blocks - 1)), blocks - 2);
            if (b1 >= b0) b1++;
        }
        const uint32_t u = b0 * bs + min((uint32_t)(sm_unit(st) * bs), bs - 1);
        const uint32_t v = b1 * bs + min((uint32_t)(sm_unit(st) * bs), bs - 1);
        from[e] = u;
        to[e] = v;
    }
}

void generate_device(int kind, uint32_t n, uint64_t m, double p0, double p1, double p2, uint64_t seed,
                     uint32_t *d_from, uint32_t *d_to, cudaStream_t s) {
    const unsigned grid = grid_for(m, kThreads, 148u * 32u);
    if (kind == 0) {
        uint32_t scale = 0;
        while ((1ull << scale) < n) scale++;
        rmat_generate(scale, m, p0, p1, p2, seed, d_from, d_to, s);
    } else if (kind == 1) {
        chung_lu_kernel<<<grid, kThreads, 0, s>>>(n, m, p0, p1 > 0 ? p1 : 1.0, seed, d_from, d_to);
    } else {
        sbm_edges_kernel<<<grid, kThreads, 0, s>>>(n, m, (uint32_t)p0, p1, seed, d_from, d_to);
    }
    PRG_CUDA(cudaGetLastError());
}

}  // namespace prg
