// resident.cu — the whole FP64 iteration of a small or mid-sized graph in one
// persistent launch, its arcs resident in shared memory (indices and weights
// are streamed when they do not fit).
//
// Why: below a few million arcs a pass over the in-CSR takes 2-10 us of
// memory time, less than the launches around it.  The graph-replayed step is
// two kernels (tiles, spanning rows) of 6-10 + 5-8 us each at 0.1-0.8 M arcs,
// the eigenvector step four; both re-read indices, row records and reduction
// partials every time.  Here one block per SM takes a contiguous range of
// rows once, keeps its column indices (and arc weights), row-end bits and its
// own part of the iterate in shared memory, and each iteration is
//   gather (8 arcs per thread, L2) -> segmented sums -> row epilogue
//   -> one record per block -> one grid barrier.
// An iteration takes 4.7 us at 0.1 M arcs, 8 us at 1 M.  (Polling records that
// carry the barrier's number, to wait and read in one round trip, was slower:
// 6.2-8.0 us; 148 x 148 polls of the same lines delay the stores they wait for.)
//
// Rows are split so that arcs + alpha x rows is equal per block; a row never
// spans blocks, so the row sums need no second kernel.  Inside a block the
// sums come from a segmented scan: a thread owns 8 consecutive arcs (two
// 16-byte shared loads, laid out so that a quarter-warp reads 128 contiguous
// bytes), sums between row ends in FP64, a warp scan joins the open tails and
// a second scan over the warps adds the tails of the warps before.  No step
// depends on the order in which blocks or warps run, so results are
// bit-reproducible.
//
// RES_POWER is the reference's update in its rounding order (pagerank.rs:107-140,
// pagerank_weighted.rs:129-159, personalized_pagerank.rs:149-182) with its
// stop rule.  RES_EIG (eigenvector.rs:286-372, 375-538, 600-720 without
// negative weights) stops at a change below 1e-14 (1e-12 with weights), which
// lies under the rounding of such vectors: in plain FP64 the iterates end in a
// cycle of last-bit flips and most graphs run to the cap of 5000.  So the sums,
// the maximum and the division carry their rounding errors along (pairs of
// doubles) and each component is rounded once per iteration; the flips then die
// out and the rule holds after the 60-150 iterations the spectrum asks for
// (power law, 50 k vertices, 0.8 M arcs: 37 ms to the cap, 1.3 ms now).  It takes
// two barriers, one for max |y| and one for the change.
//
// The barrier's wait is bounded (about 1.5 s); after that the block sets
// Ctl::status and returns.
#include "resident.cuh"

#include <algorithm>
#include <type_traits>

#include "prims.cuh"

namespace prg {

constexpr int kResNT = 1024;
constexpr int kResWarps = kResNT / 32;
constexpr uint32_t kResNone = 0xFFFFu;       // rank of a row without arcs
constexpr uint32_t kResOpen = 0xFFFFFFFFu;   // no row end
// Larger graphs are bound by L1TEX lookups of the gathers, and the launched
// kernels, with a hot prefix in shared memory, are as fast or faster there
// (16 M arcs: 77 us an iteration on R-MAT).  us per iteration, resident /
// launched: 0.1 M arcs 4.7 / 18, 1 M 8.1 / 21, 4 M 23 / 38, 8 M 38 / 56 on
// uniform random graphs (weighted 1 M 8.3 / 24, 4 M 26 / 43, 8 M 49 / 63);
// R-MAT 4 M 15 / 28, 8 M 27 / 37 (weighted 8 M 38 / 43).
// Hence kResMaxArcs.
constexpr int kResTiles = 32;                // tiles of 8192 arcs a block can take
constexpr uint32_t kResMaxChunks = kResTiles * kResNT;
// The block with the most arcs sets an iteration's time, 3.3-4.5 us per tile
// where it gathers from L2, and the launched kernels spread a row over the chip;
// so a plan that gives one block, by a long row or by the coarse splits below,
// this many arcs more than the equal share is refused.  us per iteration,
// resident / launched, one row of 32 K, 48 K, 64 K, 96 K, 128 K arcs among 0.5 M:
// 20 / 22, 22 / 23, 30 / 23, 44 / 23, 54 / 21, among 5 M: 25 / 44, 46 / 45,
// 56 / 44, 58 / 45, 81 / 45; R-MAT scale 19 with 47 K above the share 36 / 42,
// with 50 K 48 / 43, scale 20 with 87 K 60 / 50 (weighted 92 / 56).  The lines
// cross near 48 K.  Between there and 68 K a solve on a resident graph loses
// 0.1-0.2 ms, but a drop-in wins more from the build (1.3-1.5 against 0.4-0.6 ms
// for 40-400 K arcs), and both must iterate in the same kernel to give the same
// bits.
constexpr uint64_t kResExcess = 68 << 10;
// Shared memory of a block (dynamic): L1 needs the rest for the gathers in
// flight and the hot sources.  R-MAT passes of 8 M arcs took 72-84 us with
// 190 KB of shared memory and 27 us with 144 KB; a power law's of 4 M arcs 40
// and 24 us.  On degree-sorted graphs the first kResL1Hot ids are gathered
// through L1, the others without allocating there (8192 against 2048 on R-MAT:
// 27 against 43 us).
constexpr size_t kResSmem = 160 << 10;
constexpr size_t kResStatic = 2048;          // shared memory kept for the kernel's static arrays
// A row weighs as much as alpha arcs in the split: 3 balances the time
// (power law, 8 M arcs: 44 us an iteration against 54 at 6 and 72 at 12);
// graphs of many short rows need 6 or 12 to fit shared memory.
constexpr unsigned kResSplits = 3;
__host__ __device__ constexpr uint32_t res_alpha(unsigned k) { return k == 0 ? 3u : k == 1 ? 6u : 12u; }
constexpr int kResRecs = kResBlocks / 32;     // records a lane adds
constexpr uint32_t kResMinShare = 1024;      // arcs + alpha rows a block takes at least
constexpr uint32_t kResSpins = 1u << 21;     // polls before a barrier gives up (~0.7 us each)

__device__ __forceinline__ void red_release(uint32_t *p, uint32_t v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// A running sum: plain FP64, or (DD) the unevaluated sum h + l of two doubles,
// in which an addition's rounding error is kept (Dekker's and Knuth's exact
// transformations).
__device__ __forceinline__ double two_sum(double a, double b, double &e) {
    const double s = __dadd_rn(a, b), t = __dsub_rn(s, a);
    e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, t)), __dsub_rn(b, t));
    return s;
}
template <bool DD>
struct Acc {
    double h = 0.0, l = 0.0;
    __device__ __forceinline__ void add(double vh, double vl) {
        if constexpr (DD) {
            double e;
            h = two_sum(h, vh, e);
            l += e + vl;
        } else {
            h += vh;
        }
    }
    __device__ __forceinline__ void add(const Acc &o) { add(o.h, o.l); }
    // |l| <= ulp(h) / 2; where h is infinite or NaN, l (NaN there) is dropped
    __device__ __forceinline__ void normalise() {
        const double s = __dadd_rn(h, l);
        if (isfinite(s)) {
            l = __dadd_rn(__dsub_rn(h, s), l);
            h = s;
        } else {
            l = 0.0;
        }
    }
    __device__ __forceinline__ Acc up(int o) const {
        Acc r;
        r.h = __shfl_up_sync(0xffffffffu, h, o);
        if constexpr (DD) r.l = __shfl_up_sync(0xffffffffu, l, o);
        return r;
    }
};

// Inclusive scan of the lanes' open tails: a lane stops adding where a lane of
// the range it already covers holds a row end (E: the lanes that do).
template <bool DD>
__device__ __forceinline__ Acc<DD> open_scan(Acc<DD> tv, uint32_t E) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Acc<DD> ov = tv.up(o);
        if (lane >= (uint32_t)o) {
            const uint32_t upto = lane == 31u ? 0xffffffffu : ((1u << (lane + 1)) - 1u);
            const uint32_t rng = upto & ~((1u << (lane - o + 1)) - 1u);
            if ((E & rng) == 0u) tv.add(ov);
        }
    }
    return tv;
}

// (h, l) becomes the larger of itself and (oh, ol), both normalised.
__device__ __forceinline__ void dd_max(double &h, double &l, double oh, double ol) {
    if (oh > h || (oh == h && ol > l)) {
        h = oh;
        l = ol;
    }
}

// First row r in [0, n] with row_ptr[r] + alpha r >= target (one warp, 32
// probes per round).
__device__ uint32_t res_cut(const uint32_t *rp, uint32_t n, uint32_t alpha, uint64_t target) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint64_t q = (uint64_t)lo + (uint64_t)lane * step + step - 1;
        const uint32_t p = q < hi ? (uint32_t)q : hi - 1;
        const bool ge = (uint64_t)__ldg(rp + p) + (uint64_t)alpha * p >= target;
        const uint32_t b = __ballot_sync(0xffffffffu, ge);
        if (b == 0u) {
            lo = hi;
        } else {
            const int f = __ffs(b) - 1;
            const uint32_t pf = __shfl_sync(0xffffffffu, p, f);
            const uint32_t pb = __shfl_sync(0xffffffffu, p, f ? f - 1 : 0);
            lo = f ? pb + 1 : lo;
            hi = pf;
        }
    }
    return lo;
}

// A block's share of the graph in a launch of nb blocks.
struct ResShare {
    uint32_t row0, rows, arc0, arcs, chunk0, chunks;
    __device__ ResShare(const uint32_t *rp, uint32_t r0, uint32_t r1) {
        row0 = r0;
        rows = r1 - r0;
        arc0 = __ldg(rp + r0);
        arcs = __ldg(rp + r1) - arc0;
        chunk0 = arc0 >> 3;  // chunks are the 8-arc groups of col, so a block's first and last may be shared
        chunks = arcs ? ((arc0 + arcs + 7) >> 3) - chunk0 : 0u;
    }
};

__host__ __device__ inline size_t res_bytes(uint32_t rows, uint32_t chunks, int kind, bool w, bool stream) {
    const size_t r2 = (rows + 1) & ~1u;
    return r2 * 8 * ((kind == RES_EIG ? 2 : 1) + (stream ? 0 : 1)) + (stream ? 0 : (size_t)chunks * (w ? 96 : 32)) +
           (size_t)((chunks + 3) >> 2) * 4 + (size_t)chunks * 2 + (size_t)rows * 2 +
           (size_t)((chunks + kResNT - 1) / kResNT) * kResWarps * (kind == RES_EIG ? 20 : 12) + 16;
}

// Bound on a block's shared bytes: its arcs + alpha rows exceed the equal share
// by less than one row.
__host__ __device__ inline double res_bound(uint64_t total, unsigned nb, uint32_t alpha, uint32_t longest, bool w,
                                            int kind) {
    const double share = (double)(total / nb + 2) + longest + alpha;
    const double per_arc = 4.46 + (w ? 8.0 : 0.0), per_row = (kind == RES_EIG ? 26.0 : 18.0) / alpha;
    return share * (per_arc > per_row ? per_arc : per_row) + 16.0 * per_arc + 1024.0;
}

// For the splits res_alpha(k): out[3k ..] = (largest shared bytes of a block,
// the same with indices and weights streamed, most chunks of a block)
__global__ void __launch_bounds__(1024) res_plan_kernel(const uint32_t *rp, uint32_t n, uint64_t arcs, unsigned nb,
                                                        int kind, bool w, uint32_t *out) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (unsigned i = blockIdx.x * (blockDim.x >> 5) + warp; i < nb * kResSplits; i += gridDim.x * (blockDim.x >> 5)) {
        const unsigned b = i / kResSplits, k = i % kResSplits;
        const uint32_t alpha = res_alpha(k);
        const uint64_t total = arcs + (uint64_t)alpha * n;
        const uint32_t r0 = b == 0 ? 0u : res_cut(rp, n, alpha, total * b / nb);
        const uint32_t r1 = b + 1 >= nb ? n : res_cut(rp, n, alpha, total * (b + 1) / nb);
        const ResShare sh(rp, r0, r1);
        if (lane == 0) {
            atomicMax(out + 3 * k, (uint32_t)res_bytes(sh.rows, sh.chunks, kind, w, false));
            atomicMax(out + 3 * k + 1, (uint32_t)res_bytes(sh.rows, sh.chunks, kind, w, true));
            atomicMax(out + 3 * k + 2, sh.chunks);
        }
    }
}

// Gather that does not allocate in L1 (coherent, unlike the read-only path).
__device__ __forceinline__ double ld_na(const double *p) {
    double v;
    asm volatile("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Eight consecutive indices at a 32-byte aligned address, not kept in L1.
__device__ __forceinline__ void ld_idx8(const uint32_t *p, uint32_t (&c)[8]) {
    asm("ld.global.nc.L1::no_allocate.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7])
        : "l"(p));
}
// Four consecutive weights at a 32-byte aligned address (whole sectors).
__device__ __forceinline__ void ld_w4(const double *p, double (&w)[4]) {
    asm("ld.global.nc.L1::no_allocate.v4.f64 {%0,%1,%2,%3}, [%4];"
        : "=d"(w[0]), "=d"(w[1]), "=d"(w[2]), "=d"(w[3])
        : "l"(p));
}

template <int KIND, bool W, bool STREAM>
__global__ void __launch_bounds__(kResNT, 1) res_kernel(const ResArgs a) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint32_t s_cut[2];
    __shared__ uint32_t s_scan[33];
    // per tile: the open sum after its last row end, the rank of its first one
    constexpr bool DD = KIND == RES_EIG;
    __shared__ double s_ttail[2][kResTiles];
    __shared__ uint32_t s_tfirst[kResTiles];
    __shared__ double s_red[2][kResWarps];
    __shared__ double s_g[2];
    __shared__ int s_ok;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned nb = gridDim.x, blk = blockIdx.x;

    if (a.longest) {
        if (a.ctl->status != 0) return;
        if (res_bound(a.total, nb, a.alpha, *a.longest, W, KIND) > (double)a.smem) {
            if (blk == 0 && tid == 0) a.ctl->status = 1;
            return;
        }
    }
    if (warp < 2) {
        const unsigned k = blk + warp;
        const uint32_t c = k >= nb ? a.n : k == 0 ? 0u : res_cut(a.row_ptr, a.n, a.alpha, a.total * k / nb);
        if (lane == 0) s_cut[warp] = c;
    }
    __syncthreads();
    const ResShare sh(a.row_ptr, s_cut[0], s_cut[1]);
    const uint32_t R0 = sh.row0, rows = sh.rows, nchunk = sh.chunks, rows2 = (rows + 1) & ~1u;
    // arcs lo .. hi-1 of the block's chunks are its own
    const uint32_t lo = sh.arc0 - sh.chunk0 * 8, hi = lo + sh.arcs;
    const uint32_t *col = a.col + (size_t)sh.chunk0 * 8;
    const double *w64 = W ? a.w64 + (size_t)sh.chunk0 * 8 : nullptr;

    // shared layout; col and weights as planes of 16 bytes per chunk
    double *S = reinterpret_cast<double *>(s_raw);  // row sums by rank, with DD their low parts
    double *L = S + (size_t)rows2;
    const uint32_t ntiles = (nchunk + kResNT - 1) / kResNT;
    // per tile and warp: the open sum after its last row end, and the rank of
    // its first row end (kResOpen: none)
    double *s_tail = S + (size_t)rows2 * (DD ? 2 : 1);
    double *s_taill = s_tail + ntiles * kResWarps;
    uint32_t *s_first = reinterpret_cast<uint32_t *>(s_tail + ntiles * kResWarps * (DD ? 2 : 1));
    double *vec = reinterpret_cast<double *>(s_first + ntiles * kResWarps);
    // the block's part of the iterate (in memory when streaming: each thread
    // reads back what it wrote)
    double *xs = STREAM ? a.x_out + R0 : vec;
    double *w_s = vec + (STREAM ? 0 : (size_t)rows2);
    uint32_t *c_s = reinterpret_cast<uint32_t *>(w_s + (W && !STREAM ? (size_t)nchunk * 8 : 0));
    uint32_t *m_s = c_s + (STREAM ? 0 : (size_t)nchunk * 8);  // row-end bits, one byte per chunk
    uint16_t *b_s = reinterpret_cast<uint16_t *>(m_s + ((nchunk + 3) >> 2));  // row ends before each chunk
    uint16_t *rk = b_s + nchunk;                              // rank of each row, or kResNone

    if (!STREAM) {
        for (uint32_t c = tid; c < nchunk; c += kResNT) {
            uint32_t cc[8];
            ld_idx8(col + (size_t)c * 8, cc);  // col is padded past its last arc
            *reinterpret_cast<uint4 *>(c_s + (size_t)c * 4) = make_uint4(cc[0], cc[1], cc[2], cc[3]);
            *reinterpret_cast<uint4 *>(c_s + (size_t)(nchunk + c) * 4) = make_uint4(cc[4], cc[5], cc[6], cc[7]);
            if (W) {
#pragma unroll
                for (int k = 0; k < 4; k += 2) {
                    double w[4];
                    ld_w4(w64 + (size_t)c * 8 + 2 * k, w);
                    *reinterpret_cast<double2 *>(w_s + (size_t)(k * nchunk + c) * 2) = make_double2(w[0], w[1]);
                    *reinterpret_cast<double2 *>(w_s + (size_t)((k + 1) * nchunk + c) * 2) = make_double2(w[2], w[3]);
                }
            }
        }
    }
    for (uint32_t i = tid; i < ((nchunk + 3) >> 2); i += kResNT) m_s[i] = 0u;
    __syncthreads();
    uint32_t run = 0, tot = 0;
    for (uint32_t r0 = 0; r0 < rows; r0 += kResNT) {
        const uint32_t r = r0 + tid;
        uint32_t ne = 0;
        if (r < rows) {
            const uint32_t p = __ldg(a.row_ptr + R0 + r), q = __ldg(a.row_ptr + R0 + r + 1);
            ne = q > p ? 1u : 0u;
            if (ne) {
                const uint32_t e = q - 1 - sh.chunk0 * 8;
                atomicOr(&m_s[e >> 5], 1u << (e & 31));
            }
        }
        const uint32_t pre = block_excl_scan(ne, s_scan, &tot);
        if (r < rows) rk[r] = ne ? (uint16_t)(run + pre) : (uint16_t)kResNone;
        run += tot;
    }
    __syncthreads();
    const uint8_t *m8 = reinterpret_cast<const uint8_t *>(m_s);
    run = 0;
    for (uint32_t c0 = 0; c0 < nchunk; c0 += kResNT) {
        const uint32_t c = c0 + tid;
        const uint32_t pre = block_excl_scan(c < nchunk ? __popc((uint32_t)m8[c]) : 0u, s_scan, &tot);
        if (c < nchunk) b_s[c] = (uint16_t)(run + pre);
        run += tot;
    }

    // Sums (v0, v1) over the grid, or with MAX takes the largest normalised pair:
    // block tree, record, barrier, then every block reduces the records in the
    // same order.
    uint32_t phase = 0;
    auto grid_reduce = [&](double &v0, double &v1, auto max_tag) -> bool {
        constexpr bool MAX = decltype(max_tag)::value;
        auto warp_reduce = [&]() {
            if constexpr (MAX) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const double oh = __shfl_xor_sync(0xffffffffu, v0, o), ol = __shfl_xor_sync(0xffffffffu, v1, o);
                    dd_max(v0, v1, oh, ol);
                }
            } else {
                v0 = warp_sum(v0);
                v1 = warp_sum(v1);
            }
        };
        warp_reduce();
        if (lane == 0) {
            s_red[0][warp] = v0;
            s_red[1][warp] = v1;
        }
        __syncthreads();  // also orders this block's global stores before the release below
        if (warp == 0) {
            v0 = s_red[0][lane];
            v1 = s_red[1][lane];
            warp_reduce();
            double2 *rec = a.rec + (size_t)(phase & 1u) * nb;
            if (lane == 0) {
                int ok = 1;
                __stcg(rec + blk, make_double2(v0, v1));
                red_release(a.bar, 1u);
                const uint32_t target = (phase + 1u) * nb + a.bar_extra;
                for (uint32_t spins = 0; ld_acquire(a.bar) < target;) {
                    if (++spins > kResSpins) {
                        a.ctl->status = 7;  // PRG_ERR_TIMEOUT
                        ok = 0;
                        break;
                    }
                }
                s_ok = ok;
            }
            __syncwarp();
            double2 q[kResRecs];
#pragma unroll
            for (int j = 0; j < kResRecs; j++)
                q[j] = lane + 32u * j < nb ? __ldcg(rec + lane + 32u * j) : make_double2(0.0, 0.0);
            v0 = q[0].x;
            v1 = q[0].y;
#pragma unroll
            for (int j = 1; j < kResRecs; j++) {
                if constexpr (MAX) {
                    dd_max(v0, v1, q[j].x, q[j].y);
                } else {
                    v0 += q[j].x;
                    v1 += q[j].y;
                }
            }
            warp_reduce();
            if (lane == 0) {
                s_g[0] = v0;
                s_g[1] = v1;
            }
        }
        __syncthreads();
        v0 = s_g[0];
        v1 = s_g[1];
        phase++;
        return s_ok != 0;
    };
    const std::false_type sums{};
    const std::true_type maxima{};

    // Row sums S[rank] of the products w x[col].  x is rewritten every
    // iteration by other SMs; the plain loads see the new values because the
    // barrier's acquire orders them (and drops this SM's cached lines), and
    // repeated sources hit L1.
    auto row_sums = [&](const double *x) {
        uint32_t tiles = 0;
        for (uint32_t c0 = 0; c0 < nchunk; c0 += kResNT, tiles++) {
            const uint32_t c = c0 + tid;
            double v[8], vl[8];  // products, with DD their rounding errors
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = vl[k] = 0.0;
            auto times = [&](int k, double w) {
                const double p = v[k] * w;
                if constexpr (DD) vl[k] = fma(v[k], w, -p);
                v[k] = p;
            };
            uint32_t m = 0, r = 0;
            if (c < nchunk) {
                uint32_t cc[8];
                if (STREAM) {
                    ld_idx8(col + (size_t)c * 8, cc);
                } else {
                    const uint4 p = *reinterpret_cast<const uint4 *>(c_s + (size_t)c * 4);
                    const uint4 q = *reinterpret_cast<const uint4 *>(c_s + (size_t)(nchunk + c) * 4);
                    cc[0] = p.x; cc[1] = p.y; cc[2] = p.z; cc[3] = p.w;
                    cc[4] = q.x; cc[5] = q.y; cc[6] = q.z; cc[7] = q.w;
                }
#pragma unroll
                for (int k = 0; k < 8; k++) v[k] = cc[k] < a.l1hot ? x[cc[k]] : ld_na(x + cc[k]);
                m = m8[c];
                r = b_s[c];
                if (W && STREAM) {
#pragma unroll
                    for (int k = 0; k < 8; k += 4) {
                        double ww[4];
                        ld_w4(w64 + (size_t)c * 8 + k, ww);
#pragma unroll
                        for (int i = 0; i < 4; i++) times(k + i, ww[i]);
                    }
                } else if (W) {
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const double2 ww = *reinterpret_cast<const double2 *>(w_s + (size_t)(k * nchunk + c) * 2);
                        times(2 * k, ww.x);
                        times(2 * k + 1, ww.y);
                    }
                }
                if (c * 8 < lo || c * 8 + 8 > hi) {  // arcs of the neighbouring blocks, padding
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        if (c * 8 + k < lo || c * 8 + k >= hi) v[k] = vl[k] = 0.0;
                }
            }
            const uint32_t r0 = r;
            Acc<DD> acc, head;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                acc.add(v[k], vl[k]);
                if ((m >> k) & 1u) {
                    if (r == r0) {
                        head = acc;
                    } else {
                        S[r] = acc.h;
                        if (DD) L[r] = acc.l;
                    }
                    r++;
                    acc = Acc<DD>();
                }
            }
            const uint32_t E = __ballot_sync(0xffffffffu, m != 0u);
            const Acc<DD> tv = open_scan(acc, E);
            Acc<DD> cin = tv.up(1);
            if (lane == 0u) cin = Acc<DD>();
            const uint32_t at = tiles * kResWarps + warp;
            if (m != 0u) {
                head.add(cin);
                S[r0] = head.h;
                if (DD) L[r0] = head.l;
                if ((E & lanemask_lt()) == 0u) s_first[at] = r0;  // may lack what came before the warp
            }
            if (lane == 31u) {
                s_tail[at] = tv.h;
                if (DD) s_taill[at] = tv.l;
                if (E == 0u) s_first[at] = kResOpen;
            }
        }
        auto add_to = [&](uint32_t rank, const Acc<DD> &c) {
            Acc<DD> t;
            t.h = S[rank];
            if (DD) t.l = L[rank];
            t.add(c);
            S[rank] = t.h;
            if (DD) L[rank] = t.l;
        };
        __syncthreads();
        // what a warp's first row holds from the warps before it in its tile
        if (warp < tiles) {
            const uint32_t at = warp * kResWarps + lane, first = s_first[at];
            const uint32_t F = __ballot_sync(0xffffffffu, first != kResOpen);
            Acc<DD> tail;
            tail.h = s_tail[at];
            if (DD) tail.l = s_taill[at];
            const Acc<DD> tv = open_scan(tail, F);
            const Acc<DD> cin = tv.up(1);
            if (lane != 0u && first != kResOpen) add_to(first, cin);
            if (lane == 31u) {
                s_ttail[0][warp] = tv.h;
                s_ttail[1][warp] = tv.l;
            }
            const uint32_t tf = __shfl_sync(0xffffffffu, first, F ? __ffs(F) - 1 : 0);
            if (lane == 0u) s_tfirst[warp] = F ? tf : kResOpen;
        }
        __syncthreads();
        if (tiles > 1) {  // and a tile's first row from the tiles before it
            if (tid > 0 && tid < tiles && s_tfirst[tid] != kResOpen) {
                int t = (int)tid - 1;
                while (t > 0 && s_tfirst[t] == kResOpen) t--;
                Acc<DD> c;
                for (; t < (int)tid; t++) c.add(s_ttail[0][t], s_ttail[1][t]);
                add_to(s_tfirst[tid], c);
            }
            __syncthreads();
        }
    };

    uint32_t it = 0;
    double last = 0.0;  // L1 change of the newest completed iteration
    int done = 0;
    if (KIND == RES_POWER) {
        const double d = a.damping, nf = (double)a.n;
        const double tele = __ddiv_rn(1.0 - d, nf);
        double v0 = 0.0, dsum = 0.0;
        for (uint32_t r = tid; r < rows; r += kResNT) {
            const uint32_t v = R0 + r;
            const double x = a.start ? a.start[v] : a.t64 ? a.t64[v] : 1.0 / nf;
            const double dv = __ldg(a.dval + v);
            xs[r] = x;
            if (dv == 0.0) dsum += x;
            a.xt[0][v] = dv == 0.0 ? 0.0 : x / dv;
        }
        if (!grid_reduce(v0, dsum, sums)) return;
        while (it < a.max_iter && !done) {
            const double *src = a.xt[it & 1u];
            double *dst = a.xt[(it & 1u) ^ 1u];
            row_sums(src);
            const double dshare = __ddiv_rn(__dmul_rn(d, dsum), nf);
            double pd = 0.0, pds = 0.0;
            for (uint32_t r = tid; r < rows; r += kResNT) {
                const uint32_t v = R0 + r, k = rk[r];
                const double y = k == kResNone ? 0.0 : S[k];
                const double dv = __ldg(a.dval + v);
                double out;
                if (a.t64) {  // personalized_pagerank.rs:169-170
                    const double t = __ldg(a.t64 + v);
                    out = __dadd_rn(__dmul_rn(1.0 - d, t), __dmul_rn(d, __dadd_rn(y, __dmul_rn(dsum, t))));
                } else {  // pagerank.rs:129
                    out = __dadd_rn(__dadd_rn(tele, dshare), __dmul_rn(d, y));
                }
                pd += fabs(out - xs[r]);
                xs[r] = out;
                if (dv == 0.0) pds += out;
                dst[v] = dv == 0.0 ? 0.0 : out / dv;
            }
            if (!grid_reduce(pd, pds, sums)) return;
            it++;
            last = pd;
            dsum = pds;
            done = last < a.thr || it >= a.max_iter;
        }
        if (!STREAM)
            for (uint32_t r = tid; r < rows; r += kResNT) a.x_out[R0 + r] = xs[r];
    } else {
        if (!STREAM)
            for (uint32_t r = tid; r < rows; r += kResNT) xs[r] = a.x_out[R0 + r];
        // row r of (shift I + A) x as a normalised pair
        auto product = [&](uint32_t r) {
            const uint32_t q = rk[r];
            const double x = xs[r], p = a.shift * x;
            Acc<DD> y;
            y.h = p;
            y.l = fma(a.shift, x, -p);
            if (q != kResNone) y.add(S[q], L[q]);
            y.normalise();
            return y;
        };
        while (!done) {
            row_sums(a.x_out);
            double mh = 0.0, ml = 0.0;
            for (uint32_t r = tid; r < rows; r += kResNT) {
                const Acc<DD> y = product(r);
                dd_max(mh, ml, y.h, y.l);
            }
            if (!grid_reduce(mh, ml, maxima)) return;  // every block has gathered x
            double pd = 0.0, unused = 0.0;
            for (uint32_t r = tid; r < rows; r += kResNT) {
                const Acc<DD> y = product(r);
                double x = y.h;
                if (mh > 0.0) {  // y / max, rounded once; a zero vector is not scaled
                    const double q = y.h / mh;
                    x = isfinite(mh) ? q + (fma(-q, mh, y.h) + (y.l - q * ml)) / mh : q;
                }
                pd += fabs(x - xs[r]);
                xs[r] = x;
                if (!STREAM) a.x_out[R0 + r] = x;
            }
            if (!grid_reduce(pd, unused, sums)) return;
            it++;
            last = pd;
            done = last < a.thr || it >= a.max_iter;
        }
        // Rayleigh quotient of the last iterate
        row_sums(a.x_out);
        double num = 0.0, den = 0.0;
        for (uint32_t r = tid; r < rows; r += kResNT) {
            const uint32_t q = rk[r];
            const double x = xs[r];
            num += x * (q == kResNone ? 0.0 : isfinite(L[q]) ? S[q] + L[q] : S[q]);
            den += x * x;
        }
        if (!grid_reduce(num, den, sums)) return;
        if (blk == 0 && tid == 0) {
            a.ctl->dsum[0] = num;
            a.ctl->dsum[1] = den;
        }
    }
    if (blk == 0 && tid == 0) {
        a.ctl->iters = it;
        a.ctl->diff = last;
        a.ctl->done = done;
    }
}

// ------------------------------------------------------------------ host side

const DeviceLimits &device_limits() {
    static const DeviceLimits limits = []() {
        DeviceLimits d;
        int dev = 0;
        PRG_CUDA(cudaGetDevice(&dev));
        PRG_CUDA(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
        PRG_CUDA(cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        return d;
    }();
    return limits;
}

// Shared memory a block may take, and the blocks of a launch.
static size_t res_limits(uint64_t arcs, uint32_t n, unsigned &nb) {
    const DeviceLimits &d = device_limits();
    nb = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>(std::min<unsigned>(d.sms, kResBlocks), (arcs + (uint64_t)res_alpha(0) * n) / kResMinShare));
    return std::min(kResSmem, (size_t)d.smem_optin - kResStatic);
}

// Most 8-arc chunks of a block's share.
static uint64_t most_chunks(uint64_t arcs, unsigned nb) {
    return std::min<uint64_t>(kResMaxChunks, (arcs / nb + kResExcess) / 8 + 1);
}

// Whether the mean share, streamed, fits a block.
static bool res_mean_fits(uint32_t n, uint64_t arcs, bool weighted, int kind) {
    unsigned nb = 0;
    const size_t most = res_limits(arcs, n, nb);
    const uint64_t chunks = arcs / 8 / nb;
    return chunks <= kResMaxChunks && res_bytes(n / nb, (uint32_t)chunks, kind, weighted, true) <= most;
}

uint32_t res_longest_row(uint32_t n, uint64_t arcs) {
    unsigned nb = 0;
    res_limits(arcs, n, nb);
    return 8 * (uint32_t)most_chunks(arcs, nb);
}

bool res_sizes_fit(uint32_t n, uint64_t arcs, bool weighted, int kind) {
    return n >= 2 && arcs > 0 && arcs <= kResMaxArcs && res_mean_fits(n, arcs, weighted, kind);
}

ResPlan res_plan_blind(uint32_t n, uint64_t arcs, bool weighted, int kind) {
    ResPlan p;
    if (n < 2 || arcs == 0 || arcs > kResMaxArcs) return p;
    unsigned nb = 0;
    const size_t most = res_limits(arcs, n, nb);
    p.alpha = res_alpha(0);
    const uint64_t total = arcs + (uint64_t)p.alpha * n;
    // room for rows of up to 8192 arcs, or what shared memory leaves
    if (res_bound(total, nb, p.alpha, 512, weighted, kind) > (double)most) return p;
    p.smem = std::min(most, ((size_t)res_bound(total, nb, p.alpha, 8192, weighted, kind) + 15) & ~(size_t)15);
    p.grid = nb;
    return p;
}

ResPlan res_plan(const DeviceGraph &g, int kind, cudaStream_t s) {
    ResPlan p;
    if (g.n < 2 || g.arcs == 0 || g.arcs > kResMaxArcs) return p;
    unsigned nb = 0;
    const size_t most = res_limits(g.arcs, g.n, nb);
    // small graphs fit whatever their rows look like (36 K arcs in a block at most)
    p.alpha = res_alpha(0);
    const uint64_t total = g.arcs + (uint64_t)p.alpha * g.n;
    const double bound = res_bound(total, nb, p.alpha, g.max_in_degree, g.weighted, kind);
    if (bound <= (double)most) {
        p.grid = nb;
        p.smem = ((size_t)bound + 15) & ~(size_t)15;
        return p;
    }
    // otherwise the shares themselves decide, unless even the mean does not fit
    if (!res_mean_fits(g.n, g.arcs, g.weighted, kind)) return p;
    uint32_t *d = nullptr, h[3 * kResSplits];
    PRG_CUDA(cudaMallocAsync((void **)&d, sizeof(h), s));
    PRG_CUDA(cudaMemsetAsync(d, 0, sizeof(h), s));
    res_plan_kernel<<<15, 1024, 0, s>>>(g.row_ptr, g.n, g.arcs, nb, kind, g.weighted, d);
    PRG_CUDA(cudaGetLastError());
    PRG_CUDA(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, s));
    PRG_CUDA(cudaFreeAsync(d, s));
    PRG_CUDA(cudaStreamSynchronize(s));
    const uint64_t top = most_chunks(g.arcs, nb);
    for (unsigned k = 0; k < kResSplits; k++) {
        const bool stream = h[3 * k] > most;
        const uint32_t bytes = h[3 * k + (stream ? 1 : 0)];
        if (bytes > most || h[3 * k + 2] > top) continue;
        p.alpha = res_alpha(k);
        p.stream = stream;
        p.grid = nb;
        p.smem = bytes;
        break;
    }
    return p;
}

size_t res_scratch_bytes(unsigned grid) { return 256 + (size_t)grid * 2 * sizeof(double2); }

template <int KIND, bool W, bool STREAM>
static bool res_go(const ResPlan &p, const ResArgs &a, cudaStream_t s) {
    // the attribute belongs to the kernel, not to this launch: always the limit
    PRG_CUDA(cudaFuncSetAttribute(res_kernel<KIND, W, STREAM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kResSmem));
    PRG_CUDA(cudaMemsetAsync(a.bar, 0, 4, s));
    void *args[] = {(void *)&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)res_kernel<KIND, W, STREAM>, dim3(p.grid),
                                                      dim3(kResNT), args, p.smem, s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return false;
    }
    PRG_CUDA(e);
    return true;
}

bool launch_resident(int kind, const ResPlan &p, const ResArgs &args, cudaStream_t s) {
    ResArgs a = args;
    a.bar_extra = tuning().resident_barrier_extra == 1u ? 1u : 0u;
    const bool w = a.w64 != nullptr;
    if (kind == RES_EIG) {
        if (p.stream) return w ? res_go<RES_EIG, true, true>(p, a, s) : res_go<RES_EIG, false, true>(p, a, s);
        return w ? res_go<RES_EIG, true, false>(p, a, s) : res_go<RES_EIG, false, false>(p, a, s);
    }
    if (p.stream) return w ? res_go<RES_POWER, true, true>(p, a, s) : res_go<RES_POWER, false, true>(p, a, s);
    return w ? res_go<RES_POWER, true, false>(p, a, s) : res_go<RES_POWER, false, false>(p, a, s);
}

}  // namespace prg
