// small_call.cu — one-call drop-ins on small graphs in two launches.
//
// A general call builds the CSR with about 80 launches and 10 host round
// trips (radix sort passes, scans, row-blocks, sizes read back): 0.4-0.6 ms
// for G(1000, 25 000), where the build's device work is 0.2 ms and the
// iteration's 0.08.  Here one cooperative launch builds the in-CSR, its phases
// separated by grid barriers, and the iteration kernel follows without a host
// round trip in between:
//   1  every arc takes a slot of its destination (atomic count), endpoints
//      are range-checked;
//   2  the counts are scanned into row pointers (block sums, one barrier);
//   3  arc ids go to row start + slot;
//   4  every row is sorted by arc id, which restores the edge-id order the
//      reference adds in (the slots came in any order), and sources, weights
//      and divisors are filled in: a warp per row of up to kSmallWarpRow arcs
//      by counting smaller ids, a block per longer row by a bitmap of the ids.
// So the CSR, and with it every sum, is the same from run to run and the same
// as the general build's.  Vertices keep their ids (results are not affected,
// and these graphs' vectors fit L2).  Weighted directed graphs run the same
// phases a second time by source for the out-strengths.
//
// Limits: res_sizes_fit, and rows of up to res_longest_row arcs: the first arc
// past that ends the build.  Where res_plan_blind gives no plan, or the rows turn
// out too uneven for its shares (Ctl::status), the iteration is planned from the
// CSR just built, and only if that fails does the caller take the general path,
// with the edge list as uploaded here.
#include "small_call.cuh"

#include <algorithm>
#include <cstring>

#include "pool.cuh"
#include "prims.cuh"

namespace prg {

constexpr int kSmallNT = 1024;
// Rows of up to this many arcs are sorted by one warp (counting smaller ids is
// quadratic, and its loads come in chains of 32 arcs); longer ones by a block.
constexpr uint32_t kSmallWarpRow = 128;
// A warp's buffer in words: the ids of one such row, or the weights of four
// 32-arc rows.
constexpr uint32_t kSmallWarpBuf = 256;
static_assert(kSmallWarpBuf >= kSmallWarpRow && kSmallWarpBuf * 4 >= 4 * 32 * sizeof(double), "warp buffer");
constexpr uint32_t kSmallRange = 1u << 20;           // ids per bitmap of the block sort
__host__ __device__ constexpr uint32_t small_word(uint32_t i) { return i + (i >> 5); }
constexpr size_t kSmallSmem = small_word(kSmallRange / 32) * 4;  // also 32 warp buffers
constexpr uint32_t kSmallSpins = 1u << 21;
static_assert(kSmallSmem >= (size_t)(kSmallNT / 32) * kSmallWarpBuf * 4, "warp buffers");

struct SmallSide {
    uint32_t *cnt;   // n, zero: arcs per row
    uint32_t *slot;  // per arc: arrival number in its row
    uint32_t *ptr;   // n + 1
    uint32_t *ids;   // arc ids by row
    uint32_t *bsum;  // per block
    uint32_t *longs; // n: rows longer than kSmallWarpRow
};

struct SmallArgs {
    const uint32_t *from, *to;
    const double *w;
    uint32_t n, m, longest;  // longest: of a row
    uint32_t bar_extra;      // test hook: arrivals a barrier waits for beyond the grid's
    int directed, check_w, seed;  // seed 0: none, 1: ones, 2: dval / max dval (ones when that is 0)
    SmallSide in, outs;      // outs only for weighted directed graphs
    uint32_t *deg;           // directed, unweighted: out-degrees, zero at launch
    uint32_t *col;           // arcs + kColPad
    double *w64;             // arcs + kColPad
    double *dval, *start;
    // [0] largest endpoint [1] longest in-row [2] barrier [3], [4] listed in- / out-rows [5] ~first refused
    // weight's edge (0: none) [6..7] max dval bits [8] a row is too long
    uint32_t *word;          // zero at launch
    Ctl *ctl;
};

// Grid barrier number `phase`; false when its bounded wait ran out.
__device__ bool small_barrier(const SmallArgs &a, uint32_t &phase) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        phase++;
        int ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(a.word + 2), "r"(1u) : "memory");
        uint32_t seen = 0;
        for (uint32_t spins = 0;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.word + 2) : "memory");
            if (seen >= phase * gridDim.x + a.bar_extra) break;
            if (++spins > kSmallSpins) {
                a.ctl->status = 7;  // PRG_ERR_TIMEOUT
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Row of arc `id` on a side, and its other end.
__device__ __forceinline__ void small_arc(const SmallArgs &a, bool outs, uint32_t id, uint32_t &row, uint32_t &other) {
    const uint32_t e = a.directed ? id : id >> 1;
    const uint32_t u = __ldg(a.from + e), v = __ldg(a.to + e);
    const bool by_from = a.directed ? outs : (id & 1u) == 0u;  // undirected arc 2e: row u, source v
    row = by_from ? u : v;
    other = by_from ? v : u;
}

// Fills position p with arc id; returns its weight (0 without weights).
__device__ __forceinline__ double small_fill(const SmallArgs &a, bool outs, uint32_t p, uint32_t id) {
    const uint32_t e = a.directed ? id : id >> 1;
    const double we = a.w ? __ldg(a.w + e) : 0.0;
    if (outs) {
        a.outs.slot[p] = id;  // the slots are used up by now
        return we;
    }
    const uint32_t u = __ldg(a.from + e), v = __ldg(a.to + e);
    a.col[p] = a.directed || (id & 1u) ? u : v;
    if (a.w) a.w64[p] = we;
    return we;
}

// Divisor of row r once its arcs [p0, p1) are in place (one warp).
__device__ __forceinline__ void small_divisor(const SmallArgs &a, bool outs, uint32_t r, uint32_t p0, uint32_t p1) {
    const uint32_t lane = threadIdx.x & 31;
    if (!a.w) {
        if (lane == 0) a.dval[r] = (double)(a.directed ? a.deg[r] : p1 - p0);
        return;
    }
    if (a.directed && !outs) return;
    double acc = 0.0;
    for (uint32_t p = p0 + lane; p < p1; p += 32) acc += outs ? a.w[a.outs.slot[p]] : a.w64[p];
    acc = warp_sum(acc);
    if (lane == 0) a.dval[r] = acc;
}

__global__ void __launch_bounds__(kSmallNT, 1) small_build_kernel(const SmallArgs a) {
    extern __shared__ __align__(16) uint32_t s_ids[];
    __shared__ uint32_t s_scan[33];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t gtid = blockIdx.x * kSmallNT + tid, gn = gridDim.x * kSmallNT;
    const uint32_t n = a.n, m = a.m, arcs = a.directed ? m : 2 * m;
    const bool two = a.w != nullptr && a.directed;
    uint32_t phase = 0;

    // 1: slots.  A row too long for any plan ends the phase: its arcs' atomics on
    // one word and its sort by one block would be in vain (a row of 5 M arcs held
    // a call up by 20 ms).  A slot is looked at one step later, when it has arrived,
    // and the word that says so at every fourth (1 M arcs 0.77 ms a call, at every
    // step 0.79; one row of 5 M arcs 3.5 and 3.3, the general path alone 3.1).
    {
        uint32_t mx = 0, bad = 0, s0 = 0, s1 = 0, step = 0;
        uint32_t *too_long = a.word + 8;
        for (uint32_t e = gtid; e < m; e += gn) {
            const uint32_t u = a.from[e], v = a.to[e];
            if ((++step & 3u) == 0u && *(volatile uint32_t *)too_long) break;
            if (max(s0, s1) >= a.longest) *(volatile uint32_t *)too_long = 1u;
            mx = max(mx, max(u, v));
            if (a.check_w && !(a.w[e] >= 0.0 && isfinite(a.w[e]))) bad = max(bad, ~e);
            if (u >= n || v >= n) continue;
            if (a.directed) {
                a.in.slot[e] = s0 = atomicAdd(&a.in.cnt[v], 1u);
                if (two) a.outs.slot[e] = atomicAdd(&a.outs.cnt[u], 1u);
                else atomicAdd(&a.deg[u], 1u);
            } else {
                a.in.slot[2 * e] = s0 = atomicAdd(&a.in.cnt[u], 1u);
                a.in.slot[2 * e + 1] = s1 = atomicAdd(&a.in.cnt[v], 1u);
            }
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0 && mx) atomicMax(a.word, mx);
        if (bad) atomicMax(a.word + 5, bad);
    }
    if (!small_barrier(a, phase)) return;
    if (*(volatile uint32_t *)(a.word + 8) != 0u) {  // every block sees the same
        if (gtid == 0) a.ctl->status = SMALL_LONG_ROW;
        return;
    }
    if (*(volatile uint32_t *)(a.word + 5) != 0u) {
        if (gtid == 0) a.ctl->status = SMALL_BAD_WEIGHT;
        return;
    }
    if (*(volatile uint32_t *)a.word >= n) {
        if (gtid == 0) a.ctl->status = SMALL_OUT_OF_RANGE;
        return;
    }

    // 2: row pointers; rows too long for a warp are listed
    const uint32_t per = (n + gridDim.x - 1) / gridDim.x;
    const uint32_t v0 = min(n, per * blockIdx.x), v1 = min(n, v0 + per);
    for (int side = 0; side < (two ? 2 : 1); side++) {
        const SmallSide &sd = side ? a.outs : a.in;
        uint32_t run = 0, tot = 0, longest = 0;  // (of the in-rows)
        for (uint32_t b = v0; b < v1; b += kSmallNT) {
            const uint32_t v = b + tid;
            const uint32_t c = v < v1 ? __ldcg(&sd.cnt[v]) : 0u;
            if (c > kSmallWarpRow) sd.longs[atomicAdd(a.word + 3 + side, 1u)] = v;
            if (side == 0) longest = max(longest, c);
            const uint32_t pre = block_excl_scan(c, s_scan, &tot);
            if (v < v1) sd.ptr[v] = run + pre;
            run += tot;
        }
        longest = __reduce_max_sync(0xffffffffu, longest);
        if (lane == 0 && longest) atomicMax(a.word + 1, longest);
        if (tid == 0) sd.bsum[blockIdx.x] = run;
    }
    if (!small_barrier(a, phase)) return;
    for (int side = 0; side < (two ? 2 : 1); side++) {
        const SmallSide &sd = side ? a.outs : a.in;
        uint32_t below = 0;
        for (uint32_t b = lane; b < blockIdx.x; b += 32) below += __ldcg(&sd.bsum[b]);
        below = __reduce_add_sync(0xffffffffu, below);
        for (uint32_t v = v0 + tid; v < v1; v += kSmallNT) sd.ptr[v] += below;
        if (blockIdx.x == 0 && tid == 0) sd.ptr[n] = arcs;
    }
    if (!small_barrier(a, phase)) return;

    // 3: arc ids to their rows, in any order within a row
    for (uint32_t i = gtid; i < arcs; i += gn) {
        uint32_t row, other;
        small_arc(a, false, i, row, other);
        a.in.ids[__ldcg(&a.in.ptr[row]) + a.in.slot[i]] = i;
        if (two) {
            small_arc(a, true, i, row, other);
            a.outs.ids[__ldcg(&a.outs.ptr[row]) + a.outs.slot[i]] = i;
        }
    }
    if (gtid < kColPad) {
        a.col[arcs + gtid] = 0u;
        if (a.w) a.w64[arcs + gtid] = 0.0;
    }
    if (!small_barrier(a, phase)) return;

    // 4: rows in arc order
    uint32_t *buf = s_ids + warp * kSmallWarpBuf;
    for (int side = 0; side < (two ? 2 : 1); side++) {
        const bool outs = side != 0;
        const SmallSide &sd = outs ? a.outs : a.in;
        // Four rows per warp and step, their loads in flight together (a row is
        // a chain of four L2 round trips).  Neighbouring rows go to different
        // blocks: long rows often have close ids.
        const uint32_t stride = gn >> 5;
        for (uint32_t r0 = blockIdx.x + gridDim.x * warp; r0 < n; r0 += 4 * stride) {
            uint32_t p0[4], len[4], id[4], rank[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t r = r0 + k * stride;
                const uint32_t q = r < n ? __ldcg(&sd.ptr[r + 1]) : 0u;
                p0[k] = r < n ? __ldcg(&sd.ptr[r]) : 0u;
                len[k] = q - p0[k];
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                id[k] = len[k] <= 32 && lane < len[k] ? __ldcg(&sd.ids[p0[k] + lane]) : 0xFFFFFFFFu;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                rank[k] = 0;
                if (len[k] <= 32)
                    for (uint32_t j = 0; j < len[k]; j++) rank[k] += __shfl_sync(0xffffffffu, id[k], j) < id[k] ? 1u : 0u;
            }
            double *wbuf = reinterpret_cast<double *>(buf);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (len[k] > 32 || lane >= len[k]) continue;
                const double we = small_fill(a, outs, p0[k] + rank[k], id[k]);
                if (a.w) wbuf[k * 32 + rank[k]] = we;
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t r = r0 + k * stride;
                if (r >= n || len[k] > 32) continue;
                if (!a.w) {
                    if (lane == 0) a.dval[r] = (double)(a.directed ? a.deg[r] : len[k]);
                } else if (!a.directed || outs) {  // as small_divisor adds them
                    const double acc = warp_sum(lane < len[k] ? wbuf[k * 32 + lane] : 0.0);
                    if (lane == 0) a.dval[r] = acc;
                }
            }
            for (int k = 0; k < 4; k++) {
                const uint32_t r = r0 + k * stride, ln = len[k], p = p0[k];
                if (ln <= 32 || ln > kSmallWarpRow) continue;
                const uint32_t ln4 = (ln + 3) & ~3u;
                __syncwarp();
                for (uint32_t j = lane; j < ln4; j += 32) buf[j] = j < ln ? __ldcg(&sd.ids[p + j]) : 0xFFFFFFFFu;
                __syncwarp();
                for (uint32_t j = lane; j < ln; j += 32) {
                    const uint32_t x = buf[j];
                    uint32_t rk = 0;
                    for (uint32_t i = 0; i < ln4; i += 4) {
                        const uint4 q = *reinterpret_cast<const uint4 *>(buf + i);
                        rk += (q.x < x ? 1u : 0u) + (q.y < x ? 1u : 0u) + (q.z < x ? 1u : 0u) + (q.w < x ? 1u : 0u);
                    }
                    small_fill(a, outs, p + rk, x);
                }
                __syncwarp();
                small_divisor(a, outs, r, p, p + ln);
            }
        }
        __syncthreads();
        const uint32_t nlong = *(volatile uint32_t *)(a.word + 3 + side);
        for (uint32_t i = blockIdx.x; i < nlong; i += gridDim.x) {
            const uint32_t r = __ldcg(&sd.longs[i]);
            const uint32_t p0 = __ldcg(&sd.ptr[r]), p1 = __ldcg(&sd.ptr[r + 1]), len = p1 - p0;
            // ids below `base` are placed; the next kSmallRange ids as a bitmap, a
            // thread owning `words` consecutive words (one word of padding per 32
            // keeps the threads' words in different banks)
            uint32_t done = 0;
            for (uint32_t base = 0; base < arcs && done < len; base += kSmallRange) {
                const uint32_t words = (min(kSmallRange, arcs - base) + 32 * kSmallNT - 1) / (32 * kSmallNT);
                for (uint32_t j = tid; j < small_word(words * kSmallNT); j += kSmallNT) s_ids[j] = 0u;
                __syncthreads();
                for (uint32_t j = tid; j < len; j += kSmallNT) {
                    const uint32_t id = __ldcg(&sd.ids[p0 + j]) - base;
                    if (id < kSmallRange) atomicOr(&s_ids[small_word(id >> 5)], 1u << (id & 31));
                }
                __syncthreads();
                uint32_t cnt = 0, tot = 0;
                for (uint32_t k = 0; k < words; k++) cnt += __popc(s_ids[small_word(tid * words + k)]);
                uint32_t p = p0 + done + block_excl_scan(cnt, s_scan, &tot);
                for (uint32_t k = 0; k < words && cnt; k++) {
                    for (uint32_t w = s_ids[small_word(tid * words + k)]; w; w &= w - 1u)
                        small_fill(a, outs, p++, base + (tid * words + k) * 32 + __ffs(w) - 1);
                }
                done += tot;
                __syncthreads();
            }
            if (warp == 0) small_divisor(a, outs, r, p0, p1);
        }
        __syncthreads();
    }

    // the eigenvector iteration's start
    if (a.seed == 1)
        for (uint32_t v = gtid; v < n; v += gn) a.start[v] = 1.0;
    if (a.seed == 2) {
        if (!small_barrier(a, phase)) return;
        unsigned long long *top = reinterpret_cast<unsigned long long *>(a.word + 6);
        unsigned long long mx = 0;  // non-negative doubles order as their bits
        for (uint32_t v = gtid; v < n; v += gn)
            mx = max(mx, (unsigned long long)__double_as_longlong(__ldcg(&a.dval[v])));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) atomicMax(top, mx);
        if (!small_barrier(a, phase)) return;
        const double t = __longlong_as_double((long long)*(volatile unsigned long long *)top);
        for (uint32_t v = gtid; v < n; v += gn) a.start[v] = t > 0.0 ? __ldcg(&a.dval[v]) / t : 1.0;
    }
}

// ------------------------------------------------------------------ host side

SmallStatus small_call(const SmallCall &c, double *out, SmallResult &r, cudaStream_t s) {
    const uint64_t arcs = c.directed ? c.m : 2 * c.m;
    const uint32_t n = c.n;
    const bool two = c.w != nullptr && c.directed;
    // Before anything is copied: from 2.0-2.4 M vertices on (1.1-1.3 M with
    // eigenvectors) no share fits a block.  Copying and building first, to be
    // refused by the plan, made a call on 3 M vertices and 6 M edges 12.7 ms
    // instead of 8.6.
    if (!res_sizes_fit(n, arcs, c.w != nullptr, c.kind)) return SMALL_NOT_HERE;
    // without a blind plan the iteration is planned once the rows are known
    const ResPlan p = res_plan_blind(n, arcs, c.w != nullptr, c.kind);
    PRG_CUDA(cudaFuncSetAttribute(small_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
    // few arcs need few blocks: a barrier over fewer is shorter
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(device_limits().sms, (arcs + n) / 2048));

    // one allocation: first what must be zero, then the rest
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) & ~(size_t)255;
        return o;
    };
    const size_t o_ctl = take(sizeof(Ctl)), o_word = take(64), o_bar = take(4), o_cnt = take(n * 4ull),
                 o_deg = take(c.directed && !c.w ? n * 4ull : 4), o_cnt2 = take(two ? n * 4ull : 4), zeroed = at;
    const size_t o_from = take(c.m * 4), o_to = take(c.m * 4), o_w = take(c.w ? c.m * 8 : 8),
                 o_slot = take(arcs * 4), o_ptr = take((n + 1ull) * 4), o_ids = take(arcs * 4), o_bs = take(grid * 4ull),
                 o_long = take(n * 4ull), o_slot2 = take(two ? arcs * 4 : 4), o_ptr2 = take(two ? (n + 1ull) * 4 : 4),
                 o_ids2 = take(two ? arcs * 4 : 4), o_bs2 = take(grid * 4ull), o_long2 = take(two ? n * 4ull : 4),
                 o_col = take((arcs + kColPad) * 4), o_w64 = take(c.w ? (arcs + kColPad) * 8 : 8), o_dval = take(n * 8ull),
                 o_x = take(n * 8ull), o_t = take(c.reset ? n * 8ull : 8), o_xt0 = take(n * 8ull), o_xt1 = take(n * 8ull),
                 o_rec = take(res_scratch_bytes(kResBlocks));
    unsigned char *b = nullptr;
    Ctl *h = static_cast<Ctl *>(pinned_acquire());
    SmallStatus status = SMALL_DONE;
    auto give_up = [&]() {
        cudaStreamSynchronize(s);
        if (b) cudaFreeAsync(b, s);
        pinned_release(h);
    };
    try {
        PRG_CUDA(cudaMallocAsync((void **)&b, at, s));
        PRG_CUDA(cudaMemsetAsync(b, 0, zeroed, s));
        PRG_CUDA(cudaMemcpyAsync(b + o_from, c.from, c.m * 4, cudaMemcpyHostToDevice, s));
        PRG_CUDA(cudaMemcpyAsync(b + o_to, c.to, c.m * 4, cudaMemcpyHostToDevice, s));
        if (c.w) PRG_CUDA(cudaMemcpyAsync(b + o_w, c.w, c.m * 8, cudaMemcpyHostToDevice, s));
        if (c.reset) PRG_CUDA(cudaMemcpyAsync(b + o_t, c.reset, n * 8ull, cudaMemcpyHostToDevice, s));
        auto u32 = [&](size_t o) { return reinterpret_cast<uint32_t *>(b + o); };
        auto f64 = [&](size_t o) { return reinterpret_cast<double *>(b + o); };
        SmallArgs a;
        std::memset(&a, 0, sizeof(a));
        a.from = u32(o_from);
        a.to = u32(o_to);
        a.w = c.w ? f64(o_w) : nullptr;
        a.n = n;
        a.m = (uint32_t)c.m;
        a.longest = res_longest_row(n, arcs);
        a.bar_extra = tuning().resident_barrier_extra == 2u ? 1u : 0u;
        a.directed = c.directed ? 1 : 0;
        a.check_w = c.w && c.check_weights ? 1 : 0;
        a.seed = c.kind == RES_EIG ? (c.strength_seed ? 2 : 1) : 0;
        a.in = {u32(o_cnt), u32(o_slot), u32(o_ptr), u32(o_ids), u32(o_bs), u32(o_long)};
        a.outs = {u32(o_cnt2), u32(o_slot2), u32(o_ptr2), u32(o_ids2), u32(o_bs2), u32(o_long2)};
        a.deg = u32(o_deg);
        a.col = u32(o_col);
        a.w64 = f64(o_w64);
        a.dval = f64(o_dval);
        a.start = f64(o_x);
        a.word = u32(o_word);
        a.ctl = reinterpret_cast<Ctl *>(b + o_ctl);
        ResArgs q;
        std::memset(&q, 0, sizeof(q));
        q.row_ptr = a.in.ptr;
        q.col = a.col;
        q.w64 = c.w ? a.w64 : nullptr;
        q.dval = a.dval;
        q.t64 = c.reset ? f64(o_t) : nullptr;
        q.x_out = f64(o_x);
        q.xt[0] = f64(o_xt0);
        q.xt[1] = f64(o_xt1);
        q.bar = u32(o_bar);
        q.rec = reinterpret_cast<double2 *>(b + o_rec);
        q.ctl = a.ctl;
        q.total = arcs + (uint64_t)p.alpha * n;
        q.n = n;
        q.alpha = p.alpha;
        q.max_iter = c.max_iter;
        q.l1hot = 0xFFFFFFFFu;
        q.longest = a.word + 1;
        q.smem = (uint32_t)p.smem;
        q.damping = c.damping;
        q.thr = c.thr;
        q.shift = c.shift;
        void *args[] = {(void *)&a};
        cudaError_t e = cudaLaunchCooperativeKernel((const void *)small_build_kernel, dim3(grid), dim3(kSmallNT), args,
                                                    kSmallSmem, s);
        if (e == cudaErrorCooperativeLaunchTooLarge) {
            cudaGetLastError();
            status = SMALL_NOT_HERE;
        } else {
            PRG_CUDA(e);
            if (p.grid && !launch_resident(c.kind, p, q, s)) status = SMALL_NOT_HERE;
        }
        uint32_t *h_word = reinterpret_cast<uint32_t *>(h + 1);
        auto read_back = [&]() {
            PRG_CUDA(cudaMemcpyAsync(h, a.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
            PRG_CUDA(cudaMemcpyAsync(h_word, a.word, 24, cudaMemcpyDeviceToHost, s));
            PRG_CUDA(cudaStreamSynchronize(s));
        };
        read_back();
        if (status == SMALL_DONE && (h->status == SMALL_NOT_HERE || (!p.grid && h->status == 0))) {
            // not iterated yet: no blind plan, or the kernel found a share too large
            DeviceGraph g;
            g.n = n;
            g.arcs = arcs;
            g.weighted = c.w != nullptr;
            g.row_ptr = a.in.ptr;
            g.max_in_degree = h_word[1];
            const ResPlan again = res_plan(g, c.kind, s);
            if (!again.grid) {
                status = SMALL_NOT_HERE;
            } else {
                q.longest = nullptr;
                q.alpha = again.alpha;
                q.total = arcs + (uint64_t)again.alpha * n;
                PRG_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(Ctl), s));
                if (!launch_resident(c.kind, again, q, s)) status = SMALL_NOT_HERE;
                read_back();
            }
        }
        if (status == SMALL_DONE) {
            if (h->status == 7) throw TimeoutError{"small-graph call: a grid barrier timed out"};
            status = h->status == SMALL_LONG_ROW ? SMALL_NOT_HERE : (SmallStatus)h->status;
            r.max_endpoint = h_word[0];
            r.bad_edge = ~h_word[5];
            r.iterations = h->iters;
            r.eigenvalue = h->dsum[1] > 0.0 ? h->dsum[0] / h->dsum[1] : 0.0;
            if (status == SMALL_DONE) {
                PRG_CUDA(cudaMemcpyAsync(out, b + o_x, n * 8ull, cudaMemcpyDeviceToHost, s));
                PRG_CUDA(cudaStreamSynchronize(s));
            }
        }
    } catch (const CudaError &e) {
        give_up();
        if (e.err != cudaErrorMemoryAllocation) throw;
        cudaGetLastError();
        return SMALL_NOT_HERE;  // (the general path's build takes less where ids have few bits)
    } catch (...) {
        give_up();
        throw;
    }
    if (status == SMALL_NOT_HERE) {
        // the edge list in an allocation of its own: the general path should not
        // have to do without the rest of this one (nor, where even that fails,
        // without anything: it uploads again)
        const size_t ids = (c.m * 4 + 255) & ~(size_t)255, wb = c.w ? c.m * 8 : 0;
        unsigned char *eb = nullptr;
        if (cudaMallocAsync((void **)&eb, 2 * ids + wb, s) == cudaSuccess) {
            cudaMemcpyAsync(eb, b + o_from, c.m * 4, cudaMemcpyDeviceToDevice, s);
            cudaMemcpyAsync(eb + ids, b + o_to, c.m * 4, cudaMemcpyDeviceToDevice, s);
            if (c.w) cudaMemcpyAsync(eb + 2 * ids, b + o_w, wb, cudaMemcpyDeviceToDevice, s);
            r.edges.block = eb;
            r.edges.from = reinterpret_cast<uint32_t *>(eb);
            r.edges.to = reinterpret_cast<uint32_t *>(eb + ids);
            r.edges.w = c.w ? reinterpret_cast<double *>(eb + 2 * ids) : nullptr;
        } else {
            cudaGetLastError();
        }
    }
    cudaFreeAsync(b, s);
    pinned_release(h);
    return status;
}

}  // namespace prg
