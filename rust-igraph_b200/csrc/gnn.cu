// gnn.cu — learned warm start: a small two-layer message-passing network
// that predicts the PageRank vector from degree features.  Its normalised
// output only seeds the solver (prg_solve with a start vector), so the fixed
// point, the stop rule and every correctness check stay those of the plain
// method.
//
// Model (per vertex v, internal ids; s_u = 1/outdeg(u), 0 when dangling):
//   X0[v]  = degree features (16, BF16)
//   H0     = relu(X0 W1^T + b1)                 (32, BF16)   tensor cores
//   M0[u]  = s_u * (H0[u] Wm1^T)                (8, FP32)    tensor cores
//   S1[v]  = sum_{u->v} M0[u],  A1 = slog(S1)   (8 -> BF16)  in-CSR aggregation
//   H1     = relu([H0 | A1] W2^T + b2)          (32, BF16)   tensor cores
//   M1[u]  = s_u * (H1[u] Wm2^T)                (8, FP32)    tensor cores
//   S2[v]  = sum_{u->v} M1[u],  A2 = slog(S2)   (8 -> BF16)
//   y[v]   = [H1 | A2] w3 + b3                  (FP32)       tensor cores
//   start  = exp(y) / sum exp(y)                (FP64)
// The messages carry rank-like mass (scaled by 1/outdeg exactly like the
// power step), so two layers see two hops of the operator; the aggregated
// mass spans orders of magnitude (hubs), so it enters the next layer through
// slog(z) = sign(z) log(1 + |z|).  Dense layers run
// on the tensor cores (mma.sync m16n8k16, BF16 operands, FP32 accumulate).
// Training minimises sum_v w_v (y_v - log(n x*_v))^2 / n with w_v = n x*_v;
// the backward pass is hand-written (FP32 CUDA cores, deterministic block
// partials for the weight gradients, atomics only for the transposed
// aggregation), and Adam updates FP32 master weights, then refreshes the
// BF16 copies the forward pass reads.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gnn.cuh"
#include "prims.cuh"

namespace prg {
namespace gnn {

// ---- parameter layout (FP32 master, flat) --------------------------------
constexpr int kF = 16, kH = 32, kC = 8, kZ = 48;  // features, hidden, message channels, [H|A] width
constexpr int oW1 = 0;                       // [32 x 16]
constexpr int oB1 = oW1 + kH * kF;           // [32]
constexpr int oWm1 = oB1 + kH;               // [8 x 32]
constexpr int oW2 = oWm1 + kC * kH;          // [32 x 48]
constexpr int oB2 = oW2 + kH * kZ;           // [32]
constexpr int oWm2 = oB2 + kH;               // [8 x 32]
constexpr int oW3 = oWm2 + kC * kH;          // [8 x 48] (row 0 used)
constexpr int oB3 = oW3 + 8 * kZ;            // [8]      (entry 0 used)
constexpr int kParams = oB3 + 8;             // 3016

// one row of weight-gradient partials per block of the backward passes (the
// first two blocks per SM, the second up to four)
constexpr unsigned kTopBlocks = 148 * 2, kBottomBlocks = 148 * 4;
constexpr int kPartStride = 3072;
static_assert(kPartStride >= kParams, "partials");

struct Ws {  // BF16 copies of the weight matrices
    __nv_bfloat16 W1[kH * kF], Wm1[kC * kH], W2[kH * kZ], Wm2[kC * kH], W3[8 * kZ];
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&p);
}

// ---- features --------------------------------------------------------------
__global__ void features_kernel(uint32_t n, const uint32_t *row_ptr, const uint32_t *deg, __nv_bfloat16 *X0) {
    const float ln = logf((float)n) * 0.0625f;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const float li = log1pf((float)(row_ptr[v + 1] - row_ptr[v]));
        const float lo = log1pf((float)deg[v]);
        float f[kF];
#pragma unroll
        for (int i = 0; i < kF; i++) f[i] = 0.0f;
        f[0] = li * 0.125f;
        f[1] = lo * 0.125f;
        f[2] = deg[v] == 0 ? 1.0f : 0.0f;
        f[3] = 1.0f;
        f[4] = (li - lo) * 0.125f;
        f[5] = ln;
        uint4 *dst = reinterpret_cast<uint4 *>(X0 + (size_t)v * kF);
        dst[0] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
        dst[1] = make_uint4(pack_bf16(f[8], f[9]), pack_bf16(f[10], f[11]), pack_bf16(f[12], f[13]),
                            pack_bf16(f[14], f[15]));
    }
}

// ---- rowwise dense layer on the tensor cores --------------------------------
// Y[v][0..N) = sum_k A[v][k] W[j][k] for 16-row tiles per warp.  A is the
// concatenation [A0 (K0 cols) | A1 (K1 cols)] (BF16, row-major); W is
// [N x (K0+K1)] BF16 row-major (= the B operand in column-major k x n).
// Fragment layout of mma.m16n8k16 (PTX ISA): group g = lane/4, t = lane%4;
// A regs: (g, 2t..2t+1), (g+8, 2t..), (g, 2t+8..), (g+8, 2t+8..);
// B regs: (k=2t..2t+1, n=g), (k=2t+8.., n=g); C: (g, 2t..2t+1), (g+8, 2t..).
enum Epi { EPI_RELU_BF16 = 0, EPI_SCALE_F32 = 1, EPI_COL0_F32 = 2 };

template <int K0, int K1, int N, int EPI>
__global__ void __launch_bounds__(128) rowwise_kernel(uint32_t n, const __nv_bfloat16 *A0, const __nv_bfloat16 *A1,
                                                      const __nv_bfloat16 *W, const float *bias, const float *scale,
                                                      __nv_bfloat16 *out_bf, float *out_f) {
    constexpr int K = K0 + K1;
    static_assert(K % 16 == 0 && N % 8 == 0, "mma tile shape");
    __shared__ __align__(16) __nv_bfloat16 sW[N * K];
    for (int i = threadIdx.x; i < N * K; i += blockDim.x) sW[i] = W[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t ntiles = (n + 15) / 16;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t tile = warp; tile < ntiles; tile += nwarps) {
        const uint32_t r0 = tile * 16 + g, r1 = r0 + 8;
        float acc[N / 8][4];
#pragma unroll
        for (int j = 0; j < N / 8; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
        for (int kt = 0; kt < K / 16; kt++) {
            // A fragment (rows beyond n read as zero)
            const int kb = kt * 16;
            uint32_t a[4];
            auto ldA = [&](uint32_t r, int k) -> uint32_t {
                if (r >= n) return 0u;
                if (k < K0) return *reinterpret_cast<const uint32_t *>(A0 + (size_t)r * K0 + k);
                return *reinterpret_cast<const uint32_t *>(A1 + (size_t)r * K1 + (k - K0));
            };
            a[0] = ldA(r0, kb + 2 * t);
            a[1] = ldA(r1, kb + 2 * t);
            a[2] = ldA(r0, kb + 2 * t + 8);
            a[3] = ldA(r1, kb + 2 * t + 8);
#pragma unroll
            for (int j = 0; j < N / 8; j++) {
                const int col = j * 8 + g;
                const uint32_t b0 = *reinterpret_cast<const uint32_t *>(sW + col * K + kb + 2 * t);
                const uint32_t b1 = *reinterpret_cast<const uint32_t *>(sW + col * K + kb + 2 * t + 8);
                asm volatile(
                    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                    "{%0,%1,%2,%3};"
                    : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
            }
        }
        // epilogue: C(g, 2t..), C(g+8, 2t..) of each n-tile
#pragma unroll
        for (int j = 0; j < N / 8; j++) {
            const int c0 = j * 8 + 2 * t;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t r = h ? r1 : r0;
                if (r >= n) continue;
                float v0 = acc[j][2 * h], v1 = acc[j][2 * h + 1];
                if constexpr (EPI == EPI_RELU_BF16) {
                    v0 = fmaxf(v0 + bias[c0], 0.0f);
                    v1 = fmaxf(v1 + bias[c0 + 1], 0.0f);
                    *reinterpret_cast<uint32_t *>(out_bf + (size_t)r * N + c0) = pack_bf16(v0, v1);
                } else if constexpr (EPI == EPI_SCALE_F32) {
                    const float sc = scale[r];
                    out_f[(size_t)r * N + c0] = v0 * sc;
                    out_f[(size_t)r * N + c0 + 1] = v1 * sc;
                } else {
                    if (c0 == 0) out_f[r] = v0 + bias[0];
                }
            }
        }
    }
}

template <int K0, int K1, int N, int EPI>
static void rowwise(uint32_t n, const __nv_bfloat16 *A0, const __nv_bfloat16 *A1, const __nv_bfloat16 *W,
                    const float *bias, const float *scale, __nv_bfloat16 *out_bf, float *out_f, cudaStream_t s) {
    const uint32_t tiles = (n + 15) / 16;
    const unsigned grid = (unsigned)std::min<uint32_t>((tiles + 3) / 4, 148u * 16u);
    rowwise_kernel<K0, K1, N, EPI><<<std::max(grid, 1u), 128, 0, s>>>(n, A0, A1, W, bias, scale, out_bf, out_f);
    PRG_CUDA(cudaGetLastError());
}

// ---- aggregation A[v] = sum_{u->v} M[u] (8 channels) ------------------------
// Rows of up to kAggHeavy arcs: 8 lanes per row, each lane takes every 8th
// arc and gathers the source's 32-byte message; lanes combine with shuffles.
// Longer rows are queued and summed by a whole block each.
constexpr uint32_t kAggHeavy = 2048;

__device__ __forceinline__ float slog(float z) { return copysignf(log1pf(fabsf(z)), z); }

// One source's 8-channel message (32-byte aligned) in one load: two 16-byte
// loads would look the same sector up twice in L1.
__device__ __forceinline__ void ld_msg(const float *p, float (&q)[kC]) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(q[0]), "=f"(q[1]), "=f"(q[2]), "=f"(q[3]), "=f"(q[4]), "=f"(q[5]), "=f"(q[6]), "=f"(q[7])
        : "l"(p));
}

// The sources of arcs p, p + STRIDE, ... below p1, kAggAhead of them.
constexpr int kAggAhead = 4;
template <uint32_t STRIDE>
__device__ __forceinline__ void ld_sources(const uint32_t *col, uint32_t p, uint32_t p1, uint32_t (&u)[kAggAhead]) {
#pragma unroll
    for (int i = 0; i < kAggAhead; i++) u[i] = p + i * STRIDE < p1 ? __ldg(&col[p + i * STRIDE]) : 0u;
}

// acc += the messages of arcs p, p + STRIDE, ... below p1, added one by one in
// that order, with kAggAhead of them in flight.  u: the first sources, loaded
// before; while the last messages are in flight it takes those of the arcs from
// q on, below q1 (the next row's).
template <uint32_t STRIDE>
__device__ __forceinline__ void add_messages(float (&acc)[kC], uint32_t p, uint32_t p1, const uint32_t *col,
                                             const float *M, uint32_t (&u)[kAggAhead], uint32_t q, uint32_t q1) {
    bool more;
    do {
        float m[kAggAhead][kC];
#pragma unroll
        for (int i = 0; i < kAggAhead; i++)
            if (p + i * STRIDE < p1) ld_msg(M + (size_t)u[i] * kC, m[i]);
        const uint32_t at = p;
        p += STRIDE * kAggAhead;
        more = p < p1;
        ld_sources<STRIDE>(col, more ? p : q, more ? p1 : q1, u);
#pragma unroll
        for (int i = 0; i < kAggAhead; i++)
            if (at + i * STRIDE < p1) {
#pragma unroll
                for (int c = 0; c < kC; c++) acc[c] += m[i][c];
            }
    } while (more);
}

// The sums of acc over a row's 8 lanes; lane `sub` gets channel `sub`.  At each
// step a lane keeps half of its channels and gives the others away: 7 shuffles
// instead of 3 per channel, each sum added in the same order.
__device__ __forceinline__ float row_channel(const float (&acc)[kC], uint32_t sub) {
    float a[4], b[2];
    const bool up4 = (sub & 4u) != 0u, up2 = (sub & 2u) != 0u, up1 = (sub & 1u) != 0u;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const float got = __shfl_xor_sync(0xffffffffu, up4 ? acc[c] : acc[c + 4], 4);
        a[c] = (up4 ? acc[c + 4] : acc[c]) + got;
    }
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const float got = __shfl_xor_sync(0xffffffffu, up2 ? a[c] : a[c + 2], 2);
        b[c] = (up2 ? a[c + 2] : a[c]) + got;
    }
    const float got = __shfl_xor_sync(0xffffffffu, up1 ? b[0] : b[1], 1);
    return (up1 ? b[1] : b[0]) + got;
}

// Rows of more than kAggHeavy arcs, listed once per forward pass.
__global__ void heavy_rows_kernel(uint32_t n, const uint32_t *row_ptr, uint32_t *heavy, uint32_t *nheavy) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        if (row_ptr[v + 1] - row_ptr[v] > kAggHeavy) heavy[atomicAdd(nheavy, 1u)] = v;
}

// out: slog of the sums in BF16, 16 columns of which the last 8 are zero;
// out_f (null: not wanted): the sums themselves.
// The first kAggHeavyBlocks blocks take the heavy rows, one at a time, the others
// the light rows, 8 lanes per row: the longest hub's chain of loads (0.2 ms on
// R-MAT s22) runs beside the light rows instead of after them in a launch of its
// own.
constexpr unsigned kAggHeavyBlocks = 148 * 2, kAggLightBlocks = 148 * 16;
__global__ void __launch_bounds__(256, 4) aggregate_kernel(uint32_t n, const uint32_t *row_ptr, const uint32_t *col,
                                                           const float *M, __nv_bfloat16 *out, float *out_f,
                                                           const uint32_t *heavy, const uint32_t *nheavy) {
    __shared__ float sh[kC][32];
    if (blockIdx.x < kAggHeavyBlocks) {
        const uint32_t cnt = *nheavy;
        for (uint32_t i = blockIdx.x; i < cnt; i += kAggHeavyBlocks) {
            const uint32_t v = heavy[i];
            const uint32_t p0 = row_ptr[v], p1 = row_ptr[v + 1];
            float acc[kC];
#pragma unroll
            for (int c = 0; c < kC; c++) acc[c] = 0.0f;
            uint32_t u[kAggAhead];
            ld_sources<256>(col, p0 + threadIdx.x, p1, u);
            add_messages<256>(acc, p0 + threadIdx.x, p1, col, M, u, 0u, 0u);
            const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
            for (int c = 0; c < kC; c++) acc[c] = warp_sum(acc[c]);
            __syncthreads();
            if (l == 0)
                for (int c = 0; c < kC; c++) sh[c][w] = acc[c];
            __syncthreads();
            if (threadIdx.x < kC) {
                float tot = 0.0f;
                for (int k = 0; k < (int)(blockDim.x >> 5); k++) tot += sh[threadIdx.x][k];
                out[(size_t)v * 16 + threadIdx.x] = __float2bfloat16_rn(slog(tot));
                out[(size_t)v * 16 + 8 + threadIdx.x] = __float2bfloat16_rn(0.0f);
                if (out_f) out_f[(size_t)v * kC + threadIdx.x] = tot;
            }
        }
        return;
    }
    const uint32_t gid = (blockIdx.x - kAggHeavyBlocks) * blockDim.x + threadIdx.x, sub = threadIdx.x & 7;
    const uint32_t group = gid >> 3, ngroups = ((gridDim.x - kAggHeavyBlocks) * blockDim.x) >> 3;
    const uint32_t rounds = (n + ngroups - 1) / ngroups;
    // A row's arcs as an empty range when another block sums it (or there is no
    // such row).  Row ends are read two rows ahead and a row's first sources one
    // ahead, so a row waits for its messages alone, not for the chain of row
    // end, source and message (0.5 M vertices, 3 M arcs 53 us a layer with the
    // chain, 45 without; R-MAT s22, where L1's data pipe is the bound, 488 and
    // 485: a lookup per message, the messages' bytes and the shuffles share it,
    // 82 % busy with three shuffles per channel, 525 us).
    auto row = [&](uint64_t v, uint32_t &p0, uint32_t &p1) {
        p0 = p1 = 0u;
        if (v < n) {
            p0 = __ldg(&row_ptr[v]);
            p1 = __ldg(&row_ptr[v + 1]);
        }
    };
    uint32_t p0, p1, n0, n1, u[kAggAhead];
    row(group, p0, p1);
    row((uint64_t)group + ngroups, n0, n1);
    bool heavy_row = p1 - p0 > kAggHeavy;
    if (heavy_row) p1 = p0;
    ld_sources<8>(col, p0 + sub, p1, u);
    for (uint32_t rd = 0; rd < rounds; rd++) {
        const uint32_t v = rd * ngroups + group;
        float acc[kC];
#pragma unroll
        for (int c = 0; c < kC; c++) acc[c] = 0.0f;
        uint32_t f0, f1;
        row(v + 2ull * ngroups, f0, f1);
        const bool skip = v >= n || heavy_row;
        const bool next_heavy = n1 - n0 > kAggHeavy;
        add_messages<8>(acc, p0 + sub, p1, col, M, u, n0 + sub, next_heavy ? 0u : n1);
        const bool some = p1 > p0;
        p0 = n0;
        p1 = next_heavy ? n0 : n1;
        heavy_row = next_heavy;
        n0 = f0;
        n1 = f1;
        const float mine = __any_sync(0xffffffffu, some) ? row_channel(acc, sub) : 0.0f;
        const float z = slog(mine), zn = __shfl_xor_sync(0xffffffffu, z, 1);
        if (!skip) {
            uint32_t *dst = reinterpret_cast<uint32_t *>(out + (size_t)v * 16);
            if ((sub & 1u) == 0u) dst[sub >> 1] = pack_bf16(z, zn);
            else dst[4 + (sub >> 1)] = 0u;
            if (out_f) out_f[(size_t)v * kC + sub] = mine;
        }
    }
}

// ---- prediction --------------------------------------------------------------
__global__ void max_kernel(const float *y, uint32_t n, float *part) {
    float m = -INFINITY;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) m = fmaxf(m, y[v]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float sh[32];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); i++) m = fmaxf(m, sh[i]);
        m = fmaxf(m, sh[0]);
        part[blockIdx.x] = m;
    }
}

__global__ void expsum_kernel(const float *y, uint32_t n, const float *mpart, unsigned nm, double *x, double *part) {
    float m = -INFINITY;
    for (unsigned i = 0; i < nm; i++) m = fmaxf(m, mpart[i]);
    double s = 0.0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const double e = exp((double)(y[v] - m));
        x[v] = e;
        s += e;
    }
    __shared__ double sh[32];
    s = block_sum<double>(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void normalise_kernel(double *x, uint32_t n, const double *part, unsigned np) {
    double s = 0.0;
    for (unsigned i = 0; i < np; i++) s += part[i];
    const double inv = 1.0 / s;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) x[v] *= inv;
}

__global__ void scale_kernel(const uint32_t *deg, uint32_t n, float *s) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        s[v] = deg[v] ? 1.0f / (float)deg[v] : 0.0f;
}

// ---- loss ------------------------------------------------------------------
// target x* in internal ids; L = sum_v w_v (y_v - t_v)^2 / n, w_v = n x*_v; and
// the gradient through the output layer's aggregated half,
// dS2 = dy w3[H..] / (1 + |S2|) (slog'(S) = 1 / (1 + |S|)).
__global__ void loss_kernel(const float *y, const double *xs, uint32_t n, const float *P, const float *S2, float *dy,
                            float *dS2, double *part) {
    double l = 0.0;
    const double nn = (double)n;
    float w3[kC];
#pragma unroll
    for (int c = 0; c < kC; c++) w3[c] = P[oW3 + kH + c];
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const double xv = xs[v] > 1e-300 ? xs[v] : 1e-300;
        const double w = nn * xv, tv = log(nn * xv);
        const double e = (double)y[v] - tv;
        l += w * e * e;
        const float g = (float)(2.0 * w * e / nn);
        dy[v] = g;
        float s[kC];
        *reinterpret_cast<float4 *>(s) = *reinterpret_cast<const float4 *>(S2 + (size_t)v * kC);
        *reinterpret_cast<float4 *>(s + 4) = *reinterpret_cast<const float4 *>(S2 + (size_t)v * kC + 4);
#pragma unroll
        for (int c = 0; c < kC; c++) s[c] = g * w3[c] / (1.0f + fabsf(s[c]));
        *reinterpret_cast<float4 *>(dS2 + (size_t)v * kC) = *reinterpret_cast<const float4 *>(s);
        *reinterpret_cast<float4 *>(dS2 + (size_t)v * kC + 4) = *reinterpret_cast<const float4 *>(s + 4);
    }
    __shared__ double sh[32];
    l = block_sum<double>(l, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = l / nn;
}

// ---- backward (FP32 CUDA cores) -----------------------------------------------
// Transposed aggregation, dM[u] += dS[v] over every in-arc u -> v.  16 lanes per
// row: 8 arcs at a time, two lanes per arc adding four channels each with one
// 16-byte reduction (one thread per row and one 4-byte atomic per channel took
// 0.48 ms on 0.5 M vertices and 3 M arcs, this 0.04).  Rows of more than
// kAggHeavy arcs are skipped: scatter_heavy_kernel spreads them over blocks.
__device__ __forceinline__ void red_add4(float *p, const float4 &g) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(g.x), "f"(g.y), "f"(g.z),
                 "f"(g.w)
                 : "memory");
}

__global__ void scatter_kernel(uint32_t n, const uint32_t *row_ptr, const uint32_t *col, const float *dS, float *dM) {
    const uint32_t sub = (threadIdx.x & 15) >> 1, half = threadIdx.x & 1;
    const uint32_t ngroups = (gridDim.x * blockDim.x) >> 4;
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; v < n; v += ngroups) {
        const uint32_t p0 = row_ptr[v], p1 = row_ptr[v + 1];
        if (p1 == p0 || p1 - p0 > kAggHeavy) continue;
        const float4 g = __ldg(reinterpret_cast<const float4 *>(dS + (size_t)v * kC) + half);
        for (uint32_t p = p0 + sub; p < p1; p += 8) red_add4(dM + (size_t)__ldg(&col[p]) * kC + half * 4, g);
    }
}

__global__ void scatter_heavy_kernel(const uint32_t *row_ptr, const uint32_t *col, const float *dS, float *dM,
                                     const uint32_t *heavy, const uint32_t *nheavy) {
    const uint32_t cnt = *nheavy, half = threadIdx.x & 1;
    for (uint32_t i = 0; i < cnt; i++) {
        const uint32_t v = heavy[i], p0 = row_ptr[v], p1 = row_ptr[v + 1];
        const float4 g = __ldg(reinterpret_cast<const float4 *>(dS + (size_t)v * kC) + half);
        for (uint32_t p = p0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 1); p < p1; p += (gridDim.x * blockDim.x) >> 1)
            red_add4(dM + (size_t)__ldg(&col[p]) * kC + half * 4, g);
    }
}

// The two dense backward passes: one warp per vertex, lane k on hidden unit k,
// kVB vertices per step.  Everything a vertex contributes (its own gradients and
// its share of the weight gradients) is computed while its rows are on chip:
// reading per-layer buffers back for separate outer-product and matrix kernels
// took 2.4 ms on 0.5 M vertices (a thread per vertex walked 128-byte rows).  The
// rows of the next step arrive by cp.async while a step is computed (without
// that the passes waited for memory: 306 + 159 us).  What bounds them then is
// FP32 issue, about 170 instructions per vertex and warp in the first.
// Weight-gradient sums stay in registers over the warp's vertices, are added over
// the block's warps in shared memory in warp order, and leave one partial per
// block for reduce_part_kernel, so everything but the atomic scatters is
// deterministic.
constexpr int kVB = 4;
constexpr int kBwdThreads = 256, kBwdWarps = kBwdThreads / 32;

// 8 consecutive BF16 (16-byte aligned) of shared memory as floats
__device__ __forceinline__ void ld_bf8s(const unsigned char *p, float (&f)[8]) {
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}
__device__ __forceinline__ void cp16(unsigned char *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__device__ __forceinline__ float bf(const __nv_bfloat16 &x) { return __bfloat162float(x); }

// acc (one per lane) summed over the block's warps in warp order into out[lane]
__device__ __forceinline__ void block_lane_sum(float acc, float (*sh)[32], float *out) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    sh[w][l] = acc;
    __syncthreads();
    if (w == 0) {
        float t = sh[0][l];
        for (int k = 1; k < kBwdWarps; k++) t += sh[k][l];
        out[l] = t;
    }
}

// Output layer, second message layer and second hidden layer:
//   dPre1 = relu'(H1) (dy w3 + (s dM1) Wm2);  dZ1 = dPre1 W2 = [dH0 | dA1];
//   dS1 = dA1 / (1 + |S1|); partial gradients of w3, b3, Wm2, W2, b2.
__global__ void __launch_bounds__(kBwdThreads, 2) bwd_top_kernel(
    uint32_t n, const float *dy, const float *dM1, const float *s, const float *P, const __nv_bfloat16 *H1,
    const __nv_bfloat16 *A2, const __nv_bfloat16 *H0, const __nv_bfloat16 *A1, const float *S1, float *dH0, float *dS1,
    float *part) {
    __shared__ float sW2[kH][kH + kC];                         // W2[j][k], k < 40 (the rest meets zero padding)
    __shared__ __align__(16) float sD[kBwdWarps][kH][kVB];     // dPre1 of the warp's vertices
    __shared__ float sRed[kBwdWarps][32], sLast[32];
    // the rows of kVB vertices: per vertex H1 64 | H0 64 | dM1 32 | S1 32 | A1 16 | A2 16, then dy and s
    constexpr int kRow = 224, kStage = kVB * kRow + 32;
    __shared__ __align__(16) unsigned char sIn[kBwdWarps][2][kStage];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kH * (kH + kC); i += kBwdThreads)
        sW2[i / (kH + kC)][i % (kH + kC)] = P[oW2 + (i / (kH + kC)) * kZ + i % (kH + kC)];
    float wm[kC];
#pragma unroll
    for (int c = 0; c < kC; c++) wm[c] = P[oWm2 + c * kH + lane];
    const float w3 = P[oW3 + lane];
    __syncthreads();
    float aW2[kH + kC], aWm[kC], aW3h = 0.0f, aW3a = 0.0f, aB2 = 0.0f, aB3 = 0.0f;
#pragma unroll
    for (int i = 0; i < kH + kC; i++) aW2[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < kC; c++) aWm[c] = 0.0f;
    const uint32_t stride = gridDim.x * kBwdWarps * kVB;
    auto fetch = [&](uint32_t v0, int st) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int q = lane + 32 * i, b = q / 14, part_ = q % 14;
            const uint32_t v = v0 + b;
            if (q < 14 * kVB) {
                if (v >= n) continue;
                const void *src;
                if (part_ < 4) src = H1 + (size_t)v * kH + part_ * 8;
                else if (part_ < 8) src = H0 + (size_t)v * kH + (part_ - 4) * 8;
                else if (part_ < 10) src = dM1 + (size_t)v * kC + (part_ - 8) * 4;
                else if (part_ < 12) src = S1 + (size_t)v * kC + (part_ - 10) * 4;
                else src = (part_ == 12 ? A1 : A2) + (size_t)v * 16;
                cp16(&sIn[w][st][b * kRow + part_ * 16], src);
            } else if (q < 14 * kVB + 2 && v0 < n) {
                // (the buffers are padded to 256 bytes, so four values can be read at any v0 < n)
                cp16(&sIn[w][st][kVB * kRow + (q - 14 * kVB) * 16], (q == 14 * kVB ? dy : s) + v0);
            }
        }
        cp_commit();
    };
    uint32_t v0 = (blockIdx.x * kBwdWarps + w) * kVB;
    fetch(v0, 0);
    for (int st = 0; v0 < n; v0 += stride, st ^= 1) {
        __syncwarp();  // the other stage is no longer read
        fetch(v0 + stride, st ^ 1);
        cp_wait1();
        __syncwarp();
        const unsigned char *in = sIn[w][st];
        const float4 dy4 = *reinterpret_cast<const float4 *>(in + kVB * kRow);
        const float4 s4 = *reinterpret_cast<const float4 *>(in + kVB * kRow + 16);
        const float dyv[kVB] = {dy4.x, dy4.y, dy4.z, dy4.w}, sv[kVB] = {s4.x, s4.y, s4.z, s4.w};
        float d[kVB];
#pragma unroll
        for (int b = 0; b < kVB; b++) {
            d[b] = 0.0f;
            if (v0 + b >= n) continue;  // warp-uniform
            const unsigned char *row = in + b * kRow;
            const float g = dyv[b], sc = sv[b], h = bf(reinterpret_cast<const __nv_bfloat16 *>(row)[lane]);
            const float4 m0 = *reinterpret_cast<const float4 *>(row + 128);
            const float4 m1 = *reinterpret_cast<const float4 *>(row + 144);
            const float gm[kC] = {m0.x * sc, m0.y * sc, m0.z * sc, m0.w * sc, m1.x * sc, m1.y * sc, m1.z * sc, m1.w * sc};
            float t = g * w3;
#pragma unroll
            for (int c = 0; c < kC; c++) {
                t += gm[c] * wm[c];
                aWm[c] += gm[c] * h;
            }
            d[b] = h > 0.0f ? t : 0.0f;
            aB2 += d[b];
            aW3h += g * h;
            if (lane < kC) aW3a += g * bf(reinterpret_cast<const __nv_bfloat16 *>(row + 208)[lane]);
            if (lane == 0) aB3 += g;
        }
        __syncwarp();
        *reinterpret_cast<float4 *>(&sD[w][lane][0]) = make_float4(d[0], d[1], d[2], d[3]);
        __syncwarp();
        // dW2[lane][i] += dPre1[lane] Z1[i]
#pragma unroll
        for (int b = 0; b < kVB; b++) {
            const uint32_t v = v0 + b;
            if (v >= n) continue;
#pragma unroll
            for (int q = 0; q < kH / 8 + 1; q++) {
                float z[8];
                ld_bf8s(in + b * kRow + (q < kH / 8 ? 64 + q * 16 : 192), z);
#pragma unroll
                for (int i = 0; i < 8; i++) aW2[q * 8 + i] += d[b] * z[i];
            }
        }
        // dZ1: hidden unit `lane`, and channel lane & 7 from a quarter of the units
        float z[kVB] = {0.0f, 0.0f, 0.0f, 0.0f}, zc[kVB] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int j = 0; j < kH; j++) {
            const float4 q = *reinterpret_cast<const float4 *>(&sD[w][j][0]);
            const float wj = sW2[j][lane];
            z[0] += q.x * wj;
            z[1] += q.y * wj;
            z[2] += q.z * wj;
            z[3] += q.w * wj;
        }
#pragma unroll
        for (int i = 0; i < kH / 4; i++) {
            const int j = (lane >> 3) * (kH / 4) + i;
            const float4 q = *reinterpret_cast<const float4 *>(&sD[w][j][0]);
            const float wj = sW2[j][kH + (lane & 7)];
            zc[0] += q.x * wj;
            zc[1] += q.y * wj;
            zc[2] += q.z * wj;
            zc[3] += q.w * wj;
        }
#pragma unroll
        for (int b = 0; b < kVB; b++) {
            zc[b] += __shfl_xor_sync(0xffffffffu, zc[b], 8);
            zc[b] += __shfl_xor_sync(0xffffffffu, zc[b], 16);
            const uint32_t v = v0 + b;
            if (v >= n) continue;
            dH0[(size_t)v * kH + lane] = z[b];
            if (lane < kC) dS1[(size_t)v * kC + lane] =
                              zc[b] / (1.0f + fabsf(reinterpret_cast<const float *>(in + b * kRow + 160)[lane]));
        }
    }
    float *out = part + (size_t)blockIdx.x * kPartStride;
#pragma unroll
    for (int i = 0; i < kH + kC; i++) {
        // W2 is [lane][i]: transposed through the block sum
        const int wi = threadIdx.x >> 5;
        __syncthreads();
        sRed[wi][lane] = aW2[i];
        __syncthreads();
        if (wi == 0) {
            float t = sRed[0][lane];
            for (int k = 1; k < kBwdWarps; k++) t += sRed[k][lane];
            out[oW2 + lane * kZ + i] = t;
        }
    }
#pragma unroll
    for (int c = 0; c < kC; c++) block_lane_sum(aWm[c], sRed, out + oWm2 + c * kH);
    block_lane_sum(aB2, sRed, out + oB2);
    block_lane_sum(aW3h, sRed, out + oW3);
    const float b3 = __shfl_sync(0xffffffffu, aB3, 0);
    block_lane_sum(lane < kC ? aW3a : lane == kC ? b3 : 0.0f, sRed, sLast);
    __syncthreads();
    if (threadIdx.x < kC) out[oW3 + kH + threadIdx.x] = sLast[threadIdx.x];
    if (threadIdx.x == kC) out[oB3] = sLast[kC];
}

// First message layer and first hidden layer:
//   dPre0 = relu'(H0) (dH0 + (s dM0) Wm1); partial gradients of Wm1, W1, b1.
__global__ void __launch_bounds__(kBwdThreads) bwd_bottom_kernel(uint32_t n, const float *dM0, const float *s,
                                                                 const float *P, const __nv_bfloat16 *H0,
                                                                 const __nv_bfloat16 *X0, const float *dH0,
                                                                 float *part) {
    __shared__ float sRed[kBwdWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float wm[kC], aWm[kC], aW1[8], aB1 = 0.0f;
#pragma unroll
    for (int c = 0; c < kC; c++) {
        wm[c] = P[oWm1 + c * kH + lane];
        aWm[c] = aW1[c] = 0.0f;
    }
    // per vertex dH0 128 | H0 64 | dM0 32 | X0 16 (features 6 .. 15 are zero), then s
    constexpr int kRow = 240, kStage = kVB * kRow + 16;
    __shared__ __align__(16) unsigned char sIn[kBwdWarps][2][kStage];
    const uint32_t stride = gridDim.x * kBwdWarps * kVB;
    auto fetch = [&](uint32_t v0, int st) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int q = lane + 32 * i, b = q / 15, part_ = q % 15;
            const uint32_t v = v0 + b;
            if (q < 15 * kVB) {
                if (v >= n) continue;
                const void *src;
                if (part_ < 8) src = dH0 + (size_t)v * kH + part_ * 4;
                else if (part_ < 12) src = H0 + (size_t)v * kH + (part_ - 8) * 8;
                else if (part_ < 14) src = dM0 + (size_t)v * kC + (part_ - 12) * 4;
                else src = X0 + (size_t)v * kF;
                cp16(&sIn[w][st][b * kRow + part_ * 16], src);
            } else if (q == 15 * kVB && v0 < n) {
                cp16(&sIn[w][st][kVB * kRow], s + v0);
            }
        }
        cp_commit();
    };
    uint32_t v0 = (blockIdx.x * kBwdWarps + w) * kVB;
    fetch(v0, 0);
    for (int st = 0; v0 < n; v0 += stride, st ^= 1) {
        __syncwarp();
        fetch(v0 + stride, st ^ 1);
        cp_wait1();
        __syncwarp();
        const unsigned char *in = sIn[w][st];
        const float4 s4 = *reinterpret_cast<const float4 *>(in + kVB * kRow);
        const float sv[kVB] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
        for (int b = 0; b < kVB; b++) {
            if (v0 + b >= n) continue;
            const unsigned char *row = in + b * kRow;
            const float sc = sv[b], h = bf(reinterpret_cast<const __nv_bfloat16 *>(row + 128)[lane]);
            const float4 m0 = *reinterpret_cast<const float4 *>(row + 192);
            const float4 m1 = *reinterpret_cast<const float4 *>(row + 208);
            const float gm[kC] = {m0.x * sc, m0.y * sc, m0.z * sc, m0.w * sc, m1.x * sc, m1.y * sc, m1.z * sc, m1.w * sc};
            float t = reinterpret_cast<const float *>(row)[lane];
#pragma unroll
            for (int c = 0; c < kC; c++) {
                t += gm[c] * wm[c];
                aWm[c] += gm[c] * h;
            }
            const float d = h > 0.0f ? t : 0.0f;
            aB1 += d;
            float x[8];
            ld_bf8s(row + 224, x);
#pragma unroll
            for (int i = 0; i < 8; i++) aW1[i] += d * x[i];
        }
    }
    float *out = part + (size_t)blockIdx.x * kPartStride;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        __syncthreads();
        sRed[w][lane] = aW1[i];
        __syncthreads();
        if (w == 0) {
            float t = sRed[0][lane];
            for (int k = 1; k < kBwdWarps; k++) t += sRed[k][lane];
            out[oW1 + lane * kF + i] = t;
        }
    }
#pragma unroll
    for (int c = 0; c < kC; c++) block_lane_sum(aWm[c], sRed, out + oWm1 + c * kH);
    block_lane_sum(aB1, sRed, out + oB1);
}

// grad[i] = sum over blocks of part[b][i] in FP64: 32 parameters x 8 slices of
// the blocks per thread block, the slices added in order.
__global__ void __launch_bounds__(256) reduce_part_kernel(const float *part, unsigned nb_bottom, unsigned nb_top,
                                                          float *grad) {
    __shared__ double sh[8][32];
    const int l = threadIdx.x & 31, q = threadIdx.x >> 5, i = blockIdx.x * 32 + l;
    // slots no backward pass writes: W1's columns past the features it sees,
    // W2's zero padding, W3's unused rows and b3's unused entries
    bool used = i < kParams;
    if (i < oB1) used = i % kF < 8;
    else if (i >= oW2 && i < oB2) used = (i - oW2) % kZ < kH + kC;
    else if (i >= oW3 && i < oB3) used = i < oW3 + kH + kC;
    else if (i >= oB3) used = i == oB3;
    const unsigned nb = i < oW2 ? nb_bottom : nb_top;
    double s = 0.0;
    if (used)
        for (unsigned b = q; b < nb; b += 8) s += part[(size_t)b * kPartStride + i];
    sh[q][l] = s;
    __syncthreads();
    if (q == 0 && i < kParams) {
        for (int k = 1; k < 8; k++) s += sh[k][l];
        grad[i] = (float)s;
    }
}

__global__ void adam_kernel(float *P, const float *G, float *m, float *v, int count, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float g = G[i];
        const float mi = b1 * m[i] + (1.0f - b1) * g;
        const float vi = b2 * v[i] + (1.0f - b2) * g * g;
        m[i] = mi;
        v[i] = vi;
        P[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

__global__ void to_bf16_kernel(const float *P, Ws *w) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kH * kF) w->W1[i] = __float2bfloat16_rn(P[oW1 + i]);
    if (i < kC * kH) w->Wm1[i] = __float2bfloat16_rn(P[oWm1 + i]);
    if (i < kH * kZ) w->W2[i] = __float2bfloat16_rn(P[oW2 + i]);
    if (i < kC * kH) w->Wm2[i] = __float2bfloat16_rn(P[oWm2 + i]);
    if (i < 8 * kZ) w->W3[i] = __float2bfloat16_rn(P[oW3 + i]);
}


// ---- fused inference path ---------------------------------------------------
// The same layer chain as the forward pass above, with the hidden layers kept
// in registers: the FP32 accumulator fragments of one mma.m16n8k16 are the
// BF16 A-operand fragments of the next layer once packed (C tile 2k / 2k+1
// of n-columns 16k..16k+15 -> A registers {0,1} / {2,3} of k-tile k), so H0
// and H1 never reach memory (they are recomputed where needed).  The
// rounding points and the mma sequence are those of rowwise_kernel, so the
// prediction is that of the training forward pass.

// Features 2t, 2t + 1 of a vertex in BF16 (features_kernel's, zero from 6 on),
// from li = log1p(in-degree), lo = log1p(out-degree).
__device__ __forceinline__ uint32_t feat_pair(int t, float li, float lo, float ln, bool dangling) {
    const uint32_t f01 = pack_bf16(li * 0.125f, lo * 0.125f), f45 = pack_bf16((li - lo) * 0.125f, ln);
    const uint32_t f23 = dangling ? 0x3F803F80u : 0x3F800000u;  // (dangling ? 1 : 0, 1)
    return t == 0 ? f01 : t == 1 ? f23 : t == 2 ? f45 : 0u;
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// B fragments of W [8 NT x K] (row-major, k-tiles from kt0): two registers per
// n-tile and k-tile, loaded once per thread (a warp's weight tiles read from
// shared memory in every row tile kept the L1 data pipe 81 % busy with 2- and
// 4-way bank conflicts: 95 / 156 / 156 us per stage on R-MAT s22).
template <int NT, int KT>
struct BFrag {
    uint32_t b[KT][NT][2];
    __device__ __forceinline__ void load(const __nv_bfloat16 *W, int K, int g, int t) {
#pragma unroll
        for (int kt = 0; kt < KT; kt++) {
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const __nv_bfloat16 *w = W + (j * 8 + g) * K + kt * 16 + 2 * t;
                b[kt][j][0] = __ldg(reinterpret_cast<const uint32_t *>(w));
                b[kt][j][1] = __ldg(reinterpret_cast<const uint32_t *>(w + 8));
            }
        }
    }
};

// acc[j] = A(k-tiles) x W^T for n-tiles j < NT
template <int NT, int KT>
__device__ __forceinline__ void layer(float (&acc)[NT][4], const uint32_t (&a)[KT][4], const BFrag<NT, KT> &w) {
#pragma unroll
    for (int j = 0; j < NT; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
    for (int kt = 0; kt < KT; kt++) {
#pragma unroll
        for (int j = 0; j < NT; j++) mma_bf16(acc[j], a[kt], w.b[kt][j][0], w.b[kt][j][1]);
    }
}

// relu(acc + bias) -> BF16 A fragments of the next layer (32 columns = 2
// k-tiles); bias: the lane's columns 2t, 2t+1 of each n-tile
template <int KT>
__device__ __forceinline__ void to_afrag(const float (&acc)[4][4], const float2 (&bias)[4], uint32_t (&a)[KT][4]) {
#pragma unroll
    for (int kt = 0; kt < 2; kt++) {
        float v[2][4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = 2 * kt + h;
            v[h][0] = fmaxf(acc[j][0] + bias[j].x, 0.0f);
            v[h][1] = fmaxf(acc[j][1] + bias[j].y, 0.0f);
            v[h][2] = fmaxf(acc[j][2] + bias[j].x, 0.0f);
            v[h][3] = fmaxf(acc[j][3] + bias[j].y, 0.0f);
        }
        a[kt][0] = pack_bf16(v[0][0], v[0][1]);
        a[kt][1] = pack_bf16(v[0][2], v[0][3]);
        a[kt][2] = pack_bf16(v[1][0], v[1][1]);
        a[kt][3] = pack_bf16(v[1][2], v[1][3]);
    }
}

// What a tile of 16 rows reads, loaded one tile ahead.
template <int STAGE>
struct TileIn {
    uint32_t dg = 0;              // this lane's of the quad's four degrees
    uint32_t a1[2] = {0u, 0u}, a2[2] = {0u, 0u};
    float sc[2] = {0.0f, 0.0f};
    __device__ __forceinline__ void load(uint32_t tile, uint32_t n, int g, int t, const uint32_t *row_ptr,
                                         const uint32_t *deg, const __nv_bfloat16 *A1, const __nv_bfloat16 *A2,
                                         const float *scale) {
        const uint32_t r0 = tile * 16 + g, r1 = r0 + 8, rl = t < 2 ? r0 : r1;
        dg = 0;
        if (rl < n) dg = (t & 1) ? __ldg(deg + rl) : __ldg(row_ptr + rl + 1) - __ldg(row_ptr + rl);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t r = h ? r1 : r0;
            a1[h] = a2[h] = 0u;
            sc[h] = 0.0f;
            if (r >= n) continue;
            if (STAGE >= 1) a1[h] = __ldg(reinterpret_cast<const uint32_t *>(A1 + (size_t)r * 16 + 2 * t));
            if (STAGE >= 2) a2[h] = __ldg(reinterpret_cast<const uint32_t *>(A2 + (size_t)r * 16 + 2 * t));
            if (STAGE <= 1) sc[h] = __ldg(scale + r);
        }
    }
};

// STAGE 0: write M0 = s * (H0 Wm1^T); 1: write M1; 2: write y
// Each warp keeps the inputs of the next tiles in flight; more than one in the
// later stages costs the registers of a resident block (four blocks with three
// tiles ahead: 143 / 149 us, five with two spill: 159 / 223 us).
constexpr int fused_ahead(int stage) { return stage == 0 ? 3 : 1; }
constexpr unsigned fused_per_sm(int stage) { return stage == 0 ? 7 : 5; }
template <int STAGE>
__global__ void __launch_bounds__(128, fused_per_sm(STAGE)) fused_kernel(uint32_t n, const uint32_t *row_ptr, const uint32_t *deg,
                                                       const __nv_bfloat16 *A1, const __nv_bfloat16 *A2, const Ws *Wg,
                                                       const float *P, const float *scale, float *out) {
    const float ln = logf((float)n) * 0.0625f;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    BFrag<4, 1> w1;
    w1.load(Wg->W1, kF, g, t);
    BFrag<4, 3> w2;
    BFrag<1, 2> wm;
    BFrag<1, 3> w3;
    float2 b1[4], b2[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        b1[j] = make_float2(P[oB1 + j * 8 + 2 * t], P[oB1 + j * 8 + 2 * t + 1]);
        b2[j] = make_float2(P[oB2 + j * 8 + 2 * t], P[oB2 + j * 8 + 2 * t + 1]);
    }
    if (STAGE >= 1) w2.load(Wg->W2, kZ, g, t);
    if (STAGE <= 1) wm.load(STAGE == 0 ? Wg->Wm1 : Wg->Wm2, kH, g, t);
    if (STAGE == 2) w3.load(Wg->W3, kZ, g, t);
    const float b3 = P[oB3];
    const uint32_t ntiles = (n + 15) / 16;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    constexpr int kFusedAhead = fused_ahead(STAGE);
    TileIn<STAGE> ring[kFusedAhead];
#pragma unroll
    for (int i = 0; i < kFusedAhead; i++)
        if ((uint64_t)warp + (uint64_t)i * nwarps < ntiles)
            ring[i].load(warp + i * nwarps, n, g, t, row_ptr, deg, A1, A2, scale);
    auto work = [&](uint32_t tile, TileIn<STAGE> &slot) {
        const TileIn<STAGE> in = slot;
        if ((uint64_t)tile + (uint64_t)kFusedAhead * nwarps < ntiles)
            slot.load(tile + kFusedAhead * nwarps, n, g, t, row_ptr, deg, A1, A2, scale);
        const uint32_t r0 = tile * 16 + g, r1 = r0 + 8;
        // the quad's four logarithms, one per lane: in- and out-degree of both rows
        const float lg = log1pf((float)in.dg);
        const int q0 = lane & ~3;
        const float li0 = __shfl_sync(0xffffffffu, lg, q0), lo0 = __shfl_sync(0xffffffffu, lg, q0 + 1);
        const float li1 = __shfl_sync(0xffffffffu, lg, q0 + 2), lo1 = __shfl_sync(0xffffffffu, lg, q0 + 3);
        const bool z0 = __shfl_sync(0xffffffffu, in.dg, q0 + 1) == 0u, z1 = __shfl_sync(0xffffffffu, in.dg, q0 + 3) == 0u;
        uint32_t ax[1][4];
        ax[0][0] = r0 < n ? feat_pair(t, li0, lo0, ln, z0) : 0u;
        ax[0][1] = r1 < n ? feat_pair(t, li1, lo1, ln, z1) : 0u;
        ax[0][2] = ax[0][3] = 0u;  // features 8 .. 15
        float acc[4][4];
        layer<4, 1>(acc, ax, w1);
        uint32_t ah[3][4];
        to_afrag(acc, b1, ah);
        if constexpr (STAGE >= 1) {
            // k-tile 2 of [H0 | A1] (its columns 8 .. 15 are zero)
            ah[2][0] = in.a1[0];
            ah[2][1] = in.a1[1];
            ah[2][2] = ah[2][3] = 0u;
            layer<4, 3>(acc, ah, w2);
            to_afrag(acc, b2, ah);
        }
        if constexpr (STAGE <= 1) {
            const uint32_t a2[2][4] = {{ah[0][0], ah[0][1], ah[0][2], ah[0][3]}, {ah[1][0], ah[1][1], ah[1][2], ah[1][3]}};
            float m[1][4];
            layer<1, 2>(m, a2, wm);
            if (r0 < n)
                *reinterpret_cast<float2 *>(out + (size_t)r0 * kC + 2 * t) =
                    make_float2(m[0][0] * in.sc[0], m[0][1] * in.sc[0]);
            if (r1 < n)
                *reinterpret_cast<float2 *>(out + (size_t)r1 * kC + 2 * t) =
                    make_float2(m[0][2] * in.sc[1], m[0][3] * in.sc[1]);
        } else {
            ah[2][0] = in.a2[0];
            ah[2][1] = in.a2[1];
            ah[2][2] = ah[2][3] = 0u;
            float yv[1][4];
            layer<1, 3>(yv, ah, w3);
            if (t == 0) {
                if (r0 < n) out[r0] = yv[0][0] + b3;
                if (r1 < n) out[r1] = yv[0][2] + b3;
            }
        }
    };
    for (uint32_t tile = warp; tile < ntiles;) {
#pragma unroll
        for (int i = 0; i < kFusedAhead; i++) {
            if (tile < ntiles) work(tile, ring[i]);
            tile += nwarps;
        }
    }
}

template <int STAGE>
static void fused(uint32_t n, const DeviceGraph &g, const __nv_bfloat16 *A1, const __nv_bfloat16 *A2, const Ws *W,
                  const float *P, const float *scale, float *out, cudaStream_t s) {
    const uint32_t tiles = (n + 15) / 16;
    const unsigned grid = (unsigned)std::max<uint32_t>(1, std::min<uint32_t>((tiles + 3) / 4, 148u * fused_per_sm(STAGE)));
    fused_kernel<STAGE><<<grid, 128, 0, s>>>(n, g.row_ptr, g.deg, A1, A2, W, P, scale, out);
    PRG_CUDA(cudaGetLastError());
}

// ---- host side -------------------------------------------------------------

int param_count() { return kParams; }

void Net::init(uint64_t seed, cudaStream_t s) {
    std::vector<float> p(kParams, 0.0f);
    uint64_t st = seed;
    auto unit = [&]() {
        st += 0x9E3779B97F4A7C15ULL;
        uint64_t z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int rows, int cols) {
        const double a = std::sqrt(6.0 / (double)cols);
        for (int i = 0; i < rows * cols; i++) p[off + i] = (float)((2.0 * unit() - 1.0) * a);
    };
    fill(oW1, kH, kF);
    fill(oWm1, kC, kH);
    fill(oW2, kH, kZ);
    fill(oWm2, kC, kH);
    fill(oW3, 1, kZ);  // rows 1..7 of W3 stay zero
    for (int i = 0; i < kH; i++) p[oB1 + i] = 0.05f;
    for (int i = 0; i < kH; i++) p[oB2 + i] = 0.05f;
    set_params(p.data(), s);
}

void Net::alloc(cudaStream_t s) {
    if (P) return;
    PRG_CUDA(cudaMallocAsync((void **)&P, kParams * 4, s));
    PRG_CUDA(cudaMallocAsync((void **)&G, kParams * 4, s));
    PRG_CUDA(cudaMallocAsync((void **)&m, kParams * 4, s));
    PRG_CUDA(cudaMallocAsync((void **)&v, kParams * 4, s));
    PRG_CUDA(cudaMallocAsync((void **)&w, sizeof(Ws), s));
    PRG_CUDA(cudaMemsetAsync(G, 0, kParams * 4, s));
    PRG_CUDA(cudaMemsetAsync(m, 0, kParams * 4, s));
    PRG_CUDA(cudaMemsetAsync(v, 0, kParams * 4, s));
    PRG_CUDA(cudaMemsetAsync(w, 0, sizeof(Ws), s));
}

void Net::set_params(const float *host, cudaStream_t s) {
    alloc(s);
    PRG_CUDA(cudaMemcpyAsync(P, host, kParams * 4, cudaMemcpyHostToDevice, s));
    to_bf16_kernel<<<(kH * kZ + 255) / 256, 256, 0, s>>>(P, (Ws *)w);
    PRG_CUDA(cudaGetLastError());
    PRG_CUDA(cudaStreamSynchronize(s));
}

void Net::get_params(float *host, cudaStream_t s) const {
    PRG_CUDA(cudaMemcpyAsync(host, P, kParams * 4, cudaMemcpyDeviceToHost, s));
    PRG_CUDA(cudaStreamSynchronize(s));
}

void Net::free(cudaStream_t s) {
    for (void *p : {(void *)P, (void *)G, (void *)m, (void *)v, (void *)w, (void *)buf})
        if (p) cudaFreeAsync(p, s);
    P = G = m = v = nullptr;
    w = nullptr;
    buf = nullptr;
    buf_n = 0;
}

// scratch layout per vertex (bytes): X0 32, H0 64, M0 32, A1 32, H1 64, M1 32,
// A2 32, y 4, s 4, dy 4, dS2 32, dM1 32, dH0 128, dS1 32, dM0 32, S1 32, S2 32
// -> 620 bytes per vertex, plus the heavy-row list and partials.
constexpr size_t kPerVertex = 620;

void Net::ensure(uint32_t n, cudaStream_t s) {
    if (buf && buf_n >= n) return;
    if (buf) cudaFreeAsync(buf, s);
    buf_n = n;
    const size_t bytes = (size_t)n * kPerVertex + (size_t)kBottomBlocks * kPartStride * 4 + 64 * 1024 +
                         (size_t)n * 4 + 8192;
    PRG_CUDA(cudaMallocAsync((void **)&buf, bytes, s));
}

struct Views {
    __nv_bfloat16 *X0, *H0, *A1, *H1, *A2;
    float *M0, *M1, *y, *s, *dy, *dS2, *dM1, *dH0, *dS1, *dM0, *S1, *S2, *part, *fpart;
    double *dpart;
    uint32_t *heavy, *nheavy;
};

static Views views(unsigned char *b, uint32_t n) {
    Views V;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        unsigned char *p = b + o;
        o += (bytes + 255) & ~(size_t)255;
        return p;
    };
    V.X0 = (__nv_bfloat16 *)take((size_t)n * 32);
    V.H0 = (__nv_bfloat16 *)take((size_t)n * 64);
    V.M0 = (float *)take((size_t)n * 32);
    V.A1 = (__nv_bfloat16 *)take((size_t)n * 32);
    V.H1 = (__nv_bfloat16 *)take((size_t)n * 64);
    V.M1 = (float *)take((size_t)n * 32);
    V.A2 = (__nv_bfloat16 *)take((size_t)n * 32);
    V.y = (float *)take((size_t)n * 4);
    V.s = (float *)take((size_t)n * 4);
    V.dy = (float *)take((size_t)n * 4);
    V.dS2 = (float *)take((size_t)n * 32);
    V.dM1 = (float *)take((size_t)n * 32);
    V.dH0 = (float *)take((size_t)n * 128);
    V.dS1 = (float *)take((size_t)n * 32);
    V.dM0 = (float *)take((size_t)n * 32);
    V.S1 = (float *)take((size_t)n * 32);
    V.S2 = (float *)take((size_t)n * 32);
    V.heavy = (uint32_t *)take((size_t)n * 4);
    V.part = (float *)take((size_t)kBottomBlocks * kPartStride * 4);
    V.fpart = (float *)take(4096 * 4);
    V.dpart = (double *)take(4096 * 8);
    V.nheavy = (uint32_t *)take(256);
    return V;
}

static unsigned grid_n(uint32_t n) { return (unsigned)std::max<uint32_t>(1, std::min<uint32_t>((n + 255) / 256, 148 * 16)); }

void Net::forward(const DeviceGraph &g, cudaStream_t s) {
    ensure(g.n, s);
    Views V = views(buf, g.n);
    const Ws *W = (const Ws *)w;
    const uint32_t n = g.n;
    const unsigned gn = grid_n(n);
    features_kernel<<<gn, 256, 0, s>>>(n, g.row_ptr, g.deg, V.X0);
    scale_kernel<<<gn, 256, 0, s>>>(g.deg, n, V.s);
    PRG_CUDA(cudaMemsetAsync(V.nheavy, 0, 4, s));
    heavy_rows_kernel<<<gn, 256, 0, s>>>(n, g.row_ptr, V.heavy, V.nheavy);
    PRG_CUDA(cudaGetLastError());
    rowwise<kF, 0, kH, EPI_RELU_BF16>(n, V.X0, nullptr, W->W1, P + oB1, nullptr, V.H0, nullptr, s);
    rowwise<kH, 0, kC, EPI_SCALE_F32>(n, V.H0, nullptr, W->Wm1, nullptr, V.s, nullptr, V.M0, s);
    for (int layer = 0; layer < 2; layer++) {
        const float *M = layer ? V.M1 : V.M0;
        __nv_bfloat16 *A = layer ? V.A2 : V.A1;
        float *S = layer ? V.S2 : V.S1;
        aggregate_kernel<<<kAggHeavyBlocks + kAggLightBlocks, 256, 0, s>>>(n, g.row_ptr, g.col, M, A, S, V.heavy,
                                                                           V.nheavy);
        PRG_CUDA(cudaGetLastError());
        if (layer == 0) {
            rowwise<kH, 16, kH, EPI_RELU_BF16>(n, V.H0, V.A1, W->W2, P + oB2, nullptr, V.H1, nullptr, s);
            rowwise<kH, 0, kC, EPI_SCALE_F32>(n, V.H1, nullptr, W->Wm2, nullptr, V.s, nullptr, V.M1, s);
        }
    }
    rowwise<kH, 16, 8, EPI_COL0_F32>(n, V.H1, V.A2, W->W3, P + oB3, nullptr, nullptr, V.y, s);
}

void Net::predict(const DeviceGraph &g, double *x_internal, cudaStream_t s) {
    // fused inference: M0, A1, M1, A2, y without materialising H0 / H1
    ensure(g.n, s);
    Views V = views(buf, g.n);
    const Ws *W = (const Ws *)w;
    const uint32_t n = g.n;
    scale_kernel<<<grid_n(n), 256, 0, s>>>(g.deg, n, V.s);
    PRG_CUDA(cudaMemsetAsync(V.nheavy, 0, 4, s));
    heavy_rows_kernel<<<grid_n(n), 256, 0, s>>>(n, g.row_ptr, V.heavy, V.nheavy);
    fused<0>(n, g, nullptr, nullptr, W, P, V.s, V.M0, s);
    for (int layer = 0; layer < 2; layer++) {
        const float *M = layer ? V.M1 : V.M0;
        __nv_bfloat16 *A = layer ? V.A2 : V.A1;
        aggregate_kernel<<<kAggHeavyBlocks + kAggLightBlocks, 256, 0, s>>>(n, g.row_ptr, g.col, M, A, nullptr,
                                                                           V.heavy, V.nheavy);
        PRG_CUDA(cudaGetLastError());
        if (layer == 0) fused<1>(n, g, V.A1, nullptr, W, P, V.s, V.M1, s);
    }
    fused<2>(n, g, V.A1, V.A2, W, P, V.s, V.y, s);
    const unsigned gb = 296;
    max_kernel<<<gb, 256, 0, s>>>(V.y, g.n, V.fpart);
    expsum_kernel<<<gb, 256, 0, s>>>(V.y, g.n, V.fpart, gb, x_internal, V.dpart);
    normalise_kernel<<<gb, 256, 0, s>>>(x_internal, g.n, V.dpart, gb);
    PRG_CUDA(cudaGetLastError());
}

double Net::loss_grad(const DeviceGraph &g, const double *target_internal, cudaStream_t s) {
    forward(g, s);  // leaves the heavy rows' list for the scatters
    Views V = views(buf, g.n);
    const uint32_t n = g.n;
    const unsigned gb = 296;
    loss_kernel<<<gb, 256, 0, s>>>(V.y, target_internal, n, P, V.S2, V.dy, V.dS2, V.dpart);
    const uint64_t steps = ((uint64_t)n + kBwdWarps * kVB - 1) / (kBwdWarps * kVB);
    const unsigned nbt = (unsigned)std::min<uint64_t>(kTopBlocks, steps);
    const unsigned nbb = (unsigned)std::min<uint64_t>(kBottomBlocks, steps);
    auto transposed = [&](const float *dS, float *dM) {
        PRG_CUDA(cudaMemsetAsync(dM, 0, (size_t)n * 32, s));
        scatter_kernel<<<148 * 8, 256, 0, s>>>(n, g.row_ptr, g.col, dS, dM);
        scatter_heavy_kernel<<<148 * 2, 256, 0, s>>>(g.row_ptr, g.col, dS, dM, V.heavy, V.nheavy);
        PRG_CUDA(cudaGetLastError());
    };
    transposed(V.dS2, V.dM1);
    bwd_top_kernel<<<nbt, kBwdThreads, 0, s>>>(n, V.dy, V.dM1, V.s, P, V.H1, V.A2, V.H0, V.A1, V.S1, V.dH0, V.dS1,
                                              V.part);
    transposed(V.dS1, V.dM0);
    bwd_bottom_kernel<<<nbb, kBwdThreads, 0, s>>>(n, V.dM0, V.s, P, V.H0, V.X0, V.dH0, V.part);
    reduce_part_kernel<<<(kParams + 31) / 32, 256, 0, s>>>(V.part, nbb, nbt, G);
    PRG_CUDA(cudaGetLastError());
    std::vector<double> lp(gb);
    PRG_CUDA(cudaMemcpyAsync(lp.data(), V.dpart, gb * 8, cudaMemcpyDeviceToHost, s));
    PRG_CUDA(cudaStreamSynchronize(s));
    double l = 0.0;
    for (double x : lp) l += x;
    return l;
}

void Net::adam(float lr, cudaStream_t s) {
    step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
    adam_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(P, G, m, v, kParams, lr, b1, b2, 1e-8f, c1, c2);
    to_bf16_kernel<<<(kH * kZ + 255) / 256, 256, 0, s>>>(P, (Ws *)w);
    PRG_CUDA(cudaGetLastError());
}

}  // namespace gnn
}  // namespace prg
