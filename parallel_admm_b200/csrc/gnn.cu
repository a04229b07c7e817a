// gnn.cu -- the learned per-vertex block preconditioner of the PCG global step:
// a 3-layer message-passing network (width 64) over the graph of the global
// matrix A, its loss and gradients, and an Adam update, all on the GPU with
// the project's own kernels.  An addition with no reference
// counterpart; the network and loss are specified in the header of the CPU
// restatement that the tests check these kernels against.
//
// Layout: every activation is a row-major FP32 matrix with a row per vertex; per edge only a
// layer's messages pass through one E x 64 buffer, and one bit per channel is kept.  An edge layer
// W [h_i, h_j, f_ij] + b of the message from j to i gathers its operand straight into shared
// memory (k_edge_fwd_tc, BF16 weights).  With FP32 weights it is W_r h_i + b (U), W_c h_j (V) and
// W_f f_ij: U and V are products per vertex (a fourteenth of the work on a tet lattice), and one
// pass over the edges adds the three, applies the ReLU and averages; the tensor cores keep the
// product per edge, whose sums the next layer's rounding to TF32 would otherwise meet in another
// order.  The gradient needs per vertex the sums of the message gradients over its row (Gr) and
// over the reversed edges (Gc); the products with W and with h follow per vertex.
// Dense layers are Z = X W^T + b with W row-major [out][in]; with bf16 set, the forward and
// input-gradient passes use the weights rounded to BF16 and the activations rounded to TF32
// (FP32 accumulation), the sums Gr and Gc stay FP32; the master weights and Adam moments are
// FP32.  Weight gradients are per-block partial sums reduced in a fixed order, node sums over
// edges run in CSR order, so a training step is deterministic.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "admm_b200.h"
#include "umma.cuh"

namespace {

constexpr int kH = 64;        // hidden width
constexpr int kFin = 6;       // node features
constexpr int kFe = 2;        // edge features
constexpr int kEdgeIn = 2 * kH + kFe;
constexpr int kNodeIn = 2 * kH;
constexpr int kOut = 7;       // head: lower-triangular factor of the block (6), warm-start coefficient (1)
constexpr int kDwBlocks = 592;  // most partials of a weight gradient (4 x 148 SMs)

constexpr int kTcRows = 128, kTcN = 64;

__device__ __forceinline__ float wval(const float* W, int i, int bf16) {
    const float w = W[i];
    return bf16 ? __bfloat162float(__float2bfloat16_rn(w)) : w;
}

// Z[R x N] = X[R x K] W^T + b;  act: 0 none, 1 Y = relu(Z) into Y, 2 Y = res + relu(Z).
// Block: 4 rows x 64 threads (N <= 64); W and the 4 input rows in shared memory.
__global__ void __launch_bounds__(256) k_dense_fwd(const float* __restrict__ X, int R, int K, const float* __restrict__ W,
                                                   const float* __restrict__ b, int N, float* __restrict__ Z,
                                                   float* __restrict__ Y, const float* __restrict__ res, int act,
                                                   int bf16) {
    extern __shared__ float sm[];
    float* Ws = sm;             // [N * K]
    float* Xs = sm + N * K;     // [4 * K]
    for (int i = threadIdx.x; i < N * K; i += blockDim.x) Ws[i] = wval(W, i, bf16);
    const int r0 = blockIdx.x * 4;
    for (int i = threadIdx.x; i < 4 * K; i += blockDim.x) {
        const int r = r0 + i / K;
        Xs[i] = r < R ? X[(size_t)r * K + i % K] : 0.f;
    }
    __syncthreads();
    const int rl = threadIdx.x / 64, c = threadIdx.x % 64, r = r0 + rl;
    if (c >= N || r >= R) return;
    float acc = b[c];
    const float* xr = Xs + rl * K;
    const float* wr = Ws + c * K;
    for (int k = 0; k < K; k++) acc = fmaf(xr[k], wr[k], acc);
    Z[(size_t)r * N + c] = acc;
    if (act == 1) Y[(size_t)r * N + c] = fmaxf(acc, 0.f);
    else if (act == 2) Y[(size_t)r * N + c] = res[(size_t)r * N + c] + fmaxf(acc, 0.f);
}

constexpr int kTcThreads = 256;  // a warp per 32 rows and half of the output columns

// Rows of one or two row-major [R][64] matrices (columns 0..63 from X0, 64.. from X1) rounded to
// TF32 into the canonical layout: eight rows by four 16-byte chunks per warp, so that a warp
// reads 64-byte pieces of rows and writes without bank conflicts.
template <int K>
__device__ __forceinline__ void stage_rows(unsigned char* As, const float* __restrict__ X0, const float* __restrict__ X1,
                                           int row0, int R) {
    constexpr int C = K / 4;
#pragma unroll
    for (int u = 0; u < kTcRows * C / kTcThreads; u++) {
        const int i = threadIdx.x + u * kTcThreads;
        const int r = (i & 7) | ((i >> 5) & 15) << 3, c = ((i >> 3) & 3) | (i >> 9) << 2;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + r < R) v = *(const float4*)((c < 16 ? X0 : X1) + (size_t)(row0 + r) * kH + 4 * (c & 15));
        *(float4*)(As + umma::core_offset(r, c, C)) = make_float4(umma::tf32_round(v.x), umma::tf32_round(v.y),
                                                                  umma::tf32_round(v.z), umma::tf32_round(v.w));
    }
}

// The accumulator (128 rows, N columns of TMEM at td) to f(row, column, four values): warp w
// reads rows 32 (w % 4) .. + 31 of half w / 4 of the columns.
template <int N, class F>
__device__ __forceinline__ void read_rows(uint32_t td, int row0, F f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = warp & 3;
    const int row = row0 + q * 32 + lane;
    const uint32_t tw = td + ((uint32_t)(q * 32) << 16);
#pragma unroll
    for (int u = 0; u < N / 32; u++) {
        const int c0 = (warp >> 2) * (N / 2) + 16 * u;
        uint32_t r[16];
        umma::tmem_load16(tw + c0, r);
        umma::tmem_wait16(r);
#pragma unroll
        for (int j = 0; j < 16; j += 4)
            f(row, c0 + j, make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                       __uint_as_float(r[j + 3])));
    }
}

// The same layer on the tensor cores (tcgen05, kind::tf32, FP32 accumulation in
// tensor memory) for 64 outputs: one CTA per 128 rows.  The
// rows of X (K = 64 or 128: one or two [R][64] matrices side by side; K = 8: [R][Kin] padded with
// zeros) and the weights (element (n, k) at W[n * ldw + k], rounded to BF16 first) are rounded to TF32 and staged in shared memory in the canonical K-major layout;
// thread 0 issues K / 8 MMAs of 128 x 64 x 8 into 64 TMEM columns and commits them to an
// mbarrier; the warps then read the accumulator and apply bias and activation.
// Bound by the latency of staging: with K and the
// loads' trip counts known to the compiler, 64 -> 19 us for 28 k rows and K = 64 (cold caches).
// The wait for the MMAs is bounded: a wait that gives up sets err[0] and the
// CTA releases its TMEM and leaves without writing.
template <int K>
__global__ void __launch_bounds__(kTcThreads) k_dense_fwd_tc(const float* __restrict__ X, const float* __restrict__ X1,
                                                             int R, int Kin, const float* __restrict__ W, int ldw,
                                                             const float* __restrict__ b, float* __restrict__ Z,
                                                             float* __restrict__ Y, const float* __restrict__ res,
                                                             int act, int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char tc_smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_base;
    constexpr int C = K / 4;  // 16-byte K chunks per row
    unsigned char* As = tc_smem;
    unsigned char* Bs = tc_smem + (size_t)kTcRows * K * 4;
    const int row0 = blockIdx.x * kTcRows;
    if (K % kH == 0) {
        stage_rows<(K % kH == 0 ? K : kH)>(As, X, X1, row0, R);
    } else {
#pragma unroll
        for (int u = 0; u < kTcRows * K / kTcThreads; u++) {
            const int i = threadIdx.x + u * kTcThreads, m = i / K, k = i % K;
            const float v = (row0 + m < R && k < Kin) ? X[(size_t)(row0 + m) * Kin + k] : 0.f;
            *(float*)(As + umma::core_offset(m, k >> 2, C) + (k & 3) * 4) = umma::tf32_round(v);
        }
    }
#pragma unroll 16
    for (int u = 0; u < kTcN * K / kTcThreads; u++) {
        const int i = threadIdx.x + u * kTcThreads, n = i / K, k = i % K;
        const float v = k < Kin ? wval(W, n * ldw + k, 1) : 0.f;
        *(float*)(Bs + umma::core_offset(n, k >> 2, C) + (k & 3) * 4) = v;  // BF16 is exact in TF32
    }
    umma::fence_operands();
    if (threadIdx.x == 0) umma::mbar_init(&mbar, 1);
    if (threadIdx.x < 32) umma::tmem_alloc(&tmem_base, kTcN);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t td = tmem_base;
    if (threadIdx.x == 0) {
        const uint32_t idesc = umma::idesc_tf32(kTcRows, kTcN);
        const uint32_t a0 = umma::smem_u32(As), b0 = umma::smem_u32(Bs);
        for (int k = 0; k < K / 8; k++)  // 8 TF32 values of K = two 16-byte chunks per MMA
            umma::mma_tf32(td, umma::smem_desc(a0 + 256u * k, C), umma::smem_desc(b0 + 256u * k, C), idesc, k > 0);
        umma::commit(&mbar);
    }
    bool ok = umma::mbar_wait(&mbar, 0, 1 << 22);
    if (!ok) umma::mbar_wait(&mbar, 0, 1 << 22);  // the MMAs in flight, once more with a bound
    ok = __syncthreads_and(ok) != 0;              // uniform: the TMEM loads below are warp-wide
    umma::fence_after();
    if (ok) {
        read_rows<kTcN>(td, row0, [&](int row, int c, float4 v) {
            if (row >= R) return;
            v = make_float4(v.x + b[c], v.y + b[c + 1], v.z + b[c + 2], v.w + b[c + 3]);
            *(float4*)(Z + (size_t)row * kTcN + c) = v;
            if (!act) return;
            float4 q = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
            if (act == 2) {
                const float4 e = *(const float4*)(res + (size_t)row * kTcN + c);
                q = make_float4(e.x + q.x, e.y + q.y, e.z + q.z, e.w + q.w);
            }
            *(float4*)(Y + (size_t)row * kTcN + c) = q;
        });
    } else if (threadIdx.x == 0) {
        atomicExch(err, 1);
    }
    umma::fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        umma::fence_after();
        umma::tmem_dealloc(td, kTcN);
    }
}

// An edge layer's messages Z[E x 64] = [h_row, h_col, f] W^T + b on the tensor cores, the operand
// gathered as it is staged: 128 edges per tile, K = 130 padded to 136, 17 MMAs of 128 x 64 x 8.  A
// CTA keeps the weights in shared memory and takes tiles in steps of the grid (two CTAs per SM:
// one stages while the other's tile is multiplied and written).  Bound by the gathers (512 B per
// edge, from L2) and the messages' store.  The MMA wait is bounded as in k_dense_fwd_tc.
constexpr int kEdgeK = (kEdgeIn + 7) / 8 * 8;

__global__ void __launch_bounds__(kTcThreads) k_edge_fwd_tc(const float* __restrict__ h, const float* __restrict__ ef,
                                                            const int* __restrict__ rows, const int* __restrict__ col,
                                                            int E, const float* __restrict__ W,
                                                            const float* __restrict__ b, float* __restrict__ Z,
                                                            int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char tc_smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_base;
    constexpr int C = kEdgeK / 4;
    unsigned char* As = tc_smem;
    unsigned char* Bs = tc_smem + (size_t)kTcRows * kEdgeK * 4;
#pragma unroll 17
    for (int u = 0; u < kTcN * kEdgeK / kTcThreads; u++) {
        const int i = threadIdx.x + u * kTcThreads, n = i / kEdgeK, k = i % kEdgeK;
        const float v = k < kEdgeIn ? wval(W, n * kEdgeIn + k, 1) : 0.f;
        *(float*)(Bs + umma::core_offset(n, k >> 2, C) + (k & 3) * 4) = v;  // BF16 is exact in TF32
    }
    if (threadIdx.x == 0) umma::mbar_init(&mbar, 1);
    if (threadIdx.x < 32) umma::tmem_alloc(&tmem_base, kTcN);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t td = tmem_base;
    bool ok = true;
    uint32_t phase = 0;
    for (int e0 = blockIdx.x * kTcRows; e0 < E && ok; e0 += gridDim.x * kTcRows) {
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int* at = half ? col : rows;
#pragma unroll
            for (int u = 0; u < kTcRows * 16 / kTcThreads; u++) {
                const int i = threadIdx.x + u * kTcThreads;
                const int r = (i & 7) | ((i >> 5) & 15) << 3, c = ((i >> 3) & 3) | (i >> 9) << 2;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (e0 + r < E) v = *(const float4*)(h + (size_t)at[e0 + r] * kH + 4 * c);
                *(float4*)(As + umma::core_offset(r, 16 * half + c, C)) =
                    make_float4(umma::tf32_round(v.x), umma::tf32_round(v.y), umma::tf32_round(v.z), umma::tf32_round(v.w));
            }
        }
        {
            const int r = threadIdx.x & 127, c = threadIdx.x >> 7;  // chunk 32: the edge's two features, chunk 33: padding
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c == 0 && e0 + r < E) {
                const float2 f = ((const float2*)ef)[e0 + r];
                v = make_float4(umma::tf32_round(f.x), umma::tf32_round(f.y), 0.f, 0.f);
            }
            *(float4*)(As + umma::core_offset(r, 32 + c, C)) = v;
        }
        umma::fence_operands();
        umma::fence_before();
        __syncthreads();
        umma::fence_after();
        if (threadIdx.x == 0) {
            const uint32_t idesc = umma::idesc_tf32(kTcRows, kTcN);
            const uint32_t a0 = umma::smem_u32(As), b0 = umma::smem_u32(Bs);
            for (int k = 0; k < kEdgeK / 8; k++)
                umma::mma_tf32(td, umma::smem_desc(a0 + 256u * k, C), umma::smem_desc(b0 + 256u * k, C), idesc, k > 0);
            umma::commit(&mbar);
        }
        ok = umma::mbar_wait(&mbar, phase, 1 << 22);
        if (!ok) umma::mbar_wait(&mbar, phase, 1 << 22);  // the MMAs in flight, once more with a bound
        ok = __syncthreads_and(ok) != 0;                  // uniform
        phase ^= 1u;
        umma::fence_after();
        if (ok)
            read_rows<kTcN>(td, e0, [&](int row, int c, float4 v) {
                if (row < E)
                    *(float4*)(Z + (size_t)row * kTcN + c) = make_float4(v.x + b[c], v.y + b[c + 1], v.z + b[c + 2], v.w + b[c + 3]);
            });
        else if (threadIdx.x == 0)
            atomicExch(err, 1);
        umma::fence_before();
        __syncthreads();  // the accumulator has been read, the operands may be overwritten
        umma::fence_after();
    }
    umma::fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        umma::fence_after();
        umma::tmem_dealloc(td, kTcN);
    }
}

// agg_i = mean over the edges of row i of relu(Z_e), and the bits as in k_edge_agg.
template <bool BITS>
__global__ void __launch_bounds__(256) k_node_agg(const float* __restrict__ Z, const int* __restrict__ start, int n,
                                                  float* __restrict__ agg, uint2* __restrict__ bits) {
    const int lane = threadIdx.x & 15, i = (blockIdx.x * blockDim.x + threadIdx.x) / 16;
    if (i >= n) return;
    const unsigned gm = 0xffffu << (threadIdx.x & 16);
    const int shift = threadIdx.x & 16, b = start[i], e1 = start[i + 1];
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int e = b; e < e1; e++) {
        const float4 v = ((const float4*)Z)[(size_t)e * 16 + lane];
        const float z[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int t = 0; t < 4; t++) a[t] += fmaxf(z[t], 0.f);
        if (BITS) {
            unsigned m[4];
#pragma unroll
            for (int t = 0; t < 4; t++) m[t] = (__ballot_sync(gm, z[t] > 0.f) >> shift) & 0xffffu;
            if (lane == 0) bits[e] = make_uint2(m[0] | m[1] << 16, m[2] | m[3] << 16);
        }
    }
    const float d = (float)max(e1 - b, 1);
    ((float4*)agg)[(size_t)i * 16 + lane] = make_float4(a[0] / d, a[1] / d, a[2] / d, a[3] / d);
}

// The input gradients on the tensor cores (bf16 set), the same tcgen05 path as
// k_dense_fwd_tc: operands rounded to TF32 (the weights to BF16 first) and staged in
// shared memory in the canonical K-major layout, MMAs of 128 x KP x 8 issued by one
// thread into FP32 accumulators in tensor memory, one mbarrier
// (bounded waits: a wait that gives up sets err[0], waits once more with a bound for the
// MMAs in flight, releases the TMEM and leaves without writing).
//
// dX[R x K] = dZ[R x N] W[N x K]: one CTA per 128 rows; A = the rows of dZ (reduction over N,
// NP = 64 or, for the head, 8: N padded with zeros), B = W^T (row k holds W[., k]), the MMA's N = K
// (64 or 128).  Columns 0..63 of dX go to a row-major [R][64] matrix, 64..127 to the next one.
template <int NP, int K>
__global__ void __launch_bounds__(kTcThreads) k_dense_dx_tc(const float* __restrict__ dZ, int R, int N,
                                                            const float* __restrict__ W, float* __restrict__ dX,
                                                            int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char tc_smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_base;
    constexpr int C = NP / 4;
    unsigned char* As = tc_smem;
    unsigned char* Bs = tc_smem + (size_t)kTcRows * NP * 4;
    const int row0 = blockIdx.x * kTcRows;
    if (NP == kH) {
        stage_rows<kH>(As, dZ, dZ, row0, R);
    } else {
#pragma unroll
        for (int u = 0; u < kTcRows * NP / kTcThreads; u++) {
            const int i = threadIdx.x + u * kTcThreads, m = i / NP, k = i % NP;
            const float v = (row0 + m < R && k < N) ? dZ[(size_t)(row0 + m) * N + k] : 0.f;
            *(float*)(As + umma::core_offset(m, k >> 2, C) + (k & 3) * 4) = umma::tf32_round(v);
        }
    }
#pragma unroll 16
    for (int u = 0; u < (K * NP + kTcThreads - 1) / kTcThreads; u++) {
        const int i = threadIdx.x + u * kTcThreads, j = i % K, n = i / K;
        if (n < NP) {
            const float v = n < N ? wval(W, n * K + j, 1) : 0.f;
            *(float*)(Bs + umma::core_offset(j, n >> 2, C) + (n & 3) * 4) = v;
        }
    }
    umma::fence_operands();
    if (threadIdx.x == 0) umma::mbar_init(&mbar, 1);
    if (threadIdx.x < 32) umma::tmem_alloc(&tmem_base, K);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t td = tmem_base;
    if (threadIdx.x == 0) {
        const uint32_t idesc = umma::idesc_tf32(kTcRows, K);
        const uint32_t a0 = umma::smem_u32(As), b0 = umma::smem_u32(Bs);
        for (int k = 0; k < NP / 8; k++)
            umma::mma_tf32(td, umma::smem_desc(a0 + 256u * k, C), umma::smem_desc(b0 + 256u * k, C), idesc, k > 0);
        umma::commit(&mbar);
    }
    bool ok = umma::mbar_wait(&mbar, 0, 1 << 22);
    if (!ok) umma::mbar_wait(&mbar, 0, 1 << 22);
    ok = __syncthreads_and(ok) != 0;
    umma::fence_after();
    if (ok) {
        read_rows<K>(td, row0, [&](int row, int c, float4 v) {
            if (row < R) *(float4*)(dX + ((size_t)(c / kH) * R + row) * kH + c % kH) = v;
        });
    } else if (threadIdx.x == 0) {
        atomicExch(err, 1);
    }
    umma::fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        umma::fence_after();
        umma::tmem_dealloc(td, K);
    }
}

// Products per vertex on the FP32 pipes (64 output columns): for FP32 weights, and for the sums
// Gr and Gc, which TF32 would round.
// C[R x 64] = A B (+ bias, act as k_dense_fwd; + add1 + add2), A = [A0 | A1] of row-major [R][64]
// matrices (K = 64: A0 only), B(k, m) = W[m sm + (k % 64) sk + (k / 64) sx + blockIdx.y sy];
// blockIdx.y > 0: the next [R][64] output, without bias.  256 threads per 64 rows, 4 x 4
// outputs each.
struct MatIndex {
    int sm, sk, sx, sy;
};

template <int K>
__global__ void __launch_bounds__(256) k_gemm(const float* __restrict__ A0, const float* __restrict__ A1, int R,
                                              const float* __restrict__ W, MatIndex ix, const float* __restrict__ b,
                                              float* __restrict__ Z, float* __restrict__ Y,
                                              const float* __restrict__ res, int act, const float* __restrict__ add1,
                                              const float* __restrict__ add2, int bf16) {
    extern __shared__ __align__(16) float gsm[];
    constexpr int LA = K + 4, LB = 68;
    float* As = gsm;            // [64][LA]
    float* Bs = gsm + 64 * LA;  // [K][LB]
    const int row0 = blockIdx.x * 64;
    for (int i = threadIdx.x; i < 64 * (K / 4); i += 256) {
        const int r = i / (K / 4), c = i % (K / 4);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + r < R) v = *(const float4*)((c < 16 ? A0 : A1) + (size_t)(row0 + r) * kH + 4 * (c & 15));
        *(float4*)(As + r * LA + 4 * c) = v;
    }
    for (int i = threadIdx.x; i < K * 64; i += 256) {
        const int k = ix.sk == 1 ? i % K : i / 64, m = ix.sk == 1 ? i / K : i % 64;  // consecutive threads: consecutive weights
        Bs[k * LB + m] = wval(W, m * ix.sm + (k & 63) * ix.sk + (k >> 6) * ix.sx + (int)blockIdx.y * ix.sy, bf16);
    }
    __syncthreads();
    const int r0 = threadIdx.x / 16 * 4, c0 = threadIdx.x % 16 * 4;
    float acc[4][4] = {};
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        float4 a[4], w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = *(const float4*)(As + (r0 + i) * LA + k);
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = *(const float4*)(Bs + (k + j) * LB + c0);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                acc[i][0] = fmaf(av[j], w[j].x, acc[i][0]);
                acc[i][1] = fmaf(av[j], w[j].y, acc[i][1]);
                acc[i][2] = fmaf(av[j], w[j].z, acc[i][2]);
                acc[i][3] = fmaf(av[j], w[j].w, acc[i][3]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = row0 + r0 + i;
        if (row >= R) break;
        const size_t at = (size_t)row * kH + c0;
        float4 z = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if (b && blockIdx.y == 0) z = make_float4(z.x + b[c0], z.y + b[c0 + 1], z.z + b[c0 + 2], z.w + b[c0 + 3]);
        if (add1) {
            const float4 p = *(const float4*)(add1 + at), q = *(const float4*)(add2 + at);
            z = make_float4((p.x + q.x) + z.x, (p.y + q.y) + z.y, (p.z + q.z) + z.z, (p.w + q.w) + z.w);
        }
        *(float4*)(Z + (size_t)blockIdx.y * R * kH + at) = z;
        if (act) {
            float4 q = make_float4(fmaxf(z.x, 0.f), fmaxf(z.y, 0.f), fmaxf(z.z, 0.f), fmaxf(z.w, 0.f));
            if (act == 2) {
                const float4 e = *(const float4*)(res + at);
                q = make_float4(e.x + q.x, e.y + q.y, e.z + q.z, e.w + q.w);
            }
            *(float4*)(Y + at) = q;
        }
    }
}

// dX[R x K] = dZ[R x N] W  (W [N x K]).  Block: 4 rows x 256/4 threads over k.
__global__ void __launch_bounds__(256) k_dense_dx(const float* __restrict__ dZ, int R, int N, const float* __restrict__ W,
                                                  int K, float* __restrict__ dX, int bf16) {
    extern __shared__ float sm[];
    float* Ws = sm;            // [N * K]
    float* Ds = sm + N * K;    // [4 * N]
    for (int i = threadIdx.x; i < N * K; i += blockDim.x) Ws[i] = wval(W, i, bf16);
    const int r0 = blockIdx.x * 4;
    for (int i = threadIdx.x; i < 4 * N; i += blockDim.x) {
        const int r = r0 + i / N;
        Ds[i] = r < R ? dZ[(size_t)r * N + i % N] : 0.f;
    }
    __syncthreads();
    const int rl = threadIdx.x / 64, r = r0 + rl;
    if (r >= R) return;
    for (int k = threadIdx.x % 64; k < K; k += 64) {
        float acc = 0.f;
        for (int c = 0; c < N; c++) acc = fmaf(Ds[rl * N + c], Ws[c * K + k], acc);
        dX[(size_t)r * K + k] = acc;
    }
}

// Per-block partials of dW[N x K] = dZ^T X (N <= 64, K <= KT) and db[N] = sum_r dZ over the
// block's rows: part[block][n * K + k], part[block][N * K + n].  X = [X0 | X1] of row-major
// [R][64] matrices for K = 64 or 128, else X0 [R][K].  round_z / round_x: to TF32, the operands
// of a tensor-core product.  A block takes `per` consecutive rows, 64 at a time through shared
// memory, a thread 4 x KT / 16 outputs.  blockIdx.y > 0: the next [R][64] matrix of dZ, into the
// partials after the first one's.
__device__ __forceinline__ float4 round4(float4 v, int on) {
    return on ? make_float4(umma::tf32_round(v.x), umma::tf32_round(v.y), umma::tf32_round(v.z), umma::tf32_round(v.w)) : v;
}

template <int KT>
__global__ void __launch_bounds__(256) k_dense_dw(const float* __restrict__ dZ, const float* __restrict__ X0,
                                                  const float* __restrict__ X1, int R, int per, int N, int K,
                                                  int round_z, int round_x, float* __restrict__ part) {
    extern __shared__ __align__(16) float gsm[];
    constexpr int LZ = 68, LX = KT + 4;
    float* Zs = gsm;            // [64][LZ]
    float* Xs = gsm + 64 * LZ;  // [64][LX]
    const int c0 = threadIdx.x / 16 * 4, k0 = threadIdx.x % 16 * 4;
    float acc[KT / 64][4][4] = {};
    float bias = 0.f;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    dZ += (size_t)blockIdx.y * R * kH;
    const int rbeg = blockIdx.x * per, rend = min(R, rbeg + per);
    for (int rc = rbeg; rc < rend; rc += 64) {
        __syncthreads();
        if (N == 64) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = threadIdx.x + 256 * u, r = i / 16, c = i % 16 * 4;
                const float4 v = rc + r < rend ? *(const float4*)(dZ + (size_t)(rc + r) * kH + c) : zero;
                *(float4*)(Zs + r * LZ + c) = round4(v, round_z);
            }
        } else {
            for (int i = threadIdx.x; i < 64 * 64; i += 256) {
                const int r = i / 64, c = i % 64;
                const float v = (rc + r < rend && c < N) ? dZ[(size_t)(rc + r) * N + c] : 0.f;
                Zs[r * LZ + c] = round_z ? umma::tf32_round(v) : v;
            }
        }
        if (K % 64 == 0) {
#pragma unroll
            for (int u = 0; u < KT / 16; u++) {
                const int i = threadIdx.x + 256 * u, r = i / (KT / 4), k = i % (KT / 4) * 4;
                const float4 v = rc + r < rend ? *(const float4*)((k < 64 ? X0 : X1) + (size_t)(rc + r) * kH + k % 64) : zero;
                *(float4*)(Xs + r * LX + k) = round4(v, round_x);
            }
        } else {
            for (int i = threadIdx.x; i < 64 * KT; i += 256) {
                const int r = i / KT, k = i % KT;
                const float v = (rc + r < rend && k < K) ? X0[(size_t)(rc + r) * K + k] : 0.f;
                Xs[r * LX + k] = round_x ? umma::tf32_round(v) : v;
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int r = 0; r < 64; r++) {
            const float4 z = *(const float4*)(Zs + r * LZ + c0);
            const float zv[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
            for (int h = 0; h < KT / 64; h++) {
                const float4 x = *(const float4*)(Xs + r * LX + 64 * h + k0);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    acc[h][i][0] = fmaf(zv[i], x.x, acc[h][i][0]);
                    acc[h][i][1] = fmaf(zv[i], x.y, acc[h][i][1]);
                    acc[h][i][2] = fmaf(zv[i], x.z, acc[h][i][2]);
                    acc[h][i][3] = fmaf(zv[i], x.w, acc[h][i][3]);
                }
            }
        }
        if (threadIdx.x < 64) {
#pragma unroll 16
            for (int r = 0; r < 64; r++) bias += Zs[r * LZ + threadIdx.x];
        }
    }
    float* out = part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (N * K + N);
#pragma unroll
    for (int h = 0; h < KT / 64; h++)
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (c0 + i < N && 64 * h + k0 + j < K) out[(c0 + i) * K + 64 * h + k0 + j] = acc[h][i][j];
    if (threadIdx.x < (unsigned)N) out[N * K + threadIdx.x] = bias;
}

// Partials summed in a fixed order, output o = n * K + k to grad[wo + n * ldw + k] and the last N
// to grad[bo + n] (bo < 0: dropped).  A block sums 32 outputs, 32 threads each; blockIdx.y > 0: the
// next nparts partials, to weights 64 columns further.
__global__ void __launch_bounds__(1024) k_reduce_parts(const float* __restrict__ part, int nparts, int N, int K,
                                                       float* __restrict__ grad, int wo, int ldw, int bo) {
    __shared__ float sh[32][33];
    const int nout = N * K + N, tx = threadIdx.x & 31, ty = threadIdx.x >> 5, o = blockIdx.x * 32 + tx;
    part += (size_t)blockIdx.y * nparts * nout;
    float a = 0.f;
    if (o < nout)
#pragma unroll 8
        for (int b = ty; b < nparts; b += 32) a += part[(size_t)b * nout + o];
    sh[tx][ty] = a;
    __syncthreads();
    a = sh[ty][tx];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) a += __shfl_xor_sync(0xffffffffu, a, d);
    const int q = blockIdx.x * 32 + ty;
    if (tx != 0 || q >= nout) return;
    if (q < N * K) grad[wo + blockIdx.y * kH + q / K * ldw + q % K] += a;
    else if (bo >= 0) grad[bo + q - N * K] += a;
}

// The edge layer from its per-vertex halves: agg_i = mean over the edges e = (i, j) of row i of
// relu(U_i + V_j + W_f f_e), and per edge one bit per channel, set where the message's argument is
// positive (bits: the four ballots of the row's 16 lanes, lane l holding channels 4 l .. 4 l + 3).
// 16 lanes per vertex; U and V are the two halves of UV.  Bound by the gathers of V (256 B per
// edge, from L2).  BITS = false: without the bits, which only the gradient reads.
template <bool BITS>
__global__ void __launch_bounds__(256) k_edge_agg(const float* __restrict__ UV, const float* __restrict__ We,
                                                  const float* __restrict__ ef, const int* __restrict__ start,
                                                  const int* __restrict__ col, int n, float* __restrict__ agg,
                                                  uint2* __restrict__ bits) {
    const int lane = threadIdx.x & 15, i = (blockIdx.x * blockDim.x + threadIdx.x) / 16;
    if (i >= n) return;
    const unsigned gm = 0xffffu << (threadIdx.x & 16);
    const int shift = threadIdx.x & 16;
    const float4* V = (const float4*)(UV + (size_t)n * kH) + lane;
    const float4 u = ((const float4*)UV)[(size_t)i * 16 + lane];
    float w0[4], w1[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        w0[t] = wval(We, (4 * lane + t) * kEdgeIn + 2 * kH, 0);
        w1[t] = wval(We, (4 * lane + t) * kEdgeIn + 2 * kH + 1, 0);
    }
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    const int b = start[i], e1 = start[i + 1];
#pragma unroll 4
    for (int e = b; e < e1; e++) {
        const float4 v = V[(size_t)col[e] * 16];
        const float2 f = ((const float2*)ef)[e];
        const float z[4] = {fmaf(f.y, w1[0], fmaf(f.x, w0[0], u.x + v.x)), fmaf(f.y, w1[1], fmaf(f.x, w0[1], u.y + v.y)),
                            fmaf(f.y, w1[2], fmaf(f.x, w0[2], u.z + v.z)), fmaf(f.y, w1[3], fmaf(f.x, w0[3], u.w + v.w))};
#pragma unroll
        for (int t = 0; t < 4; t++) a[t] += fmaxf(z[t], 0.f);
        if (BITS) {
            unsigned m[4];
#pragma unroll
            for (int t = 0; t < 4; t++) m[t] = (__ballot_sync(gm, z[t] > 0.f) >> shift) & 0xffffu;
            if (lane == 0) bits[e] = make_uint2(m[0] | m[1] << 16, m[2] | m[3] << 16);
        }
    }
    const float d = (float)max(e1 - b, 1);
    ((float4*)agg)[(size_t)i * 16 + lane] = make_float4(a[0] / d, a[1] / d, a[2] / d, a[3] / d);
}

// B_i = L_i L_i^T / a_ii from the head output o_i (L: exp of o0..2 clamped to
// [-8, 8] on the diagonal, o3, o4, o5 at (1,0), (2,0), (2,1)).
__device__ __forceinline__ float clamp8(float v) { return fminf(fmaxf(v, -8.f), 8.f); }

__device__ __forceinline__ void lower_of(const float* o, float L[9]) {
    L[0] = expf(clamp8(o[0])); L[1] = 0.f; L[2] = 0.f;
    L[3] = o[3]; L[4] = expf(clamp8(o[1])); L[5] = 0.f;
    L[6] = o[4]; L[7] = o[5]; L[8] = expf(clamp8(o[2]));
}

// The head o = W h + b (7 outputs) and what is made of it: B, and the learned global step's outputs
// m_i = trace(B_i) / 3 (the isotropic part of the block: the system is A (x) I3),
// theta_i = clamp(o_i6, -1, 1).  64 rows per block, an output (row, c) per thread at a time.
__global__ void __launch_bounds__(256) k_head(const float* __restrict__ h, const float* __restrict__ W,
                                              const float* __restrict__ b, const float* __restrict__ adiag, int n,
                                              float* __restrict__ o, float* __restrict__ B, float* __restrict__ m,
                                              float* __restrict__ th, int bf16) {
    __shared__ __align__(16) float Hs[64][68];
    __shared__ float Ws[kOut][kH];
    __shared__ float Os[64][kOut];
    const int row0 = blockIdx.x * 64;
    for (int i = threadIdx.x; i < kOut * kH; i += 256) Ws[i / kH][i % kH] = wval(W, i, bf16);
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int i = threadIdx.x + 256 * u, r = i / 16, c = i % 16 * 4;
        *(float4*)&Hs[r][c] = row0 + r < n ? *(const float4*)(h + (size_t)(row0 + r) * kH + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 64 * kOut; i += 256) {
        const int r = i % 64, c = i / 64;
        float acc = b[c];
#pragma unroll 16
        for (int k = 0; k < kH; k++) acc = fmaf(Hs[r][k], Ws[c][k], acc);
        Os[r][c] = acc;
        if (row0 + r < n) o[(size_t)(row0 + r) * kOut + c] = acc;
    }
    __syncthreads();
    const int i = row0 + threadIdx.x;
    if (threadIdx.x >= 64 || i >= n) return;
    float L[9], d = 0.f;
    lower_of(Os[threadIdx.x], L);
    const float ia = 1.f / adiag[i];
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) {
            float a = 0.f;
            for (int k = 0; k < 3; k++) a = fmaf(L[3 * r + k], L[3 * c + k], a);
            a *= ia;
            B[(size_t)i * 9 + 3 * r + c] = a;
            if (r == c) d += a;
        }
    m[i] = d * (1.f / 3.f);
    th[i] = fminf(fmaxf(Os[threadIdx.x][6], -1.f), 1.f);
}

// out = A v  (A = diag + CSR off-diagonal), v and out [n x 3]
__global__ void k_spmv3(const int* __restrict__ start, const int* __restrict__ col, const float* __restrict__ val,
                        const float* __restrict__ adiag, const float* __restrict__ v, int n, float* __restrict__ out,
                        const float* __restrict__ sub) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float a0 = adiag[i] * v[3 * i], a1 = adiag[i] * v[3 * i + 1], a2 = adiag[i] * v[3 * i + 2];
    for (int e = start[i]; e < start[i + 1]; e++) {
        const int j = col[e];
        a0 = fmaf(val[e], v[3 * j], a0);
        a1 = fmaf(val[e], v[3 * j + 1], a1);
        a2 = fmaf(val[e], v[3 * j + 2], a2);
    }
    if (sub) {
        a0 -= sub[3 * i];
        a1 -= sub[3 * i + 1];
        a2 -= sub[3 * i + 2];
    }
    out[3 * i] = a0;
    out[3 * i + 1] = a1;
    out[3 * i + 2] = a2;
}

__global__ void k_apply_blocks(const float* __restrict__ B, const float* __restrict__ r, int n, float* __restrict__ z) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* b = B + (size_t)i * 9;
    const float x = r[3 * i], y = r[3 * i + 1], w = r[3 * i + 2];
    z[3 * i] = b[0] * x + b[1] * y + b[2] * w;
    z[3 * i + 1] = b[3] * x + b[4] * y + b[5] * w;
    z[3 * i + 2] = b[6] * x + b[7] * y + b[8] * w;
}

// per-block partial sums of a . b (FP64) over 3n entries; one reduction slot per block
__global__ void k_dot_parts(const float* __restrict__ a, const float* __restrict__ b, int m, double* __restrict__ part) {
    __shared__ double sh[256];
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) s += (double)a[i] * (double)b[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// gB_i += (scale_k * gz_i) r_i^T with scale_k = 2 / (|r_k|^2 K) read from dots[k]
__global__ void k_accum_gB(const float* __restrict__ gz, const float* __restrict__ r, int n, const double* __restrict__ scale,
                           float* __restrict__ gB) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float s = (float)scale[0];
    for (int a = 0; a < 3; a++)
        for (int b = 0; b < 3; b++) gB[(size_t)i * 9 + 3 * a + b] += s * gz[3 * i + a] * r[3 * i + b];
}

// Head backward: go from gB (dL/dB) -- G = gB / a, gL = (G + G^T) L, go as in the header.
__global__ void k_head_grad(const float* __restrict__ gB, const float* __restrict__ o, const float* __restrict__ adiag,
                            int n, float* __restrict__ go, const float* __restrict__ gth) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float L[9], G[9], gL[9];
    lower_of(o + (size_t)i * kOut, L);
    const float ia = 1.f / adiag[i];
    for (int k = 0; k < 9; k++) G[k] = gB[(size_t)i * 9 + k] * ia;
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) {
            float a = 0.f;
            for (int k = 0; k < 3; k++) a = fmaf(G[3 * r + k] + G[3 * k + r], L[3 * k + c], a);
            gL[3 * r + c] = a;
        }
    float* g = go + (size_t)i * kOut;
    const float* oi = o + (size_t)i * kOut;
    g[0] = fabsf(oi[0]) < 8.f ? gL[0] * L[0] : 0.f;
    g[1] = fabsf(oi[1]) < 8.f ? gL[4] * L[4] : 0.f;
    g[2] = fabsf(oi[2]) < 8.f ? gL[8] * L[8] : 0.f;
    g[3] = gL[3];
    g[4] = gL[6];
    g[5] = gL[7];
    g[6] = (gth && fabsf(oi[6]) < 1.f) ? gth[i] : 0.f;
}

// gB_i = (gm_i / 3) I
__global__ void k_gm_to_gB(const float* __restrict__ gm, int n, float* __restrict__ gB) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = gm[i] * (1.f / 3.f);
    for (int k = 0; k < 9; k++) gB[(size_t)i * 9 + k] = (k % 4 == 0) ? v : 0.f;
}

// d = g * (z > 0)
__global__ void k_relu_mask(const float* __restrict__ g, const float* __restrict__ z, size_t m, float* __restrict__ d) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < m) d[t] = z[t] > 0.f ? g[t] : 0.f;
}

// q_i = g_i / deg_i: the gradient that vertex i's mean hands to each of its messages (rounded to
// TF32 with bf16 set, as the operand of a tensor-core product).
__global__ void k_mean_grad(const float* __restrict__ g, const int* __restrict__ start, int n, float* __restrict__ q,
                            int bf16) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / kH;
    if (i >= n) return;
    const float v = g[t] / (float)max(start[i + 1] - start[i], 1);
    q[t] = bf16 ? umma::tf32_round(v) : v;
}

// The message gradients q_i (where their bit is set) of the edges e = (i, j), summed per vertex:
// Gr_i over row i, Gc_i over the reversed edges of row i; and the block partials of
// sum_e gradient f_e^T (2 columns) and sum_e gradient (part[block][c * 2 + k],
// part[block][128 + c], the layout of k_dense_dw for K = 2).  16 lanes per vertex, a block takes
// vertices in steps of the grid.
__global__ void __launch_bounds__(256) k_edge_grad(const float* __restrict__ q, const uint2* __restrict__ bits,
                                                   const float* __restrict__ ef, const int* __restrict__ start,
                                                   const int* __restrict__ col, const int* __restrict__ rev, int n,
                                                   float* __restrict__ Gr, float* __restrict__ Gc,
                                                   float* __restrict__ part, int bf16) {
    __shared__ float sh[16][12 * 16];
    const int lane = threadIdx.x & 15, grp = threadIdx.x / 16;
    float pe[4][2] = {}, pb[4] = {};
    for (int i = blockIdx.x * 16 + grp; i < n; i += gridDim.x * 16) {
        const float4 qi4 = ((const float4*)q)[(size_t)i * 16 + lane];
        const float qi[4] = {qi4.x, qi4.y, qi4.z, qi4.w};
        float gr[4] = {0.f, 0.f, 0.f, 0.f}, gc[4] = {0.f, 0.f, 0.f, 0.f};
        const int e1 = start[i + 1];
#pragma unroll 2
        for (int e = start[i]; e < e1; e++) {
            const uint2 m = bits[e], mr = bits[rev[e]];
            const float4 qj4 = ((const float4*)q)[(size_t)col[e] * 16 + lane];
            const float qj[4] = {qj4.x, qj4.y, qj4.z, qj4.w};
            float2 f = ((const float2*)ef)[e];
            if (bf16) f = make_float2(umma::tf32_round(f.x), umma::tf32_round(f.y));
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const unsigned w = t < 2 ? m.x : m.y, wr = t < 2 ? mr.x : mr.y;
                const int at = lane + (t & 1) * 16;
                const float g = (w >> at) & 1u ? qi[t] : 0.f;
                gr[t] += g;
                if ((wr >> at) & 1u) gc[t] += qj[t];
                pe[t][0] = fmaf(g, f.x, pe[t][0]);
                pe[t][1] = fmaf(g, f.y, pe[t][1]);
            }
        }
        ((float4*)Gr)[(size_t)i * 16 + lane] = make_float4(gr[0], gr[1], gr[2], gr[3]);
        ((float4*)Gc)[(size_t)i * 16 + lane] = make_float4(gc[0], gc[1], gc[2], gc[3]);
#pragma unroll
        for (int t = 0; t < 4; t++) pb[t] += gr[t];
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
        sh[grp][(4 * lane + t) * 2] = pe[t][0];
        sh[grp][(4 * lane + t) * 2 + 1] = pe[t][1];
        sh[grp][128 + 4 * lane + t] = pb[t];
    }
    __syncthreads();
    if (threadIdx.x < 192) {
        float a = 0.f;
        for (int k = 0; k < 16; k++) a += sh[k][threadIdx.x];
        part[(size_t)blockIdx.x * 192 + threadIdx.x] = a;
    }
}

__global__ void k_adam(float* __restrict__ th, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int n, float lr, float b1, float b2, float c1, float c2, float eps) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    th[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

inline int nblk(size_t n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

struct AdmmGnn {
    int n = 0, E = 0, P = 0, bf16 = 1, steps = 0;
    std::vector<void*> allocs, gallocs;  // parameters and optimiser state; per-graph buffers
    int *start = nullptr, *col = nullptr, *rows = nullptr, *rev = nullptr;
    float *val = nullptr, *adiag = nullptr, *x = nullptr, *ef = nullptr;
    float *theta = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
    float *z0 = nullptr, *h[4] = {nullptr, nullptr, nullptr, nullptr};
    float *zm = nullptr, *uv = nullptr;  // messages of a layer (BF16 weights), U then V (FP32)
    float *agg[3] = {nullptr, nullptr, nullptr}, *zn[3] = {nullptr, nullptr, nullptr};
    uint2* bits[3] = {nullptr, nullptr, nullptr};  // per edge: which channels of its message are positive
    float *o = nullptr, *B = nullptr;
    float *gh = nullptr, *gh2 = nullptr, *gz = nullptr, *gnin = nullptr, *go = nullptr, *gB = nullptr;
    float *q = nullptr, *grc = nullptr;  // message gradients per vertex; Gr then Gc
    float *om = nullptr, *oth = nullptr;  // outputs m, theta
    float *part = nullptr, *r = nullptr, *zv = nullptr, *res = nullptr, *gzv = nullptr;
    double *dots = nullptr, *scal = nullptr;
    int* derr = nullptr;    // set by a tensor-core layer whose bounded wait gave up
    bool failed = false;    // a tensor-core layer timed out: outputs undefined, the handle refuses work
    cudaStream_t st = nullptr;
    std::string err;
};

namespace {

// parameter offsets (same order as the CPU restatement)
struct Off {
    int W0, b0, We[3], be[3], Wn[3], bn[3], Wo, bo, total;
};
Off offsets() {
    Off f;
    int k = 0;
    f.W0 = k; k += kH * kFin;
    f.b0 = k; k += kH;
    for (int l = 0; l < 3; l++) {
        f.We[l] = k; k += kH * kEdgeIn;
        f.be[l] = k; k += kH;
        f.Wn[l] = k; k += kH * kNodeIn;
        f.bn[l] = k; k += kH;
    }
    f.Wo = k; k += kOut * kH;
    f.bo = k; k += kOut;
    f.total = k;
    return f;
}

template <class T>
int galloc(AdmmGnn* g, T** p, size_t count, bool graph) {
    if (count == 0) count = 1;
    if (cudaMalloc((void**)p, count * sizeof(T)) != cudaSuccess) return ADMM_ERR_OOM;
    (graph ? g->gallocs : g->allocs).push_back(*p);
    cudaMemset(*p, 0, count * sizeof(T));
    return ADMM_OK;
}

#define GTRY(x)                  \
    do {                         \
        int r_ = (x);            \
        if (r_) return r_;       \
    } while (0)

constexpr size_t gemm_smem(int K) { return sizeof(float) * (size_t)(64 * (K + 4) + K * 68); }
constexpr size_t dw_smem(int KT) { return sizeof(float) * (size_t)(64 * 68 + 64 * (KT + 4)); }
constexpr size_t fwd_smem(int K) { return sizeof(float) * (size_t)(kTcRows + kTcN) * K; }
// no more CTAs per SM than TMEM's 512 columns hold: four of 128 columns, eight of 64
constexpr size_t dx_smem(int NP, int K) {
    const size_t need = sizeof(float) * (size_t)(kTcRows + K) * NP, least = K > 64 ? 52 * 1024 : 26 * 1024;
    return need > least ? need : least;
}

// U (with the bias) and V of layer l with FP32 weights: the two halves of the edge layer's weights.
void edge_halves(AdmmGnn* g, const Off& f, int l) {
    const MatIndex ix = {kEdgeIn, 1, 0, kH};
    k_gemm<kH><<<dim3(nblk(g->n, 64), 2), 256, gemm_smem(kH), g->st>>>(
        g->h[l], g->h[l], g->n, g->theta + f.We[l], ix, g->theta + f.be[l], g->uv, nullptr, nullptr, 0, nullptr, nullptr, 0);
}

// The node layer l: h[l + 1] = h[l] + relu(W [h[l], agg] + b), on the tensor cores with BF16 weights.
void node_layer(AdmmGnn* g, const Off& f, int l) {
    const float *W = g->theta + f.Wn[l], *b = g->theta + f.bn[l];
    if (g->bf16) {
        k_dense_fwd_tc<kNodeIn><<<nblk(g->n, kTcRows), kTcThreads, fwd_smem(kNodeIn), g->st>>>(
            g->h[l], g->agg[l], g->n, kNodeIn, W, kNodeIn, b, g->zn[l], g->h[l + 1], g->h[l], 2, g->derr);
        return;
    }
    const MatIndex ix = {kNodeIn, 1, kH, 0};
    k_gemm<kNodeIn><<<nblk(g->n, 64), 256, gemm_smem(kNodeIn), g->st>>>(g->h[l], g->agg[l], g->n, W, ix, b, g->zn[l],
                                                                       g->h[l + 1], g->h[l], 2, nullptr, nullptr, 0);
}

// dX = dZ W (K = 64 or 128 columns, in [R][64] matrices one after the other): on the tensor cores
// with BF16 weights.
void dense_dx(AdmmGnn* g, const float* dZ, int R, int K, int wo, int N, float* dX) {
    const float* W = g->theta + wo;
    if (g->bf16) {
        const int grid = nblk(R, kTcRows);
        if (N == kH) k_dense_dx_tc<kH, 2 * kH><<<grid, kTcThreads, dx_smem(kH, 2 * kH), g->st>>>(dZ, R, N, W, dX, g->derr);
        else k_dense_dx_tc<8, kH><<<grid, kTcThreads, dx_smem(8, kH), g->st>>>(dZ, R, N, W, dX, g->derr);
    } else if (N == kH) {
        const MatIndex ix = {1, K, 0, kH};
        k_gemm<kH><<<dim3(nblk(R, 64), K / kH), 256, gemm_smem(kH), g->st>>>(dZ, dZ, R, W, ix, nullptr, dX, nullptr,
                                                                            nullptr, 0, nullptr, nullptr, 0);
    } else {
        const size_t sm = sizeof(float) * (size_t)(N * K + 4 * N);
        k_dense_dx<<<nblk(R, 4), 256, sm, g->st>>>(dZ, R, N, W, K, dX, 0);
    }
}

// grad[wo + n ldw + k] += (dZ^T X)[n][k], grad[bo + n] += sum_r dZ[r][n] (bo < 0: none); halves = 2:
// also the next [R][64] matrix of dZ, to weights 64 columns further.
void dense_dw(AdmmGnn* g, const float* dZ, const float* X0, const float* X1, int R, int K, int wo, int ldw, int bo, int N,
              int round_z, int round_x, int halves = 1) {
    const int per = std::max(64, (nblk(R, kDwBlocks) + 63) / 64 * 64), nparts = nblk(R, per);
    const dim3 grid(nparts, halves);
    if (K <= kH) k_dense_dw<kH><<<grid, 256, dw_smem(kH), g->st>>>(dZ, X0, X1, R, per, N, K, round_z, round_x, g->part);
    else k_dense_dw<2 * kH><<<grid, 256, dw_smem(2 * kH), g->st>>>(dZ, X0, X1, R, per, N, K, round_z, round_x, g->part);
    k_reduce_parts<<<dim3(nblk(N * K + N, 32), halves), 1024, 0, g->st>>>(g->part, nparts, N, K, g->grad, wo, ldw, bo);
}

// bits: keep what the gradient needs.  The outputs m and theta go to g->om and g->oth.
void forward(AdmmGnn* g, bool bits) {
    const Off f = offsets();
    const int n = g->n;
    if (g->bf16)
        k_dense_fwd_tc<8><<<nblk(n, kTcRows), kTcThreads, fwd_smem(8), g->st>>>(
            g->x, g->x, n, kFin, g->theta + f.W0, kFin, g->theta + f.b0, g->z0, g->h[0], nullptr, 1, g->derr);
    else
        k_dense_fwd<<<nblk(n, 4), 256, sizeof(float) * (kH * kFin + 4 * kFin), g->st>>>(
            g->x, n, kFin, g->theta + f.W0, g->theta + f.b0, kH, g->z0, g->h[0], nullptr, 1, 0);
    for (int l = 0; l < 3; l++) {
        if (g->bf16) {
            if (g->E > 0)
                k_edge_fwd_tc<<<std::min(nblk(g->E, kTcRows), 2 * 148), kTcThreads, fwd_smem(kEdgeK), g->st>>>(
                    g->h[l], g->ef, g->rows, g->col, g->E, g->theta + f.We[l], g->theta + f.be[l], g->zm, g->derr);
            (bits ? k_node_agg<true> : k_node_agg<false>)<<<nblk((size_t)n * 16, 256), 256, 0, g->st>>>(
                g->zm, g->start, n, g->agg[l], g->bits[l]);
        } else {
            edge_halves(g, f, l);
            (bits ? k_edge_agg<true> : k_edge_agg<false>)<<<nblk((size_t)n * 16, 256), 256, 0, g->st>>>(
                g->uv, g->theta + f.We[l], g->ef, g->start, g->col, n, g->agg[l], g->bits[l]);
        }
        node_layer(g, f, l);
    }
    k_head<<<nblk(n, 64), 256, 0, g->st>>>(g->h[3], g->theta + f.Wo, g->theta + f.bo, g->adiag, n, g->o, g->B, g->om,
                                           g->oth, g->bf16);
}

// ADMM_ERR_TIMEOUT once a tensor-core layer gave up waiting for its MMAs (the
// flag is cleared for the next call).
int tc_status(AdmmGnn* g) {
    int e = 0;
    if (cudaMemcpy(&e, g->derr, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return ADMM_ERR_CUDA;
    if (!e) return ADMM_OK;
    // a CTA that gave up may have left its MMAs reading shared memory and writing TMEM:
    // the outputs of that launch are undefined and the handle takes no further work
    g->failed = true;
    return ADMM_ERR_TIMEOUT;
}

void backward_from_head(AdmmGnn* g);

}  // namespace

extern "C" {

int admm_gnn_create(int bf16, AdmmGnn** out) {
    if (!out) return ADMM_ERR_INVALID;
    *out = nullptr;
    AdmmGnn* g = new (std::nothrow) AdmmGnn;
    if (!g) return ADMM_ERR_OOM;
    g->bf16 = bf16 ? 1 : 0;
    g->P = offsets().total;
    int rc;
    if ((rc = galloc(g, &g->theta, g->P, false)) || (rc = galloc(g, &g->grad, g->P, false)) ||
        (rc = galloc(g, &g->m, g->P, false)) || (rc = galloc(g, &g->v, g->P, false)) ||
        (rc = galloc(g, &g->derr, 1, false))) {
        admm_gnn_destroy(g);
        return rc;
    }
    if (cudaStreamCreateWithFlags(&g->st, cudaStreamNonBlocking) != cudaSuccess) {
        admm_gnn_destroy(g);
        return ADMM_ERR_CUDA;
    }
    cudaFuncSetAttribute(k_dense_fwd_tc<2 * kH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem(2 * kH));
    cudaFuncSetAttribute(k_edge_fwd_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem(kEdgeK));
    cudaFuncSetAttribute(k_dense_dx_tc<kH, 2 * kH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dx_smem(kH, 2 * kH));
    cudaFuncSetAttribute(k_gemm<kH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(kH));
    cudaFuncSetAttribute(k_gemm<2 * kH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(2 * kH));
    cudaFuncSetAttribute(k_dense_dw<kH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dw_smem(kH));
    cudaFuncSetAttribute(k_dense_dw<2 * kH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dw_smem(2 * kH));
    *out = g;
    return ADMM_OK;
}

// The graph the next calls work on (replaces the previous one; parameters and
// optimiser state are kept, so one network trains on many systems).
int admm_gnn_set_graph(AdmmGnn* g, int n, int n_edges, const int32_t* start, const int32_t* col, const float* val,
                       const float* adiag, const float* node_feat, const float* edge_feat) {
    if (!g || n <= 0 || n_edges < 0 || !start || !adiag || !node_feat || (n_edges > 0 && (!col || !val || !edge_feat)))
        return ADMM_ERR_INVALID;
    cudaStreamSynchronize(g->st);
    for (void* p : g->gallocs) cudaFree(p);
    g->gallocs.clear();
    g->n = n;
    g->E = n_edges;
    std::vector<int> rows(n_edges), rev(n_edges, 0);
    for (int i = 0; i < n; i++)
        for (int e = start[i]; e < start[i + 1]; e++) rows[e] = i;
    for (int i = 0; i < n; i++)  // reverse edge: (j -> i) in row j, binary search (columns sorted)
        for (int e = start[i]; e < start[i + 1]; e++) {
            const int j = col[e];
            int lo = start[j], hi = start[j + 1] - 1, k = -1;
            while (lo <= hi) {
                const int mid = (lo + hi) / 2;
                if (col[mid] == i) { k = mid; break; }
                if (col[mid] < i) lo = mid + 1; else hi = mid - 1;
            }
            if (k < 0) return ADMM_ERR_INVALID;  // the pattern must be symmetric with sorted columns
            rev[e] = k;
        }
    auto up = [&](auto** p, const auto* src, size_t cnt) -> int {
        GTRY(galloc(g, p, cnt, true));
        if (cnt && src) cudaMemcpy(*p, src, cnt * sizeof(**p), cudaMemcpyHostToDevice);
        return ADMM_OK;
    };
    auto ga = [&](auto** p, size_t cnt) -> int { return galloc(g, p, cnt, true); };
    const size_t H = kH, N = n, Ee = n_edges;
    int rc = ADMM_OK;
    if ((rc = up(&g->start, start, N + 1)) || (rc = up(&g->col, col, Ee)) || (rc = up(&g->rows, rows.data(), Ee)) ||
        (rc = up(&g->rev, rev.data(), Ee)) || (rc = up(&g->val, val, Ee)) || (rc = up(&g->adiag, adiag, N)) ||
        (rc = up(&g->x, node_feat, N * kFin)) || (rc = up(&g->ef, edge_feat, Ee * kFe)) || (rc = ga(&g->z0, N * H)) ||
        (rc = ga(&g->o, N * kOut)) || (rc = ga(&g->B, N * 9)) || (rc = ga(&g->gh, N * H)) || (rc = ga(&g->gh2, N * H)) ||
        (rc = ga(&g->gz, N * H)) || (rc = ga(&g->gnin, N * kNodeIn)) || (rc = g->bf16 ? ga(&g->zm, Ee * H) : ga(&g->uv, 2 * N * H)) ||
        (rc = ga(&g->q, N * H)) || (rc = ga(&g->grc, 2 * N * H)) || (rc = ga(&g->om, N)) || (rc = ga(&g->oth, N)) ||
        (rc = ga(&g->go, N * kOut)) || (rc = ga(&g->gB, N * 9)) ||
        (rc = ga(&g->part, (size_t)std::min(kDwBlocks, nblk(N, 64)) * 2 * (kH * kNodeIn + kH))) ||
        (rc = ga(&g->r, N * 3)) || (rc = ga(&g->zv, N * 3)) || (rc = ga(&g->res, N * 3)) || (rc = ga(&g->gzv, N * 3)) ||
        (rc = ga(&g->dots, 1024)) || (rc = ga(&g->scal, 4)))
        return rc;
    for (int l = 0; l < 4; l++) GTRY(ga(&g->h[l], N * H));
    for (int l = 0; l < 3; l++) {
        GTRY(ga(&g->agg[l], N * H));
        GTRY(ga(&g->bits[l], Ee));
        GTRY(ga(&g->zn[l], N * H));
    }
    return cudaGetLastError() == cudaSuccess ? ADMM_OK : ADMM_ERR_CUDA;
}

void admm_gnn_destroy(AdmmGnn* g) {
    if (!g) return;
    if (g->st) {
        cudaStreamSynchronize(g->st);
        cudaStreamDestroy(g->st);
    }
    for (void* p : g->allocs) cudaFree(p);
    for (void* p : g->gallocs) cudaFree(p);
    delete g;
}

int admm_gnn_num_params(void) { return offsets().total; }

int admm_gnn_set_params(AdmmGnn* g, const float* theta, int P) {
    if (!g || !theta || P != g->P) return ADMM_ERR_INVALID;
    if (cudaMemcpy(g->theta, theta, sizeof(float) * P, cudaMemcpyHostToDevice) != cudaSuccess) return ADMM_ERR_CUDA;
    cudaMemset(g->m, 0, sizeof(float) * P);  // a new starting point: the optimiser starts afresh
    cudaMemset(g->v, 0, sizeof(float) * P);
    g->steps = 0;
    return ADMM_OK;
}

int admm_gnn_get_params(AdmmGnn* g, float* theta, int P) {
    if (!g || !theta || P != g->P) return ADMM_ERR_INVALID;
    cudaStreamSynchronize(g->st);
    return cudaMemcpy(theta, g->theta, sizeof(float) * P, cudaMemcpyDeviceToHost) == cudaSuccess ? ADMM_OK : ADMM_ERR_CUDA;
}

// Forward pass; blocks9 (host, n x 9 row-major) receives B_i = L_i L_i^T / a_ii.
int admm_gnn_forward(AdmmGnn* g, float* blocks9) {
    if (!g || g->n <= 0) return ADMM_ERR_INVALID;
    if (g->failed) return ADMM_ERR_STATE;
    forward(g, false);
    if (blocks9 && cudaMemcpyAsync(blocks9, g->B, sizeof(float) * 9 * (size_t)g->n, cudaMemcpyDeviceToHost, g->st) != cudaSuccess)
        return ADMM_ERR_CUDA;
    if (cudaStreamSynchronize(g->st) != cudaSuccess) return ADMM_ERR_CUDA;
    if (cudaGetLastError() != cudaSuccess) return ADMM_ERR_CUDA;
    return tc_status(g);
}

// Loss mean_k |A B r_k - r_k|^2 / |r_k|^2 over K residual samples (host, K x n x 3)
// and, into the gradient buffer (zeroed first), its gradient; grad (host, may be
// null) receives it.
int admm_gnn_loss_grad(AdmmGnn* g, const float* R, int K, double* loss, float* grad) {
    if (!g || g->n <= 0 || !R || K <= 0) return ADMM_ERR_INVALID;
    if (g->failed) return ADMM_ERR_STATE;
    const int n = g->n;
    forward(g, true);
    cudaMemsetAsync(g->grad, 0, sizeof(float) * g->P, g->st);
    cudaMemsetAsync(g->gB, 0, sizeof(float) * 9 * (size_t)n, g->st);
    double total = 0.0;
    const int nb = 256;
    for (int k = 0; k < K; k++) {
        cudaMemcpyAsync(g->r, R + (size_t)k * n * 3, sizeof(float) * 3 * (size_t)n, cudaMemcpyHostToDevice, g->st);
        k_apply_blocks<<<nblk(n, 256), 256, 0, g->st>>>(g->B, g->r, n, g->zv);
        k_spmv3<<<nblk(n, 256), 256, 0, g->st>>>(g->start, g->col, g->val, g->adiag, g->zv, n, g->res, g->r);
        k_dot_parts<<<nb, 256, 0, g->st>>>(g->r, g->r, 3 * n, g->dots);
        k_dot_parts<<<nb, 256, 0, g->st>>>(g->res, g->res, 3 * n, g->dots + nb);
        std::vector<double> d(2 * nb);
        cudaMemcpyAsync(d.data(), g->dots, sizeof(double) * 2 * nb, cudaMemcpyDeviceToHost, g->st);
        if (cudaStreamSynchronize(g->st) != cudaSuccess) return ADMM_ERR_CUDA;
        double rr = 0.0, ee = 0.0;
        for (int b = 0; b < nb; b++) { rr += d[b]; ee += d[nb + b]; }
        if (!(rr > 0.0)) continue;
        total += ee / rr / K;
        const double sc = 2.0 / (rr * K);
        cudaMemcpyAsync(g->scal, &sc, sizeof(double), cudaMemcpyHostToDevice, g->st);
        k_spmv3<<<nblk(n, 256), 256, 0, g->st>>>(g->start, g->col, g->val, g->adiag, g->res, n, g->gzv, nullptr);
        k_accum_gB<<<nblk(n, 256), 256, 0, g->st>>>(g->gzv, g->r, n, g->scal, g->gB);
        if (cudaStreamSynchronize(g->st) != cudaSuccess) return ADMM_ERR_CUDA;
    }
    k_head_grad<<<nblk(n, 256), 256, 0, g->st>>>(g->gB, g->o, g->adiag, n, g->go, nullptr);
    backward_from_head(g);
    if (grad) cudaMemcpyAsync(grad, g->grad, sizeof(float) * g->P, cudaMemcpyDeviceToHost, g->st);
    if (cudaStreamSynchronize(g->st) != cudaSuccess || cudaGetLastError() != cudaSuccess) return ADMM_ERR_CUDA;
    if (loss) *loss = total;
    return tc_status(g);
}

// Per-vertex outputs of the learned global step: m (n) and theta (n), host.
int admm_gnn_outputs(AdmmGnn* g, float* m, float* theta) {
    if (!g || g->n <= 0 || !m || !theta) return ADMM_ERR_INVALID;
    if (g->failed) return ADMM_ERR_STATE;
    forward(g, false);
    cudaMemcpyAsync(m, g->om, sizeof(float) * g->n, cudaMemcpyDeviceToHost, g->st);
    cudaMemcpyAsync(theta, g->oth, sizeof(float) * g->n, cudaMemcpyDeviceToHost, g->st);
    if (cudaStreamSynchronize(g->st) != cudaSuccess || cudaGetLastError() != cudaSuccess) return ADMM_ERR_CUDA;
    return tc_status(g);
}

// Gradient of a loss with respect to the parameters, given its gradients gm and
// gtheta (host, n each) with respect to the outputs of admm_gnn_outputs (at the
// current parameters and graph); grad (host, may be null) receives it, and the
// next admm_gnn_adam applies it.
int admm_gnn_backward(AdmmGnn* g, const float* gm, const float* gtheta, float* grad) {
    if (!g || g->n <= 0 || !gm || !gtheta) return ADMM_ERR_INVALID;
    if (g->failed) return ADMM_ERR_STATE;
    const int n = g->n;
    forward(g, true);
    cudaMemsetAsync(g->grad, 0, sizeof(float) * g->P, g->st);
    cudaMemcpyAsync(g->r, gm, sizeof(float) * n, cudaMemcpyHostToDevice, g->st);
    cudaMemcpyAsync(g->zv, gtheta, sizeof(float) * n, cudaMemcpyHostToDevice, g->st);
    k_gm_to_gB<<<nblk(n, 256), 256, 0, g->st>>>(g->r, n, g->gB);
    k_head_grad<<<nblk(n, 256), 256, 0, g->st>>>(g->gB, g->o, g->adiag, n, g->go, g->zv);
    backward_from_head(g);
    if (grad) cudaMemcpyAsync(grad, g->grad, sizeof(float) * g->P, cudaMemcpyDeviceToHost, g->st);
    if (cudaStreamSynchronize(g->st) != cudaSuccess || cudaGetLastError() != cudaSuccess) return ADMM_ERR_CUDA;
    return tc_status(g);
}

}  // extern "C"

namespace {

// The backward pass from the head gradient go (dL/do) into g->grad.
void backward_from_head(AdmmGnn* g) {
    const Off f = offsets();
    const int n = g->n;
    const int tc = g->bf16;
    const size_t nh = (size_t)n * kH;
    dense_dx(g, g->go, n, kH, f.Wo, kOut, g->gh);  // gh = dL/dh3
    dense_dw(g, g->go, g->h[3], g->h[3], n, kH, f.Wo, kH, f.bo, kOut, tc, tc);
    for (int l = 2; l >= 0; l--) {
        k_relu_mask<<<nblk(nh, 256), 256, 0, g->st>>>(g->gh, g->zn[l], nh, g->gz);  // gzn
        dense_dx(g, g->gz, n, kNodeIn, f.Wn[l], kH, g->gnin);
        dense_dw(g, g->gz, g->h[l], g->agg[l], n, kNodeIn, f.Wn[l], kNodeIn, f.bn[l], kH, tc, tc);
        k_mean_grad<<<nblk(nh, 256), 256, 0, g->st>>>(g->gnin + nh, g->start, n, g->q, tc);
        const int eb = std::min(nblk(n, 16), kDwBlocks);
        float* gc = g->grc + nh;
        k_edge_grad<<<eb, 256, 0, g->st>>>(g->q, g->bits[l], g->ef, g->start, g->col, g->rev, n, g->grc, gc, g->part, tc);
        k_reduce_parts<<<nblk(3 * kH, 32), 1024, 0, g->st>>>(g->part, eb, kH, kFe, g->grad, f.We[l] + 2 * kH, kEdgeIn, f.be[l]);
        dense_dw(g, g->grc, g->h[l], g->h[l], n, kH, f.We[l], kEdgeIn, -1, kH, 0, tc, 2);
        // gh <- gh + (h half of gnin) + Gr W_r + Gc W_c
        const MatIndex ix = {1, kEdgeIn, kH, 0};
        k_gemm<2 * kH><<<nblk(n, 64), 256, gemm_smem(2 * kH), g->st>>>(g->grc, gc, n, g->theta + f.We[l], ix, nullptr,
                                                                      g->gh2, nullptr, nullptr, 0, g->gh, g->gnin, tc);
        std::swap(g->gh, g->gh2);
    }
    k_relu_mask<<<nblk(nh, 256), 256, 0, g->st>>>(g->gh, g->z0, nh, g->gz);
    dense_dw(g, g->gz, g->x, g->x, n, kFin, f.W0, kFin, f.b0, kH, tc, tc);
}

}  // namespace

extern "C" {

// One Adam step on the gradient of the last admm_gnn_loss_grad.
int admm_gnn_adam(AdmmGnn* g, float lr) {
    if (!g) return ADMM_ERR_INVALID;
    g->steps++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)g->steps), c2 = 1.f - std::pow(b2, (float)g->steps);
    k_adam<<<nblk(g->P, 256), 256, 0, g->st>>>(g->theta, g->grad, g->m, g->v, g->P, lr, b1, b2, c1, c2, 1e-8f);
    return cudaStreamSynchronize(g->st) == cudaSuccess ? ADMM_OK : ADMM_ERR_CUDA;
}

}  // extern "C"
