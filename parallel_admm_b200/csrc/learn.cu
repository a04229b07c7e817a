// learn.cu -- training of the learned global step (an addition with no
// reference counterpart): the loss of K unrolled sweeps of
//
//     x_0 = x_c + theta (x_c - x_l),
//     x_{k+1} = x_k + omega_k m (b - A x_k) + beta_k (x_k - x_{k-1})   (beta_0 = 0),
//
// L = (x_K - x*)^T A (x_K - x*) / ((x_c - x*)^T A (x_c - x*))
//     + mu |b - A x_K|^2 / |b - A x_c|^2   (mu = 0 unless set: the relative residual of the last iterate),
// averaged over samples (b, x_c, x_l, x*) that plain runs produce, and its gradient with
// respect to omega, beta (per sweep), m and theta (per vertex) by the adjoint
// recursion (A symmetric, b - A x = -A (x - x*)):
//
//     g_K = 2 A (x_K - x*) / E_c + mu 2 A A (x_K - x*) / R_c,
//     g_k = (1 + beta_k) g_{k+1} - omega_k A (m g_{k+1}) - beta_{k+1} g_{k+2},
//     dL/domega_k = g_{k+1} . m r_k,   dL/dbeta_k = g_{k+1} . (x_k - x_{k-1}),
//     dL/dm_i = sum_k omega_k g_{k+1,i} . r_{k,i},   dL/dtheta_i = g_{0,i} . (x_c - x_l)_i.
//
// Also a conjugate-gradient solve of A x* = b (the converged solution of a
// sample).  One thread per row over a CSR copy of A (off-diagonal part plus
// diagonal), all samples of a batch in one launch; the dot products are FP64 block partials
// summed in a fixed order on the device, so a gradient is deterministic.  The FP64 restatement that the
// tests check these kernels against is in the oracle directory.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <new>
#include <vector>

#include "admm_b200.h"
#include "common.cuh"

namespace {

constexpr int kT = 128;
constexpr int kParts = 592;  // most blocks of the reduction kernels (4 x 148 SMs)
// CG iterations queued between two looks at their state: a look costs some 10 us, an iteration
// queued past the end 3 us.
constexpr int kCgChunk = 16;
constexpr int kCgAhead = 16;  // entries of a row loaded before the dependency wait
// most blocks of a conjugate-gradient kernel (16 x 148 SMs: every thread the device holds at once;
// 1.45 M rows, 128 iterations: 23 ms against 28 with kParts)
constexpr int kCgParts = 2368;
constexpr int kMaxK = 32;

inline int nblk(size_t n, int t) { return (int)((n + t - 1) / t); }

// out_i = (A v)_i over 3 columns
__device__ __forceinline__ void row_spmv(const int* __restrict__ start, const int* __restrict__ col,
                                         const float* __restrict__ val, const float* __restrict__ diag,
                                         const float* __restrict__ v, int i, float out[3]) {
    float a0 = diag[i] * v[3 * i], a1 = diag[i] * v[3 * i + 1], a2 = diag[i] * v[3 * i + 2];
#pragma unroll 4
    for (int e = start[i]; e < start[i + 1]; e++) {
        const int j = col[e];
        const float w = val[e];
        a0 = fmaf(w, v[3 * j], a0);
        a1 = fmaf(w, v[3 * j + 1], a1);
        a2 = fmaf(w, v[3 * j + 2], a2);
    }
    out[0] = a0;
    out[1] = a1;
    out[2] = a2;
}

// Block sum of two doubles (fixed order) into out0[0], out1[0] by thread 0; sh: 2 x kT.
__device__ __forceinline__ void block_sum2(double a, double b, double* sh, double* out0, double* out1) {
    sh[threadIdx.x] = a;
    sh[kT + threadIdx.x] = b;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            sh[threadIdx.x] += sh[threadIdx.x + o];
            sh[kT + threadIdx.x] += sh[kT + threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *out0 = sh[0];
        if (out1) *out1 = sh[kT];
    }
}

// The kernels of a loss and its gradient take all samples of a batch at once: blockIdx.y is the
// sample, its vectors at sample * n3.  Everything between the upload and the download stays on
// the device (with the sums read back by the host, a sample of K = 6 sweeps waited 8 times).
struct TrainMat {
    const int *start, *col;
    const float *val, *diag;
    int n;
    size_t n3;
};

// ae = A (x - xs); block partials of (x - xs) . A (x - xs) and of |A (x - xs)|^2 into
// part[sample][0 / 1][block].  x0 (first pass): x0 = xc + theta (xc - xl), xc = x.
__global__ void __launch_bounds__(kT) k_t_error(TrainMat M, const float* __restrict__ x, const float* __restrict__ xs,
                                                const float* __restrict__ xl, const float* __restrict__ th,
                                                float* __restrict__ x0, float* __restrict__ ae,
                                                double* __restrict__ part) {
    __shared__ double sh[2 * kT];
    const size_t off = blockIdx.y * M.n3;
    x += off;
    xs += off;
    double e2 = 0.0, r2 = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M.n; i += gridDim.x * blockDim.x) {
        const float e[3] = {x[3 * i] - xs[3 * i], x[3 * i + 1] - xs[3 * i + 1], x[3 * i + 2] - xs[3 * i + 2]};
        float a[3] = {M.diag[i] * e[0], M.diag[i] * e[1], M.diag[i] * e[2]};
#pragma unroll 4
        for (int k = M.start[i]; k < M.start[i + 1]; k++) {
            const int j = M.col[k];
            const float w = M.val[k];
            for (int c = 0; c < 3; c++) a[c] = fmaf(w, x[3 * j + c] - xs[3 * j + c], a[c]);
        }
        for (int c = 0; c < 3; c++) {
            ae[off + 3 * i + c] = a[c];
            e2 += (double)a[c] * (double)e[c];
            r2 += (double)a[c] * (double)a[c];
            if (x0) x0[off + 3 * i + c] = fmaf(th[i], x[3 * i + c] - xl[off + 3 * i + c], x[3 * i + c]);
        }
    }
    double* p = part + (size_t)blockIdx.y * 2 * gridDim.x;
    block_sum2(e2, r2, sh, p + blockIdx.x, p + gridDim.x + blockIdx.x);
}

// r_k = b - A x_k; x_{k+1} = x_k + omega m r_k + beta (x_k - x_{k-1})
__global__ void __launch_bounds__(kT) k_t_sweep(TrainMat M, const float* __restrict__ m, const float* __restrict__ b,
                                                const float* __restrict__ xk, const float* __restrict__ xkm1,
                                                float omega, float beta, float* __restrict__ rk,
                                                float* __restrict__ xk1) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M.n) return;
    const size_t off = blockIdx.y * M.n3;
    float ax[3];
    row_spmv(M.start, M.col, M.val, M.diag, xk + off, i, ax);
    for (int c = 0; c < 3; c++) {
        const size_t q = off + 3 * i + c;
        const float r = b[q] - ax[c];
        rk[q] = r;
        xk1[q] = fmaf(omega * m[i], r, fmaf(beta, xk[q] - xkm1[q], xk[q]));
    }
}

// Sum of n partials in a fixed order, the same in every thread of the block; sh: 2 x kT.
__device__ __forceinline__ double parts_sum(const double* p, int n, double* sh) {
    double a = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) a += p[k];
    __shared__ double total;
    __syncthreads();
    block_sum2(a, 0.0, sh, &total, nullptr);
    __syncthreads();
    return total;
}

// Per sample (blockIdx.x): scal = E_c, R_c, E_K, R_K from the partials of the two k_t_error passes.
__global__ void __launch_bounds__(kT) k_t_scalars(const double* __restrict__ pc, const double* __restrict__ pK, int nb,
                                                  double* __restrict__ scal) {
    __shared__ double sh[2 * kT];
    const size_t at = (size_t)blockIdx.x * 2 * nb;
    for (int k = 0; k < 4; k++) {
        const double v = parts_sum((k < 2 ? pc : pK) + at + (k & 1) * nb, nb, sh);
        if (threadIdx.x == 0) scal[4 * blockIdx.x + k] = v;
    }
}

// The adjoint's seed g_K = 2 A e_K / (E_c nsamp) (+ mu 2 A A e_K / (R_c nsamp)); a sample whose x_c is
// the solution (E_c = 0) is left out.
__global__ void __launch_bounds__(kT) k_t_seed(TrainMat M, const float* __restrict__ ae, const double* __restrict__ scal,
                                               double mu, int nsamp, float* __restrict__ g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M.n) return;
    const size_t off = blockIdx.y * M.n3;
    const double Ec = scal[4 * blockIdx.y], Rc = scal[4 * blockIdx.y + 1];
    const bool used = Ec > 0.0, res = mu > 0.0 && Rc > 0.0;
    float a2[3] = {0.f, 0.f, 0.f};
    if (used && res) row_spmv(M.start, M.col, M.val, M.diag, ae + off, i, a2);
    for (int c = 0; c < 3; c++) {
        const size_t q = off + 3 * i + c;
        double v = used ? (double)ae[q] * (2.0 / (Ec * nsamp)) : 0.0;
        if (used && res) v += (double)a2[c] * (mu * 2.0 / (Rc * nsamp));
        g[q] = (float)v;
    }
}

// One adjoint step k: gk = (1 + beta_k) g1 - omega_k A (m g1) - beta_{k+1} g2 (g2 may be
// null); partials of g1 . m r_k and g1 . (x_k - x_{k-1}) into part[0 / 1][sample][block];
// gm_i (+)= omega_k g1_i . r_k,i per sample (first: set).
__global__ void __launch_bounds__(kT) k_t_adjoint(TrainMat M, const float* __restrict__ m, const double* __restrict__ scal,
                                                  const float* __restrict__ g1, const float* __restrict__ g2,
                                                  const float* __restrict__ rk, const float* __restrict__ xk,
                                                  const float* __restrict__ xkm1, float omega, float beta_k,
                                                  float beta_k1, int first, float* __restrict__ gk,
                                                  float* __restrict__ gm, double* __restrict__ part) {
    __shared__ double sh[2 * kT];
    const size_t off = blockIdx.y * M.n3;
    const bool used = scal[4 * blockIdx.y] > 0.0;
    double ao = 0.0, ab = 0.0;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M.n) {
        float gmi = 0.f;
        if (used) {
            const float* g = g1 + off;
            // A (m g1) row i
            float a0 = M.diag[i] * m[i] * g[3 * i], a1 = M.diag[i] * m[i] * g[3 * i + 1],
                  a2 = M.diag[i] * m[i] * g[3 * i + 2];
#pragma unroll 4
            for (int e = M.start[i]; e < M.start[i + 1]; e++) {
                const int j = M.col[e];
                const float w = M.val[e] * m[j];
                a0 = fmaf(w, g[3 * j], a0);
                a1 = fmaf(w, g[3 * j + 1], a1);
                a2 = fmaf(w, g[3 * j + 2], a2);
            }
            const float amg[3] = {a0, a1, a2};
            for (int c = 0; c < 3; c++) {
                const size_t q = off + 3 * i + c;
                const float gi = g1[q], ri = rk[q];
                float v = fmaf(1.f + beta_k, gi, -omega * amg[c]);
                if (g2) v = fmaf(-beta_k1, g2[q], v);
                gk[q] = v;
                ao += (double)gi * (double)m[i] * (double)ri;
                ab += (double)gi * ((double)xk[q] - (double)xkm1[q]);
                gmi = fmaf(gi, ri, gmi);
            }
        } else {
            for (int c = 0; c < 3; c++) gk[off + 3 * i + c] = 0.f;
        }
        const size_t at = (size_t)blockIdx.y * M.n + i;
        gm[at] = fmaf(omega, gmi, first ? 0.f : gm[at]);
    }
    const size_t at = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
    block_sum2(ao, ab, sh, part + at, part + (size_t)gridDim.y * gridDim.x + at);
}

// gm_i += the samples' gm_i, gth_i += sum over the samples of g0_i . (xc - xl)_i; the last blocks:
// the sums over all partials of dL/domega_k (block -> 2 k) and dL/dbeta_k (2 k + 1) onto coef.
__global__ void __launch_bounds__(kT) k_t_collect(TrainMat M, const double* __restrict__ scal, const float* __restrict__ g0,
                                                  const float* __restrict__ xc, const float* __restrict__ xl,
                                                  const float* __restrict__ gms, int S, int row_blocks,
                                                  const double* __restrict__ part, int parts, float* __restrict__ gm,
                                                  float* __restrict__ gth, double* __restrict__ coef) {
    __shared__ double sh[2 * kT];
    if ((int)blockIdx.x >= row_blocks) {
        const int k = blockIdx.x - row_blocks;
        const double v = parts_sum(part + (size_t)k * parts, parts, sh);
        if (threadIdx.x == 0) coef[k] += v;
        return;
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M.n) return;
    float a = gm[i], t = gth[i];
    for (int s = 0; s < S; s++) {
        a += gms[(size_t)s * M.n + i];
        if (!(scal[4 * s] > 0.0)) continue;
        float d = 0.f;
        for (int c = 0; c < 3; c++) {
            const size_t q = s * M.n3 + 3 * i + c;
            d = fmaf(g0[q], xc[q] - xl[q], d);
        }
        t += d;
    }
    gm[i] = a;
    gth[i] = t;
}

// ---- conjugate gradients (diag(A) preconditioned) for the converged solution ----
// Two launches per iteration (three above kFusedRows rows), the scalars on the device: every block of a kernel sums the
// partials that the kernel before it left.  Once the iteration has ended (done), the kernels
// still queued do nothing.  The kernels start before their predecessor has ended (programmatic
// launch) and load what does not change, the matrix and its diagonal, before they wait for it: at
// 9261 rows, where the launches and each row's chain of loads bound the time, 17 against 24 us per
// iteration.
struct CgState {
    double rz0, rz, pq;  // (r, z) at the start, now; (p, A p)
    int iters, done;
};

// r = b - A x, z = r / a; part = r . z
__global__ void __launch_bounds__(kT) k_cg_init(TrainMat M, const float* __restrict__ b, const float* __restrict__ x,
                                                float* __restrict__ r, float* __restrict__ z, double* __restrict__ part) {
    __shared__ double sh[2 * kT];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M.n; i += gridDim.x * blockDim.x) {
        float a[3];
        row_spmv(M.start, M.col, M.val, M.diag, x, i, a);
        for (int c = 0; c < 3; c++) {
            const int q = 3 * i + c;
            const float rr = b[q] - a[c], zz = rr / M.diag[i];
            r[q] = rr;
            z[q] = zz;
            acc += (double)rr * (double)zz;
        }
    }
    block_sum2(acc, 0.0, sh, part + blockIdx.x, nullptr);
}

// Up to so many rows k_cg_q makes the direction itself: a launch less, but every neighbour's z and p
// gathered and combined in FP64.  128 iterations on rows of 14 entries, direction in k_cg_q / in k_cg_p:
// 9 k rows 1.85 / 1.92 ms, 16 k 1.88 / 1.85, 100 k 4.0 / 3.2, 1.45 M 30.7 / 22.7.
constexpr int kFusedRows = 16384;

// Entry q of the direction z + beta p (p null: z).
__device__ __forceinline__ float cg_direction(const float* z, const float* p, int q,
                                              double beta) {
    return p ? (float)((double)z[q] + beta * (double)p[q]) : z[q];
}

// The state at the start of iteration `it`, by every block alike: rz = the sum of the partials of the
// last kernel; ends here (false) once rz has dropped by rel_tol^2, or is 0; else *beta for the new
// direction.
__device__ __forceinline__ bool cg_begin(int nparts, const double* parts_in, double rel_tol2, int it, const CgState* old,
                                         CgState* cur, double* sh, double* beta) {
    const CgState s0 = *old;
    const double rz = s0.done ? s0.rz : parts_sum(parts_in, nparts, sh);
    const double rz0 = it == 0 ? rz : s0.rz0;
    const bool done = s0.done || !(rz > rel_tol2 * rz0 && rz > 0.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        CgState c = s0;
        c.rz0 = rz0;
        c.rz = rz;
        c.done = done;
        *cur = c;
    }
    *beta = it == 0 ? 0.0 : rz / s0.rz;
    return !done;
}

// The direction of iteration `it` on its own, before k_cg_q<false>: p = z + (rz / rz_old) p.
__global__ void __launch_bounds__(kT) k_cg_p(TrainMat M, const float* z, float* p, int nparts, const double* parts_in,
                                             double rel_tol2, int it, const CgState* old, CgState* cur) {
    __shared__ double sh[2 * kT];
    ADMM_PDL_PROLOGUE();
    double beta;
    if (!cg_begin(nparts, parts_in, rel_tol2, it, old, cur, sh, &beta)) return;
    for (size_t k = blockIdx.x * blockDim.x + threadIdx.x; k < M.n3; k += gridDim.x * blockDim.x)
        p[k] = it == 0 ? z[k] : (float)((double)z[k] + beta * (double)p[k]);
}

// Iteration `it`, unless it ends in cg_begin: p_new = z + (rz / rz_old) p and q = A p_new (the
// neighbours' p_new computed from their z and p), part = p_new . q.  FUSED = false: p_new is z, and
// the state cur, from k_cg_p.
template <bool FUSED>
__global__ void __launch_bounds__(kT) k_cg_q(TrainMat M, const float* z, const float* p,
                                             int nparts, const double* parts_in, double rel_tol2, int it,
                                             const CgState* old, CgState* cur,
                                             float* pn, float* q, double* part) {
    __shared__ double sh[2 * kT];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int first = blockIdx.x * blockDim.x + threadIdx.x;
    int e0 = 0, e1 = 0, ahead_col[kCgAhead];
    float ahead_val[kCgAhead], diag0 = 0.f;
    if (first < M.n) {
        e0 = M.start[first];
        e1 = M.start[first + 1];
        diag0 = M.diag[first];
    }
#pragma unroll
    for (int k = 0; k < kCgAhead; k++) {
        ahead_col[k] = e0 + k < e1 ? M.col[e0 + k] : 0;
        ahead_val[k] = e0 + k < e1 ? M.val[e0 + k] : 0.f;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    double beta = 0.0;
    if (FUSED ? !cg_begin(nparts, parts_in, rel_tol2, it, old, cur, sh, &beta) : cur->done != 0) return;
    const float* pp = FUSED && it > 0 ? p : nullptr;
    double acc = 0.0;
    for (int i = first; i < M.n; i += gridDim.x * blockDim.x) {
        const bool ahead = i == first;
        const float d = ahead ? diag0 : M.diag[i];
        float pi[3], a[3];
        for (int c = 0; c < 3; c++) {
            pi[c] = cg_direction(z, pp, 3 * i + c, beta);
            a[c] = d * pi[c];
        }
        int e = ahead ? e0 : M.start[i];
        const int end = ahead ? e1 : M.start[i + 1];
        if (ahead) {
#pragma unroll
            for (int k = 0; k < kCgAhead; k++)
                if (e0 + k < e1)
                    for (int c = 0; c < 3; c++)
                        a[c] = fmaf(ahead_val[k], cg_direction(z, pp, 3 * ahead_col[k] + c, beta), a[c]);
            e += kCgAhead;
        }
#pragma unroll 4
        for (; e < end; e++) {
            const int j = M.col[e];
            const float w = M.val[e];
            for (int c = 0; c < 3; c++) a[c] = fmaf(w, cg_direction(z, pp, 3 * j + c, beta), a[c]);
        }
        for (int c = 0; c < 3; c++) {
            if (FUSED) pn[3 * i + c] = pi[c];
            q[3 * i + c] = a[c];
            acc += (double)a[c] * (double)pi[c];
        }
    }
    block_sum2(acc, 0.0, sh, part + blockIdx.x, nullptr);
}

// alpha = rz / (p . q) (ends the iteration when p . q is not positive); x += alpha p, r -= alpha q;
// z = r / a, part = r . z (the new rz)
__global__ void __launch_bounds__(kT) k_cg_xr(TrainMat M, const float* p, const float* q,
                                              int nparts, const double* parts_in,
                                              const CgState* old, CgState* cur,
                                              float* x, float* r, float* z,
                                              double* part) {
    __shared__ double sh[2 * kT];
    ADMM_PDL_PROLOGUE();
    const CgState s0 = *old;
    const double pq = s0.done ? 1.0 : parts_sum(parts_in, nparts, sh);
    const bool done = s0.done || !(pq > 0.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        CgState c = s0;
        c.done = done;
        if (!done) c.iters = s0.iters + 1;
        *cur = c;
    }
    if (done) return;
    const double alpha = s0.rz / pq;
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M.n; i += gridDim.x * blockDim.x)
        for (int c = 0; c < 3; c++) {
            const int k = 3 * i + c;
            x[k] = (float)((double)x[k] + alpha * (double)p[k]);
            const float rr = (float)((double)r[k] - alpha * (double)q[k]);
            const float zz = rr / M.diag[i];
            r[k] = rr;
            z[k] = zz;
            acc += (double)rr * (double)zz;
        }
    block_sum2(acc, 0.0, sh, part + blockIdx.x, nullptr);
}

}  // namespace

struct AdmmLearn {
    int n = 0, nnz = 0;
    std::vector<void*> allocs;
    int *start = nullptr, *col = nullptr;
    float *val = nullptr, *diag = nullptr, *m = nullptr, *th = nullptr;
    float *gm = nullptr, *gth = nullptr;
    double* coef = nullptr;  // [2 kMaxK] dL/domega_k, dL/dbeta_k interleaved
    double mu = 0.0;         // weight of the residual term
    size_t batch_bytes = (size_t)2 << 30;  // most a batch's vectors may take (one sample at least)
    // workspaces, one sample's from the start, grown to the largest call: a batch's vectors; the
    // partials and scalars
    float* work = nullptr;
    size_t work_floats = 0;
    double* dwork = nullptr;
    size_t dwork_doubles = 0;
    cudaStream_t st = nullptr;
};

namespace {

template <class T>
int lalloc(AdmmLearn* L, T** p, size_t count) {
    if (count == 0) count = 1;
    if (cudaMalloc((void**)p, count * sizeof(T)) != cudaSuccess) return ADMM_ERR_OOM;
    L->allocs.push_back(*p);
    cudaMemset(*p, 0, count * sizeof(T));
    return ADMM_OK;
}

// At least `count` elements at *p (their contents are lost when it grows); *p stays as it is when
// they cannot be had.
template <class T>
int grow(T** p, size_t* have, size_t count) {
    if (*have >= count) return ADMM_OK;
    T* q = nullptr;
    if (cudaMalloc((void**)&q, count * sizeof(T)) != cudaSuccess) {
        cudaGetLastError();
        return ADMM_ERR_OOM;
    }
    cudaFree(*p);
    *p = q;
    *have = count;
    return ADMM_OK;
}

// Workspace of `samples` samples of K sweeps.
int grow_batch(AdmmLearn* L, int K, int samples) {
    const size_t n = L->n, gb = nblk(n, kT), ge = std::min<size_t>(gb, kParts);
    if (int rc = grow(&L->work, &L->work_floats, samples * ((2 * K + 9) * 3 * n + n))) return rc;
    return grow(&L->dwork, &L->dwork_doubles, samples * (4 + 4 * ge + 2 * K * gb));
}

TrainMat matrix_of(const AdmmLearn* L) { return {L->start, L->col, L->val, L->diag, L->n, 3 * (size_t)L->n}; }

}  // namespace

extern "C" {

int admm_learn_create(int n, const int32_t* start, const int32_t* col, const float* val, const float* diag,
                      AdmmLearn** out) {
    if (!out || n <= 0 || !start || !diag) return ADMM_ERR_INVALID;
    *out = nullptr;
    const int nnz = start[n];
    if (nnz < 0 || (nnz > 0 && (!col || !val))) return ADMM_ERR_INVALID;
    AdmmLearn* L = new (std::nothrow) AdmmLearn;
    if (!L) return ADMM_ERR_OOM;
    L->n = n;
    L->nnz = nnz;
    int rc = ADMM_OK;
    if ((rc = lalloc(L, &L->start, n + 1)) || (rc = lalloc(L, &L->col, nnz)) || (rc = lalloc(L, &L->val, nnz)) ||
        (rc = lalloc(L, &L->diag, n)) || (rc = lalloc(L, &L->m, n)) || (rc = lalloc(L, &L->th, n)) ||
        (rc = lalloc(L, &L->gm, n)) || (rc = lalloc(L, &L->gth, n)) || (rc = lalloc(L, &L->coef, 2 * kMaxK)) ||
        (rc = grow_batch(L, kMaxK, 1))) {
        admm_learn_destroy(L);
        return rc;
    }
    if (cudaStreamCreateWithFlags(&L->st, cudaStreamNonBlocking) != cudaSuccess) {
        admm_learn_destroy(L);
        return ADMM_ERR_CUDA;
    }
    cudaMemcpy(L->start, start, sizeof(int) * (n + 1), cudaMemcpyHostToDevice);
    if (nnz) {
        cudaMemcpy(L->col, col, sizeof(int) * nnz, cudaMemcpyHostToDevice);
        cudaMemcpy(L->val, val, sizeof(float) * nnz, cudaMemcpyHostToDevice);
    }
    cudaMemcpy(L->diag, diag, sizeof(float) * n, cudaMemcpyHostToDevice);
    if (cudaGetLastError() != cudaSuccess) {
        admm_learn_destroy(L);
        return ADMM_ERR_CUDA;
    }
    *out = L;
    return ADMM_OK;
}

void admm_learn_destroy(AdmmLearn* L) {
    if (!L) return;
    if (L->st) {
        cudaStreamSynchronize(L->st);
        cudaStreamDestroy(L->st);
    }
    for (void* p : L->allocs) cudaFree(p);
    cudaFree(L->work);
    cudaFree(L->dwork);
    delete L;
}

int admm_learn_loss_grad(AdmmLearn* L, int K, const float* omega, const float* beta, const float* m, const float* theta,
                         int nsamp, const float* b, const float* xc, const float* xl, const float* xs, double* loss,
                         float* g_omega, float* g_beta, float* g_m, float* g_theta) {
    if (!L || K < 1 || K > kMaxK || !omega || !beta || !m || !theta || nsamp < 1 || !b || !xc || !xl || !xs)
        return ADMM_ERR_INVALID;
    const int n = L->n;
    const size_t N3 = 3 * (size_t)n;
    const TrainMat M = matrix_of(L);
    const int gb = nblk(n, kT), ge = std::min(gb, kParts);
    cudaStream_t st = L->st;
    // samples per batch: 2 K + 9 vectors each, and fewer where the device has no memory for them (the
    // workspace of one has been there from the start)
    const size_t per = (size_t)(2 * K + 9) * N3 + n;
    int most = (int)std::max<size_t>(1, std::min<size_t>({(size_t)nsamp, L->batch_bytes / (4 * per), 32768}));
    while (grow_batch(L, K, most) != ADMM_OK) {
        if (most == 1) return ADMM_ERR_OOM;
        most /= 2;
    }
    cudaMemcpyAsync(L->m, m, sizeof(float) * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(L->th, theta, sizeof(float) * n, cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(L->gm, 0, sizeof(float) * n, st);
    cudaMemsetAsync(L->gth, 0, sizeof(float) * n, st);
    cudaMemsetAsync(L->coef, 0, sizeof(double) * 2 * kMaxK, st);
    double total = 0.0;
    int used = 0;
    std::vector<double> hs;
    for (int s0 = 0; s0 < nsamp; s0 += most) {
        const int S = std::min(most, nsamp - s0);
        const size_t SN = S * N3, bytes = sizeof(float) * SN, off = (size_t)s0 * N3;
        float* w = L->work;
        auto take = [&](size_t cnt) {
            float* p = w;
            w += cnt;
            return p;
        };
        float *db = take(SN), *dxc = take(SN), *dxl = take(SN), *dxs = take(SN);
        float *X = take((K + 1) * SN), *Rk = take(K * SN), *ae = take(SN);
        float* g[3] = {take(SN), take(SN), take(SN)};
        float* gms = take((size_t)S * n);
        double *scal = L->dwork, *pc = scal + 4 * (size_t)S, *pK = pc + 2 * (size_t)S * ge, *pa = pK + 2 * (size_t)S * ge;
        cudaMemcpyAsync(dxc, xc + off, bytes, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(dxs, xs + off, bytes, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(dxl, xl + off, bytes, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(db, b + off, bytes, cudaMemcpyHostToDevice, st);
        // E_c = (xc - x*)^T A (xc - x*), R_c = |A (xc - x*)|^2 = |b - A xc|^2, and x_0
        k_t_error<<<dim3(ge, S), kT, 0, st>>>(M, dxc, dxs, dxl, L->th, X, ae, pc);
        for (int k = 0; k < K; k++)
            k_t_sweep<<<dim3(gb, S), kT, 0, st>>>(M, L->m, db, X + k * SN, X + (k > 0 ? k - 1 : 0) * SN, omega[k],
                                                  k > 0 ? beta[k] : 0.f, Rk + k * SN, X + (k + 1) * SN);
        k_t_error<<<dim3(ge, S), kT, 0, st>>>(M, X + K * SN, dxs, nullptr, nullptr, nullptr, ae, pK);
        k_t_scalars<<<S, kT, 0, st>>>(pc, pK, ge, scal);
        // adjoint from g_K, g_k in g[k % 3]
        k_t_seed<<<dim3(gb, S), kT, 0, st>>>(M, ae, scal, L->mu, nsamp, g[K % 3]);
        for (int k = K - 1; k >= 0; k--)
            k_t_adjoint<<<dim3(gb, S), kT, 0, st>>>(M, L->m, scal, g[(k + 1) % 3], k + 2 <= K ? g[(k + 2) % 3] : nullptr,
                                                    Rk + k * SN, X + k * SN, X + (k > 0 ? k - 1 : 0) * SN, omega[k],
                                                    k > 0 ? beta[k] : 0.f, k + 1 < K ? beta[k + 1] : 0.f, k == K - 1,
                                                    g[k % 3], gms, pa + 2 * (size_t)k * S * gb);
        k_t_collect<<<gb + 2 * K, kT, 0, st>>>(M, scal, g[0], dxc, dxl, gms, S, gb, pa, S * gb, L->gm, L->gth, L->coef);
        const size_t have = hs.size();
        hs.resize(have + 4 * (size_t)S);
        if (cudaMemcpyAsync(hs.data() + have, scal, sizeof(double) * 4 * S, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return ADMM_ERR_CUDA;
    }
    for (int s = 0; s < nsamp; s++) {
        const double Ec = hs[4 * s], Rc = hs[4 * s + 1], EK = hs[4 * s + 2], RK = hs[4 * s + 3];
        if (!(Ec > 0.0)) continue;
        used++;
        total += EK / Ec;
        if (L->mu > 0.0 && Rc > 0.0) total += L->mu * RK / Rc;
    }
    double coef[2 * kMaxK];
    if (cudaMemcpyAsync(coef, L->coef, sizeof(double) * 2 * K, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        (g_m && cudaMemcpyAsync(g_m, L->gm, sizeof(float) * n, cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        (g_theta && cudaMemcpyAsync(g_theta, L->gth, sizeof(float) * n, cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return ADMM_ERR_CUDA;
    if (loss) *loss = used ? total / nsamp : 0.0;
    if (g_omega)
        for (int k = 0; k < K; k++) g_omega[k] = (float)coef[2 * k];
    if (g_beta)
        for (int k = 0; k < K; k++) g_beta[k] = k > 0 ? (float)coef[2 * k + 1] : 0.f;
    return ADMM_OK;
}

int admm_learn_set_batch_bytes(AdmmLearn* L, size_t bytes) {
    if (!L) return ADMM_ERR_INVALID;
    L->batch_bytes = bytes;
    return ADMM_OK;
}

int admm_learn_set_residual_weight(AdmmLearn* L, double mu) {
    if (!L || !(mu >= 0.0) || !std::isfinite(mu)) return ADMM_ERR_INVALID;
    L->mu = mu;
    return ADMM_OK;
}

int admm_learn_solve(AdmmLearn* L, const float* b, float* x, double rel_tol, int max_iter, int* iters) {
    if (!L || !b || !x || max_iter < 0) return ADMM_ERR_INVALID;
    const int n = L->n;
    const size_t N3 = 3 * (size_t)n;
    const TrainMat M = matrix_of(L);
    const int ge = std::min(nblk(n, kT), kCgParts);
    cudaStream_t st = L->st;
    if (int rc = grow(&L->work, &L->work_floats, 7 * N3)) return rc;
    constexpr size_t kState = sizeof(CgState) / sizeof(double);
    static_assert(sizeof(CgState) % sizeof(double) == 0, "the states lie in the double workspace");
    if (int rc = grow(&L->dwork, &L->dwork_doubles, 2 * kState + 2 * (size_t)ge)) return rc;
    float *db = L->work, *dx = db + N3, *r = dx + N3, *z = r + N3, *q = z + N3, *p[2] = {q + N3, q + 2 * N3};
    CgState* state[2] = {(CgState*)L->dwork, (CgState*)(L->dwork + kState)};
    double* part[2] = {L->dwork + 2 * kState, L->dwork + 2 * kState + ge};
    cudaMemsetAsync(state[0], 0, sizeof(CgState), st);
    cudaMemcpyAsync(db, b, sizeof(float) * N3, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dx, x, sizeof(float) * N3, cudaMemcpyHostToDevice, st);
    k_cg_init<<<ge, kT, 0, st>>>(M, db, dx, r, z, part[0]);
    CgState now = {};
    const bool fused = n <= kFusedRows;
    for (int it = 0; it < max_iter && !now.done;) {
        for (const int end = std::min(max_iter, it + kCgChunk); it < end; it++) {
            float* pn = p[fused ? (it + 1) & 1 : 0];
            if (fused) {
                admm::launch_k(k_cg_q<true>, ge, kT, 0, st, true, M, z, p[it & 1], ge, part[0], rel_tol * rel_tol, it,
                               state[0], state[1], pn, q, part[1]);
            } else {
                admm::launch_k(k_cg_p, ge, kT, 0, st, true, M, z, pn, ge, part[0], rel_tol * rel_tol, it, state[0],
                               state[1]);
                admm::launch_k(k_cg_q<false>, ge, kT, 0, st, true, M, pn, nullptr, ge, part[0], rel_tol * rel_tol, it,
                               state[0], state[1], nullptr, q, part[1]);
            }
            admm::launch_k(k_cg_xr, ge, kT, 0, st, true, M, pn, q, ge, part[1], state[1], state[0], dx, r, z, part[0]);
        }
        if (cudaMemcpyAsync(&now, state[0], sizeof(now), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return ADMM_ERR_CUDA;
    }
    if (cudaMemcpyAsync(x, dx, sizeof(float) * N3, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return ADMM_ERR_CUDA;
    if (iters) *iters = now.iters;
    return cudaGetLastError() == cudaSuccess ? ADMM_OK : ADMM_ERR_CUDA;
}

}  // extern "C"
