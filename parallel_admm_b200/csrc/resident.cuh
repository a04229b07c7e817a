// resident.cuh -- the global step with the matrix and the iterate resident in shared memory
// (plan: resident.hpp).  One thread-block cluster per group of connected components runs all
// sweeps of a global step in one launch: a launch per sweep moves the whole matrix from L2 or
// HBM each time and costs a kernel boundary, this kernel reads it once.  Same row sums as
// k_jacobi / k_lsweep / k_ljudge, so the iterates are the same bits.
#pragma once
#include "kernels.cuh"
#include "learn.cuh"
#include "resident.hpp"

namespace admm {

struct ResidentDev {
    const ResidentCta* cta = nullptr;    // [groups * cluster]
    const unsigned char* blob = nullptr;
    int cluster = 0, groups = 0, tp = 0, q = 0, threads = 0;
    int max_own = 0, max_local = 0;      // max_own rounded up to a multiple of 4
};

ADMM_DEV uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

ADMM_DEV uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Address of the same shared-memory location in CTA `rank` of the cluster, and a 16-byte store there.
ADMM_DEV uint32_t cluster_map(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
ADMM_DEV void cluster_store(uint32_t addr, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z),
                 "f"(v.w)
                 : "memory");
}

// Every thread of every CTA of the cluster; what was written before it (in shared memory of any
// CTA of the cluster, and in global memory) is visible after it.  A cluster of one: the block.
template <bool CLUSTER>
ADMM_DEV void cluster_sync() {
    if (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// The CTA's shared memory: iterate a, iterate b, own-row arrays, blob.
struct ResidentSmem {
    float4 *xa, *xb, *own;
    unsigned char* blob;
};

ADMM_DEV ResidentSmem resident_smem_of(const ResidentDev& p, unsigned char* base, int own_arrays) {
    ResidentSmem m;
    m.xa = (float4*)base;
    m.xb = m.xa + p.max_local;
    m.own = m.xb + p.max_local;
    m.blob = (unsigned char*)(m.own + own_arrays * p.max_own);
    return m;
}

// The sections of the blob in shared memory.
struct ResidentView {
    const float2* val;       // + lane
    const uint32_t* col;     // + lane
    const int* sptr;
    const uint16_t* pptr;
    const uint32_t* push;
    const int* grow;
    const float* diag;
    int own, halo, slices;
};

ADMM_DEV ResidentView resident_view(const ResidentCta& d, const unsigned char* blob) {
    const int lane = threadIdx.x & 31;
    ResidentView v;
    v.val = (const float2*)(blob + d.off_val) + lane;
    v.col = (const uint32_t*)(blob + d.off_col) + lane;
    v.sptr = (const int*)(blob + d.off_sptr);
    v.pptr = (const uint16_t*)(blob + d.off_pptr);
    v.push = (const uint32_t*)(blob + d.off_push);
    v.grow = (const int*)(blob + d.off_grow);
    v.diag = (const float*)blob;
    v.own = d.own;
    v.halo = d.halo;
    v.slices = d.slices;
    return v;
}

// The blob into shared memory (constant data: before the dependency wait); complete after a
// block barrier.
ADMM_DEV void resident_load(const ResidentDev& p, const ResidentCta& d, unsigned char* dst) {
    const uint32_t to = smem_addr(dst);
    const unsigned char* from = p.blob + d.blob;
    for (int k = 16 * threadIdx.x; k < d.bytes; k += 16 * blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + k), "l"(from + k) : "memory");
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// The partial sums of a row combined: over the thread's own, then over the row's threads.
template <int Q, int TP>
ADMM_DEV float4 resident_combine(float (&ax)[Q], float (&ay)[Q], float (&az)[Q]) {
#pragma unroll
    for (int o = 1; o < Q; o <<= 1)
#pragma unroll
        for (int q = 0; q < Q; q += 2 * o) {
            ax[q] += ax[q + o];
            ay[q] += ay[q + o];
            az[q] += az[q + o];
        }
#pragma unroll
    for (int o = 1; o < TP; o <<= 1) {
        ax[0] += __shfl_xor_sync(0xffffffffu, ax[0], o);
        ay[0] += __shfl_xor_sync(0xffffffffu, ay[0], o);
        az[0] += __shfl_xor_sync(0xffffffffu, az[0], o);
    }
    return f4(ax[0], ay[0], az[0]);
}

// Pair steps [k, e) of a row, from shared memory, onto its partial sums (k a multiple of a round
// of the partial sums).
template <int Q>
ADMM_DEV void resident_steps(const float2* __restrict__ val, const uint32_t* __restrict__ col,
                             const float4* __restrict__ x, int k, int e, float (&ax)[Q], float (&ay)[Q], float (&az)[Q]) {
    constexpr int U = Q >= 4 ? Q / 2 : 1;  // pair steps per round
#pragma unroll 2
    for (; k < e; k += U) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float2 v = val[32 * (k + u)];
            const uint32_t c = col[32 * (k + u)];
            const float4 p0 = x[c & 0xffffu], p1 = x[c >> 16];
            const int q0 = (2 * u) % Q, q1 = (2 * u + 1) % Q;
            ax[q0] = fmaf(v.x, p0.x, ax[q0]);
            ay[q0] = fmaf(v.x, p0.y, ay[q0]);
            az[q0] = fmaf(v.x, p0.z, az[q0]);
            ax[q1] = fmaf(v.y, p1.x, ax[q1]);
            ay[q1] = fmaf(v.y, p1.y, ay[q1]);
            az[q1] = fmaf(v.y, p1.z, az[q1]);
        }
    }
}

// sum_k a_ik x_k of the thread's row over the off-diagonal entries, in every thread of the row.
template <int Q, int TP>
ADMM_DEV float4 resident_row(const ResidentView& w, const float4* __restrict__ x, int slice) {
    float ax[Q], ay[Q], az[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) ax[q] = ay[q] = az[q] = 0.f;
    resident_steps<Q>(w.val, w.col, x, w.sptr[slice], w.sptr[slice + 1], ax, ay, az);
    return resident_combine<Q, TP>(ax, ay, az);
}

// The matrix entries of a thread's row, kept in registers over the sweeps: up to NP pair steps
// (rows of 20 entries), the rest stays in shared memory.  The steps past the row's end are 0 times
// the row's own value, like the plan's padding: a CTA holds rows of several bodies, and 0 times
// another body's value is NaN once that body has diverged.
constexpr int kResidentRows = 2;  // rows per thread in registers

template <int Q, int TP>
struct ResidentRow {
    static constexpr int T = Q * TP;
    static constexpr int NP = ((20 + T - 1) / T * Q + 1) / 2;
    static constexpr int CH = Q >= 4 ? 2 : (NP + 2) / 3;  // pair steps whose gathers are in flight together
    float2 v[NP];
    uint32_t c[NP];
    int b, n;

    ADMM_DEV void load(const ResidentView& w, int sl) {
        const int r = sl * (32 / TP) + (threadIdx.x & 31) / TP;
        const uint32_t self = r < w.own ? (uint32_t)r | (uint32_t)r << 16 : 0u;
        b = n = 0;
#pragma unroll
        for (int u = 0; u < NP; u++) {
            v[u] = make_float2(0.f, 0.f);
            c[u] = self;
        }
        if (sl >= w.slices) return;
        b = w.sptr[sl];
        n = w.sptr[sl + 1] - b;
#pragma unroll
        for (int u = 0; u < NP; u++)
            if (u < n) {
                v[u] = w.val[32 * (b + u)];
                c[u] = w.col[32 * (b + u)];
            }
    }

    ADMM_DEV float4 sum(const ResidentView& w, const float4* __restrict__ x) const {
        float ax[Q], ay[Q], az[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) ax[q] = ay[q] = az[q] = 0.f;
#pragma unroll
        for (int u0 = 0; u0 < NP; u0 += CH) {
            if (u0 < n) {  // the same in the whole warp
                float4 p[2 * CH];
#pragma unroll
                for (int u = 0; u < CH; u++)
                    if (u0 + u < NP) {
                        p[2 * u] = x[c[u0 + u] & 0xffffu];
                        p[2 * u + 1] = x[c[u0 + u] >> 16];
                    }
#pragma unroll
                for (int u = 0; u < CH; u++)
                    if (u0 + u < NP) {
                        const int q0 = (2 * (u0 + u)) % Q, q1 = (2 * (u0 + u) + 1) % Q;
                        const float2 a = v[u0 + u];
                        ax[q0] = fmaf(a.x, p[2 * u].x, ax[q0]);
                        ay[q0] = fmaf(a.x, p[2 * u].y, ay[q0]);
                        az[q0] = fmaf(a.x, p[2 * u].z, az[q0]);
                        ax[q1] = fmaf(a.y, p[2 * u + 1].x, ax[q1]);
                        ay[q1] = fmaf(a.y, p[2 * u + 1].y, ay[q1]);
                        az[q1] = fmaf(a.y, p[2 * u + 1].z, az[q1]);
                    }
            }
        }
        if (n > NP) resident_steps<Q>(w.val, w.col, x, b + NP, b + n, ax, ay, az);
        return resident_combine<Q, TP>(ax, ay, az);
    }
};

// The new value of own row r into slot r here and into its halo slots in the cluster (buffer
// `dst`, the same place in every CTA); thread j of the row's TP writes every TP-th halo slot.
template <int TP>
ADMM_DEV void resident_put(const ResidentView& w, float4* dst, int r, int j, int pbeg, int pend, float4 v) {
    if (j == 0) dst[r] = v;
    const uint32_t base = smem_addr(dst);
    for (int k = pbeg + j; k < pend; k += TP) {
        const uint32_t t = w.push[k];
        cluster_store(cluster_map(base + 16u * (t & 0xffffu), t >> 16), v);
    }
}

// `sweeps` >= 1 Jacobi sweeps (JacobiFunctor, jacobi_solver.cu:52-98) on b from x into x.
template <int Q, int TP, bool CLUSTER>
__global__ void __launch_bounds__(kResidentThreads, 1) k_resident_jacobi(DevScene s, ResidentDev p, int sweeps) {
    extern __shared__ __align__(128) unsigned char rsm[];
    ADMM_PDL_TRIGGER();
    const ResidentCta d = p.cta[blockIdx.x];
    const ResidentSmem m = resident_smem_of(p, rsm, 1);
    resident_load(p, d, m.blob);
    __syncthreads();
    const ResidentView w = resident_view(d, m.blob);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, j = lane % TP;
    ResidentRow<Q, TP> row[kResidentRows];
#pragma unroll
    for (int i = 0; i < kResidentRows; i++) row[i].load(w, warp + i * nw);
    ADMM_PDL_WAIT();
    for (int k = threadIdx.x; k < w.own + w.halo; k += blockDim.x) m.xa[k] = s.x[w.grow[k]];
    for (int k = threadIdx.x; k < w.own; k += blockDim.x) {
        float4 b = s.b[w.grow[k]];
        b.w = w.diag[k];
        m.own[k] = b;
    }
    // the cluster's CTAs have all started before anyone writes into another's shared memory
    cluster_sync<CLUSTER>();
    float4 breg[kResidentRows];
    int preg[kResidentRows];
#pragma unroll
    for (int i = 0; i < kResidentRows; i++) {
        const int r = (warp + i * nw) * (32 / TP) + lane / TP;
        breg[i] = r < w.own ? m.own[r] : f4(0.f, 0.f, 0.f, 1.f);
        preg[i] = r < w.own ? w.pptr[r] | w.pptr[r + 1] << 16 : 0;
    }
    for (int k = 0; k < sweeps; k++) {
        const float4* src = k & 1 ? m.xb : m.xa;
        float4* dst = k & 1 ? m.xa : m.xb;
        const bool last = k == sweeps - 1;
        auto finish = [&](int sl, float4 acc, float4 b, int push) {
            const int r = sl * (32 / TP) + lane / TP;
            if (r < w.own) {
                const float4 v = f4((b.x - acc.x) / b.w, (b.y - acc.y) / b.w, (b.z - acc.z) / b.w);
                if (!last) resident_put<TP>(w, dst, r, j, push & 0xffff, (int)((unsigned)push >> 16), v);
                else if (j == 0) s.x[w.grow[r]] = v;
            }
        };
#pragma unroll
        for (int i = 0; i < kResidentRows; i++)
            if (warp + i * nw < w.slices) finish(warp + i * nw, row[i].sum(w, src), breg[i], preg[i]);
        for (int sl = warp + kResidentRows * nw; sl < w.slices; sl += nw) {
            const int r = min(sl * (32 / TP) + lane / TP, w.own - 1);
            finish(sl, resident_row<Q, TP>(w, src, sl), m.own[r], w.pptr[r] | w.pptr[r + 1] << 16);
        }
        if (!last) cluster_sync<CLUSTER>();
    }
}

// The learned global step after k_rhs_learn: K second-order sweeps from x0 (the warm start)
// into x, with the sums of the first sweep (k_lsweep<T, true>) and of the judge's pass
// (k_ljudge) as one partial per CTA.
struct LearnCoef {
    float omega[kLearnMaxSweeps], beta[kLearnMaxSweeps];
};

template <int Q, int TP, bool CLUSTER>
__global__ void __launch_bounds__(kResidentThreads, 1)
    k_resident_learned(DevScene s, ResidentDev p, LearnDev L, const float4* x0, LearnCoef coef, int sweeps,
                       int extrap) {
    extern __shared__ __align__(128) unsigned char rsm[];
    __shared__ double sh[32];
    ADMM_PDL_TRIGGER();
    const ResidentCta d = p.cta[blockIdx.x];
    const ResidentSmem m = resident_smem_of(p, rsm, 2);
    resident_load(p, d, m.blob);
    __syncthreads();
    const ResidentView w = resident_view(d, m.blob);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, j = lane % TP;
    ResidentRow<Q, TP> row[kResidentRows];
#pragma unroll
    for (int i = 0; i < kResidentRows; i++) row[i].load(w, warp + i * nw);
    float4* prev = m.own + p.max_own;  // x_{k-1} of the own rows, w = m_i
    for (int k = threadIdx.x; k < w.own; k += blockDim.x) prev[k].w = __ldg(&L.minv[w.grow[k]]);
    ADMM_PDL_WAIT();
    for (int k = threadIdx.x; k < w.own + w.halo; k += blockDim.x) m.xa[k] = x0[w.grow[k]];
    for (int k = threadIdx.x; k < w.own; k += blockDim.x) {
        float4 b = s.b[w.grow[k]];
        b.w = w.diag[k];
        m.own[k] = b;
    }
    cluster_sync<CLUSTER>();
    double rr = 0.0, bb = 0.0, rc = 0.0, rk = 0.0;
    for (int k = 0; k <= sweeps; k++) {  // k == sweeps: the judge's pass
        const float4* src = k & 1 ? m.xb : m.xa;
        float4* dst = k & 1 ? m.xa : m.xb;
        const float omega = k < sweeps ? coef.omega[k] : 0.f, beta = k < sweeps ? coef.beta[k] : 0.f;
        auto finish = [&](int sl, float4 acc) {
            const int r = sl * (32 / TP) + lane / TP;
            const bool in = r < w.own;
            float4 xi = f4(0.f, 0.f, 0.f), pm = xi;
            if (in) {
                const float4 b = m.own[r];
                xi = src[r];
                pm = prev[r];
                const float4 a = f4(fmaf(b.w, xi.x, acc.x), fmaf(b.w, xi.y, acc.y), fmaf(b.w, xi.z, acc.z));
                const float rx = b.x - a.x, ry = b.y - a.y, rz = b.z - a.z;
                const double r2 = (double)rx * rx + (double)ry * ry + (double)rz * rz;
                if (k == sweeps) {
                    if (j == 0) {
                        L.ax[w.grow[r]] = a;
                        rk += r2;
                    }
                } else {
                    const float4 xp = k == 0 ? xi : pm;
                    const float ox = omega * pm.w;
                    const float4 v = f4(fmaf(ox, rx, fmaf(beta, xi.x - xp.x, xi.x)),
                                        fmaf(ox, ry, fmaf(beta, xi.y - xp.y, xi.y)),
                                        fmaf(ox, rz, fmaf(beta, xi.z - xp.z, xi.z)));
                    resident_put<TP>(w, dst, r, j, w.pptr[r], w.pptr[r + 1], v);
                    if (j == 0 && k == sweeps - 1) s.x[w.grow[r]] = v;
                    if (j == 0 && k == 0) {
                        rr += r2;
                        bb += (double)b.x * b.x + (double)b.y * b.y + (double)b.z * b.z;
                        if (extrap) {
                            const float4 ai = L.ax[w.grow[r]];
                            const float cx = b.x - ai.x, cy = b.y - ai.y, cz = b.z - ai.z;
                            rc += (double)cx * cx + (double)cy * cy + (double)cz * cz;
                        }
                    }
                }
            }
            __syncwarp();  // every thread of the row has read prev
            if (in && j == 0) prev[r] = make_float4(xi.x, xi.y, xi.z, pm.w);
        };
#pragma unroll
        for (int i = 0; i < kResidentRows; i++)
            if (warp + i * nw < w.slices) finish(warp + i * nw, row[i].sum(w, src));
        for (int sl = warp + kResidentRows * nw; sl < w.slices; sl += nw)
            finish(sl, resident_row<Q, TP>(w, src, sl));
        if (k < sweeps) cluster_sync<CLUSTER>();
    }
    rr = block_sum(rr, sh);
    bb = block_sum(bb, sh);
    rc = block_sum(rc, sh);
    rk = block_sum(rk, sh);
    if (threadIdx.x == 0) {
        L.part[blockIdx.x] = rr;
        L.part[L.blocks + blockIdx.x] = rk;
        L.part[2 * L.blocks + blockIdx.x] = bb;
        L.part_c[blockIdx.x] = rc;
    }
}

// The PCG global step (k_pcg_init / k_pcg_spmv / k_pcg_update, same operations per row) of a
// scene that fits one cluster, all iterations in one launch: two cluster barriers per iteration,
// one after the new u is in its halo slots, one after every CTA has the others' partial sums of
// (r, u) and (A u, u).  Those FP64 sums are added in another order than the per-iteration
// kernels' block partials.
ADMM_DEV void cluster_store(uint32_t addr, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}

// M^-1 r of own row i with diagonal r.w (or with the caller's 3x3 blocks).
ADMM_DEV float4 resident_precond(const DevScene& s, const PcgDev& g, int i, float4 r) {
    if (g.block) return pcg_precond(s, g, i, r);
    return f4(r.x / r.w, r.y / r.w, r.z / r.w);
}

constexpr int kResidentPcgArrays = 5;  // own-row arrays: r (w = a_ii), A u, p, s, x

template <int Q, int TP, bool CLUSTER>
__global__ void __launch_bounds__(kResidentThreads, 1) k_resident_pcg(DevScene s, ResidentDev p, PcgDev g, int iters) {
    extern __shared__ __align__(128) unsigned char rsm[];
    __shared__ double2 red[2][16];   // the cluster's partials, by parity of the iteration
    __shared__ double2 wsum[kResidentThreads / 32];
    ADMM_PDL_TRIGGER();
    const ResidentCta d = p.cta[blockIdx.x];
    const ResidentSmem m = resident_smem_of(p, rsm, kResidentPcgArrays);
    resident_load(p, d, m.blob);
    __syncthreads();
    const ResidentView w = resident_view(d, m.blob);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, j = lane % TP;
    const uint32_t rank = CLUSTER ? cluster_rank() : 0u;
    float4 *R = m.own, *W = R + p.max_own, *P = W + p.max_own, *S = P + p.max_own, *X = S + p.max_own;
    ResidentRow<Q, TP> row[kResidentRows];
#pragma unroll
    for (int i = 0; i < kResidentRows; i++) row[i].load(w, warp + i * nw);
    ADMM_PDL_WAIT();
    for (int k = threadIdx.x; k < w.own + w.halo; k += blockDim.x) m.xb[k] = s.x[w.grow[k]];
    for (int k = threadIdx.x; k < w.own; k += blockDim.x) {
        float4 b = s.b[w.grow[k]];
        b.w = w.diag[k];
        R[k] = b;
        P[k] = S[k] = f4(0.f, 0.f, 0.f);
    }
    cluster_sync<CLUSTER>();
    // A v of every own row: f(row, sum over the off-diagonal entries) in the row's first thread
    auto spmv = [&](const float4* v, auto f) {
#pragma unroll
        for (int i = 0; i < kResidentRows; i++)
            if (warp + i * nw < w.slices) {
                const float4 acc = row[i].sum(w, v);
                const int r = (warp + i * nw) * (32 / TP) + lane / TP;
                if (r < w.own && j == 0) f(r, acc);
            }
        for (int sl = warp + kResidentRows * nw; sl < w.slices; sl += nw) {
            const float4 acc = resident_row<Q, TP>(w, v, sl);
            const int r = sl * (32 / TP) + lane / TP;
            if (r < w.own && j == 0) f(r, acc);
        }
    };
    float4* u = m.xa;
    spmv(m.xb, [&](int r, float4 acc) {
        const float4 b = R[r], xi = m.xb[r];
        const float4 rr = make_float4(b.x - fmaf(b.w, xi.x, acc.x), b.y - fmaf(b.w, xi.y, acc.y),
                                      b.z - fmaf(b.w, xi.z, acc.z), b.w);
        R[r] = rr;
        X[r] = xi;
        resident_put<1>(w, u, r, 0, w.pptr[r], w.pptr[r + 1], resident_precond(s, g, w.grow[r], rr));
    });
    cluster_sync<CLUSTER>();
    double gamma0 = 0.0, alpha0 = 0.0;  // of the previous iteration
    for (int it = 0; it < iters; it++) {
        double2 part = make_double2(0.0, 0.0);
        spmv(u, [&](int r, float4 acc) {
            const float4 rr = R[r], ui = u[r];
            const float4 au = f4(fmaf(rr.w, ui.x, acc.x), fmaf(rr.w, ui.y, acc.y), fmaf(rr.w, ui.z, acc.z));
            W[r] = au;
            part.x += dot3d(rr, ui);
            part.y += dot3d(au, ui);
        });
        part.x = warp_sum(part.x);
        part.y = warp_sum(part.y);
        if (lane == 0) wsum[warp] = part;
        __syncthreads();
        if (warp == 0) {
            part = lane < nw ? wsum[lane] : make_double2(0.0, 0.0);
            part.x = warp_sum(part.x);
            part.y = warp_sum(part.y);
            double2* slot = &red[it & 1][rank];
            if (CLUSTER) {
                if (lane < p.cluster) cluster_store(cluster_map(smem_addr(slot), lane), part);
            } else if (lane == 0) {
                *slot = part;
            }
        }
        cluster_sync<CLUSTER>();
        double2 sum = lane < p.cluster ? red[it & 1][lane] : make_double2(0.0, 0.0);
        const double gamma = warp_sum(sum.x), delta = warp_sum(sum.y);
        double alpha, beta;
        if (it == 0) {
            beta = 0.0;
            alpha = delta != 0.0 ? gamma / delta : 0.0;
        } else {
            beta = gamma0 != 0.0 ? gamma / gamma0 : 0.0;
            const double den = delta - beta * gamma / (alpha0 != 0.0 ? alpha0 : 1.0);
            alpha = den != 0.0 ? gamma / den : 0.0;
        }
        gamma0 = gamma;
        alpha0 = alpha;
        const float a = (float)alpha, bt = (float)beta;
        for (int r = threadIdx.x; r < w.own; r += blockDim.x) {
            const float4 ui = u[r], au = W[r];
            float4 pv = P[r], sv = S[r], x = X[r], rr = R[r];
            pv = f4(fmaf(bt, pv.x, ui.x), fmaf(bt, pv.y, ui.y), fmaf(bt, pv.z, ui.z));
            sv = f4(fmaf(bt, sv.x, au.x), fmaf(bt, sv.y, au.y), fmaf(bt, sv.z, au.z));
            x = f4(fmaf(a, pv.x, x.x), fmaf(a, pv.y, x.y), fmaf(a, pv.z, x.z));
            rr = make_float4(fmaf(-a, sv.x, rr.x), fmaf(-a, sv.y, rr.y), fmaf(-a, sv.z, rr.z), rr.w);
            P[r] = pv;
            S[r] = sv;
            X[r] = x;
            R[r] = rr;
            if (it + 1 < iters)
                resident_put<1>(w, u, r, 0, w.pptr[r], w.pptr[r + 1], resident_precond(s, g, w.grow[r], rr));
            else
                s.x[w.grow[r]] = x;
        }
        if (it + 1 < iters) cluster_sync<CLUSTER>();
    }
}

}  // namespace admm
