// noalloc.cu -- a Jacobi solve of the global system that allocates nothing.
//
// The handle API (admm_b200_create) allocates every device buffer it needs up
// front.  Some callers cannot do that: a host application whose device memory is
// entirely owned by its own pool allocator and that forbids any other cudaMalloc,
// a real-time loop that cannot afford cudaMalloc's latency and implicit device
// synchronisation, or a plug-in host that only hands out buffers it allocated
// itself.  admm_b200_jacobi_noalloc serves them: the caller passes the matrix,
// the right-hand side and the input/output positions in its own device memory,
// and the two ping-pong buffers the sweeps need live in a file-scope
// __device__ array of fixed size, g_jacobi_scratch, reserved in every GPU that
// loads the library until the process exits.
//
// Limits and contract:
//  * at most kNoAllocMaxRows rows (262144, i.e. 2 x 262144 x 3 floats = 6 MiB of
//    static device memory); larger systems are rejected with ADMM_ERR_INVALID;
//  * the scratch is shared by every call in the process: calls whose work
//    overlaps on the GPU (different streams, or different host threads on one
//    device) race on it and must be ordered by the caller;
//  * nothing in the scratch needs to start at zero: every sweep overwrites all
//    rows it later reads, so a call never sees the previous call's contents;
//  * the device address of the scratch is looked up (cudaGetSymbolAddress) in the
//    context that is current on the calling thread, on every call made outside
//    stream capture, and remembered per context; a call made while its stream is
//    being captured uses the address remembered for the current context, so a call
//    in that context must have run outside capture first (else ADMM_ERR_STATE).
//    Keying by context keeps the address right for callers that run in their own
//    driver-API contexts and across a cudaDeviceReset;
//  * an error already pending on the calling thread (from the caller's own work)
//    is left untouched and the call returns ADMM_ERR_CUDA without launching.
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>
#include <vector>

#include "admm_b200.h"
#include "common.cuh"

namespace {

constexpr int kNoAllocMaxRows = 262144;
// Two ping-pong buffers of row-major n x 3 floats.
static __device__ __align__(256) float g_jacobi_scratch[2][kNoAllocMaxRows * 3];

// Address of g_jacobi_scratch per CUDA context (CUcontext as an opaque pointer).
struct ScratchEntry {
    void* ctx;
    float* ptr;
};
std::mutex g_mu;
std::vector<ScratchEntry> g_scratch;

typedef int (*CtxGetCurrentFn)(void**);

// The context current on this thread (the runtime's primary context unless the
// caller made its own current), through the driver's cuCtxGetCurrent.
void* current_context() {
    static CtxGetCurrentFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<CtxGetCurrentFn>(f);
    });
    void* ctx = nullptr;
    if (!fn || fn(&ctx) != 0) return nullptr;
    return ctx;
}

// One Jacobi sweep on CSR (off-diagonal part, JacobiFunctor of the reference's
// jacobi_solver.cu:52-98): dst_i = (b_i - sum_{j != i} a_ij src_j) / a_ii,
// row-major n x 3 vectors.  Bound by the chain of dependent loads of a row, not by bytes: four (or
// two) lanes share a row, its first kPre entries per lane are loaded before the dependency wait (the
// sweeps after a call's first one launch while the sweep before them drains; the first one
// starts after everything before it, so the matrix and b are complete by then).  src and dst are
// not __restrict__: the sweep before still writes src when this one starts, so src must not be
// read through the read-only path, nor before the wait.  28 k rows of 11
// entries, 20 sweeps: 157 us with a thread per row.
template <int kRowLanes, int kPre>  // lanes per row, entries per lane before the wait
__global__ void __launch_bounds__(128) k_jacobi_csr(int n, const int32_t* __restrict__ start,
                                                    const int32_t* __restrict__ cols, const float* __restrict__ vals,
                                                    const float* __restrict__ diag, const float* __restrict__ b,
                                                    const float* src, float* dst) {
    ADMM_PDL_TRIGGER();
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / kRowLanes, sub = t % kRowLanes;
    const bool own = i < n;
    const int k0 = own ? start[i] + sub : 0, e = own ? start[i + 1] : 0;
    int c[kPre];
    float a[kPre];
#pragma unroll
    for (int j = 0; j < kPre; j++) {
        const int k = k0 + j * kRowLanes;
        c[j] = k < e ? cols[k] : 0;
        a[j] = k < e ? vals[k] : 0.f;
    }
    const float d = own ? diag[i] : 1.f;
    const float b0 = own ? b[3 * (size_t)i] : 0.f, b1 = own ? b[3 * (size_t)i + 1] : 0.f,
                b2 = own ? b[3 * (size_t)i + 2] : 0.f;
    ADMM_PDL_WAIT();
    float ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll
    for (int j = 0; j < kPre; j++)
        if (k0 + j * kRowLanes < e) {
            const float* q = src + 3 * (size_t)c[j];
            ax = fmaf(a[j], q[0], ax);
            ay = fmaf(a[j], q[1], ay);
            az = fmaf(a[j], q[2], az);
        }
#pragma unroll 4
    for (int k = k0 + kPre * kRowLanes; k < e; k += kRowLanes) {
        const float* q = src + 3 * (size_t)cols[k];
        const float w = vals[k];
        ax = fmaf(w, q[0], ax);
        ay = fmaf(w, q[1], ay);
        az = fmaf(w, q[2], az);
    }
#pragma unroll
    for (int o = 1; o < kRowLanes; o <<= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
        az += __shfl_xor_sync(0xffffffffu, az, o);
    }
    if (!own || sub != 0) return;
    dst[3 * (size_t)i] = (b0 - ax) / d;
    dst[3 * (size_t)i + 1] = (b1 - ay) / d;
    dst[3 * (size_t)i + 2] = (b2 - az) / d;
}

// More rows than two lanes each fill the device with at once (148 SMs of 2048 threads) have two: there
// the rounds of blocks count, and short rows waste four lanes.  262144 rows of 2 / 14 / 40 entries, 20
// sweeps: 117 / 158 / 548 us with two lanes, 195 / 207 / 404 with four, 124 / 215 / 942 with one.
constexpr int kFourLaneRows = 148 * 2048 / 2;

// Device address of g_jacobi_scratch in the current context: looked up again on
// every call outside capture (cheap), taken from the per-context record during
// capture.
int scratch_address(cudaStream_t st, float** out) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) return ADMM_ERR_CUDA;  // also makes a context current
    void* ctx = current_context();
    if (!ctx) {
        fprintf(stderr, "admm_b200_jacobi_noalloc: no current CUDA context\n");
        return ADMM_ERR_NO_DEVICE;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    ScratchEntry* e = nullptr;
    for (auto& x : g_scratch)
        if (x.ctx == ctx) e = &x;
    if (cs != cudaStreamCaptureStatusNone) {
        if (!e) {
            fprintf(stderr, "admm_b200_jacobi_noalloc: first call in this context made during stream capture; "
                            "call it once outside capture first\n");
            return ADMM_ERR_STATE;
        }
        *out = e->ptr;
        return ADMM_OK;
    }
    void* p = nullptr;
    const cudaError_t err = cudaGetSymbolAddress(&p, g_jacobi_scratch);
    if (err != cudaSuccess) {
        fprintf(stderr, "admm_b200_jacobi_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(err));
        return ADMM_ERR_CUDA;
    }
    if (e)
        e->ptr = static_cast<float*>(p);
    else
        g_scratch.push_back({ctx, static_cast<float*>(p)});
    *out = static_cast<float*>(p);
    return ADMM_OK;
}

}  // namespace

extern "C" int admm_b200_jacobi_noalloc(int n, const int32_t* row_start, const int32_t* cols, const float* vals,
                                        const float* diag, const float* b, const float* x_in, float* x_out, int sweeps,
                                        void* stream) {
    if (n <= 0 || n > kNoAllocMaxRows) {
        fprintf(stderr, "admm_b200_jacobi_noalloc: n = %d rows is outside 1..%d (the static scratch holds %d rows)\n",
                n, kNoAllocMaxRows, kNoAllocMaxRows);
        return ADMM_ERR_INVALID;
    }
    if (sweeps < 0 || !row_start || !cols || !vals || !diag || !b || !x_in || !x_out) {
        fprintf(stderr, "admm_b200_jacobi_noalloc: null pointer or negative sweep count\n");
        return ADMM_ERR_INVALID;
    }
    if (cudaPeekAtLastError() != cudaSuccess) {
        fprintf(stderr, "admm_b200_jacobi_noalloc: a CUDA error is already pending on this thread (%s); "
                        "nothing launched\n", cudaGetErrorString(cudaPeekAtLastError()));
        return ADMM_ERR_CUDA;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* scratch = nullptr;
    const int rc = scratch_address(st, &scratch);
    if (rc != ADMM_OK) return rc;
    const size_t bytes = sizeof(float) * 3 * (size_t)n;
    if (sweeps == 0) {
        if (x_out != x_in && cudaMemcpyAsync(x_out, x_in, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return ADMM_ERR_CUDA;
        return ADMM_OK;
    }
    float* buf[2] = {scratch, scratch + (size_t)kNoAllocMaxRows * 3};
    const int lanes = n > kFourLaneRows ? 2 : 4;
    const int threads = 128, blocks = (n * lanes + threads - 1) / threads;
    for (int k = 0; k < sweeps; k++) {
        const float* src = k == 0 ? x_in : buf[(k - 1) & 1];
        // the last sweep writes x_out directly unless x_out is also its source
        float* dst = (k == sweeps - 1 && src != x_out) ? x_out : buf[k & 1];
        if (admm::launch_k(lanes == 2 ? k_jacobi_csr<2, 6> : k_jacobi_csr<4, 4>, dim3(blocks), dim3(threads), 0, st, k > 0,
                           n, row_start, cols, vals, diag, b, src, dst) != cudaSuccess)
            return ADMM_ERR_CUDA;
        if (k == sweeps - 1 && dst != x_out &&
            cudaMemcpyAsync(x_out, dst, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return ADMM_ERR_CUDA;
    }
    return ADMM_OK;
}
