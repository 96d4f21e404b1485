// PageRank on an inbound CSR that the caller already holds in device memory,
// without allocating anything: egpr_pagerank_device_noalloc.
//
// Who needs it: code that runs where it may not call cudaMalloc — inside a
// framework that owns all device memory through its own pool, on a serving
// thread with a fixed memory budget, or in a plug-in whose host forbids
// allocations while a request is in flight.  Such a caller brings its own
// inputs and outputs; every other buffer the solve needs lives in one
// file-scope device array of fixed size (g_scratch below).  Its size is set by
// kNoAllocMaxVertices: every GPU that loads this library holds these bytes until
// the process exits, whether or not the entry point is ever called.
//
// The solve is the one-kernel solve of small.cu (same arithmetic as the prepared
// graph's), whose state and vectors are placed in that array.
//
// Every call shares the one scratch array and leaves the last call's contents
// in it; each call clears what must start at zero.  Calls that overlap on the
// GPU (another host thread, or another stream) race on it and give wrong
// answers: callers serialise them.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <mutex>

#include "egpr_internal.cuh"

namespace egpr {
int arg_error(const char* why);
}

namespace {

using egpr::set_cuda_error;

constexpr int32_t kNoAllocMaxVertices = 1 << 18;  // 262,144 vertices
constexpr size_t kStateBytes = 256;
static_assert(sizeof(egpr::SmallState) <= kStateBytes, "state fits its slot");
// The state, then x0, x1, z0, z1 (FP32, kNoAllocMaxVertices each): 4 MiB + 256 B.
constexpr size_t kScratchBytes = kStateBytes + 4 * (size_t)kNoAllocMaxVertices * sizeof(float);

static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];

// Device address of g_scratch, looked up once per device with that device
// current.  In host code the name g_scratch stands for a host-side shadow, not
// for device memory, so kernels get this address instead.
std::mutex g_scratch_mu;
unsigned char* g_scratch_dev[64] = {};

int scratch_address(int dev, unsigned char** out) {
    if (dev < 0 || dev >= 64) return egpr::arg_error("egpr_pagerank_device_noalloc: device index out of range");
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_dev[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_scratch);
        if (e != cudaSuccess || !p) return set_cuda_error(e != cudaSuccess ? e : cudaErrorInvalidSymbol,
                                                         "cudaGetSymbolAddress (no-alloc scratch)");
        g_scratch_dev[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_scratch_dev[dev];
    return EGPR_SUCC;
}

}  // namespace

extern "C" EGPR_API int egpr_pagerank_device_noalloc(int32_t n, int64_t nnz, const int32_t* in_row,
                                                     const int32_t* in_col, const float* in_w,
                                                     const double* out_weight, double alpha, int32_t max_iter,
                                                     double tol, uint32_t flags, double* ranks, void* stream,
                                                     egpr_stats* stats) {
    using namespace egpr;
    const auto t0 = std::chrono::steady_clock::now();
    if (n <= 0) {
        if (stats) *stats = egpr_stats{};  // nothing to solve: zero sweeps, zero time
        return EGPR_SUCC;
    }
    if (n > kNoAllocMaxVertices)
        return arg_error("egpr_pagerank_device_noalloc: n exceeds the 262144-vertex limit of its fixed scratch");
    if (nnz < 0 || nnz > (int64_t)INT32_MAX) return arg_error("egpr_pagerank_device_noalloc: nnz out of range");
    if (!in_row || (nnz > 0 && !in_col) || !out_weight || !ranks)
        return arg_error("egpr_pagerank_device_noalloc: a required device pointer is NULL");
    if (!(alpha >= 0.0 && alpha < 1.0)) return arg_error("egpr_pagerank_device_noalloc: alpha must be in [0, 1)");
    if (max_iter < 1) max_iter = 1;
    if (!(tol > 0.0)) tol = 0.0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_cuda_error(e, "cudaGetDevice");
    unsigned char* base = nullptr;
    int rc = scratch_address(dev, &base);
    if (rc) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    SmallGraph G{n, nnz, in_row, in_col, in_w, out_weight, nullptr};
    float* f = reinterpret_cast<float*>(base + kStateBytes);
    constexpr size_t N = kNoAllocMaxVertices;
    SmallWork V{reinterpret_cast<SmallState*>(base), {f, f + N}, {f + 2 * N, f + 3 * N},
                reinterpret_cast<double*>(f + 2 * N)};  // the correction sweep's values, over both z buffers
    const int32_t others = small_in_flight(dev).load(std::memory_order_relaxed);
    if ((rc = small_solve(G, V, alpha, tol, max_iter, !(flags & EGPR_FLAG_NO_CORRECTION), ranks, others, s))) return rc;
    if (stats) {
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return set_cuda_error(e, "no-alloc solve");
        SmallState h;
        if ((e = cudaMemcpy(&h, base, sizeof(egpr::SmallState), cudaMemcpyDeviceToHost)) != cudaSuccess)
            return set_cuda_error(e, "no-alloc solve state");
        if (h.error) {
            egpr::arg_error("egpr_pagerank_device_noalloc: a barrier of the solve ran out of time");
            return h.error;
        }
        const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        stats->iterations = h.iter;
        stats->converged = h.converged;
        stats->residual = h.residual;
        stats->kernel_seconds = h.t_end > h.t_begin ? (double)(h.t_end - h.t_begin) * 1e-9 : 0.0;
        stats->total_seconds = secs;
        stats->bytes_per_iter = (int64_t)(n + 1) * 4 + nnz * (in_w ? 8 : 4) + (int64_t)n * 20;
        stats->launches = 2;
        stats->reserved = 0;
    }
    return EGPR_SUCC;
}
