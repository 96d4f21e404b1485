// The whole solve of a small graph in one cooperative kernel: single-vector
// PageRank / personalised PageRank on an inbound CSR (pagerank.py:75-139 restated as
// a pull), for prepared graphs of few entries (api.cu), for the no-allocation entry
// (noalloc.cu), and for an alpha outside [0, 1] on a graph of any size.
//
// Such a graph sweeps in a few microseconds, about what one launch costs, and its
// vectors live in L2, so nothing is laid out for it: a few lanes per row gather the
// carried values, all CTAs are resident and the sweeps are separated by grid
// barriers, and the kernel ends at the stop rule.  FP32 iterates, FP64 residual,
// dangling mass and rank sums added as order-free fixed-point integers, a final
// FP64 sweep from x_{k-1}, then normalisation.
//
// What bounds it: latency.  A sweep is a chain of dependent L2 reads (row offsets,
// sources, values, the row's data), about 5 us with its barrier on 1,000 vertices.
// Measured per solve: 1,000 vertices, 6 sweeps: 51 us on the device (165 us as a
// launch per phase); R-MAT scale 14, 5 sweeps: 141 us (160); the no-allocation entry on
// 50,001 weighted vertices with a limit of 100 sweeps: 176 us (720 as a launch per
// sweep).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "egpr_internal.cuh"

namespace egpr {
namespace {

constexpr int kThreadsNa = 1024;
constexpr int kWarpsNa = kThreadsNa / 32;
constexpr int32_t kWideRow = 128;   // entries: longer rows are summed by a warp,
constexpr int32_t kHugeRow = 1024;  // and these by the whole CTA (longer ones only where rows are long on average)
constexpr int64_t kCtaEntries = 2048;  // a CTA more per so many entries, while there are rows for its warps
constexpr int32_t kShares = 8;      // solves at a time that the SMs are shared by
constexpr int32_t kCtaRows = 4;     // rows per CTA from which long ones are left to the warps
constexpr unsigned long long kBarrierNs = 2000000000ull;  // bound of a barrier wait (2 s)
constexpr unsigned kFullNa = 0xffffffffu;

// Sums over rows that do not depend on how rows are dealt to threads: each number is
// rounded to a multiple of a unit u so large that the sums stay exact in FP64 (adding and
// subtracting 1.5 * 2^52 u rounds to one).  Ranks sum to 1: the FP32 sweeps' sums take
// u = 2^-50, of which FP32 ranks of 2^-27 and more are multiples (all ranks of a uniform
// teleport at the sizes served here), so nothing is lost there.  The FP64 sweep's rank
// sum, by which the result is divided, has a second part for what that leaves, with u = 2^-64.
__device__ __forceinline__ double na_round50(double v) { return (v + 6.0) - 6.0; }
__device__ __forceinline__ double na_round64(double v) {
    constexpr double m = 1.5 / 4096.0;
    return (v + m) - m;
}

// Adds multiples of 2^-64 to two words, two's-complement fixed point in units of 2^-32 and
// 2^-64: integer adds, so the totals do not depend on the order in which blocks finish.
__device__ __forceinline__ void na_fx_add(unsigned long long* a, double v) {
    const double t = v * 4294967296.0;
    const double f = floor(t);
    atomicAdd(a, (unsigned long long)(long long)f);
    atomicAdd(a + 1, (unsigned long long)rint((t - f) * 4294967296.0));
}

__device__ __forceinline__ double na_fx_join(unsigned long long hi, unsigned long long lo) {
    return (double)(long long)hi * (1.0 / 4294967296.0) + (double)lo * (1.0 / 18446744073709551616.0);
}

__device__ __forceinline__ unsigned long long na_global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__global__ void k_na_reset(SmallState* st) {
    st->t_begin = na_global_ns();
    st->t_end = 0ull;
    for (int i = 0; i < 18; ++i) (&st->acc[0][0])[i] = 0ull;
    st->residual = 0.0;
    st->iter = 0;
    st->converged = 0;
    st->ndang = 0;
    st->arrived = 0u;
    st->error = 0;
}

// Grid barrier number `k` (1, 2, ...) of the kernel; false when it gave up waiting
// (the kernel then ends, reports EGPR_TIMEOUT and leaves NaN for ranks).  The fences
// order every thread's accesses: thread 0's cover its CTA through the CTA barriers.
// The count of arrivals wraps in solves of very many sweeps: compared by difference.
__device__ bool na_barrier(SmallState* st, uint32_t k) {
    __shared__ int32_t s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&st->arrived, 1u);
        const uint32_t want = k * gridDim.x;
        bool ok = (int32_t)(__ldcg(&st->arrived) - want) >= 0;
        if (!ok) {
            const unsigned long long t0 = na_global_ns();
            while (!(ok = (int32_t)(*reinterpret_cast<volatile uint32_t*>(&st->arrived) - want) >= 0) &&
                   na_global_ns() - t0 < kBarrierNs) {
            }
        }
        if (!ok) atomicExch(&st->error, EGPR_TIMEOUT);
        __threadfence();
        s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}

// Rows are clamped to [0, nnz] and sources to [0, n): no access outside the inputs.
__device__ __forceinline__ void na_range(const SmallGraph& G, int32_t r, int64_t& b, int64_t& e) {
    b = __ldg(G.in_row + r);
    e = __ldg(G.in_row + r + 1);
    b = b < 0 ? 0 : (b > G.nnz ? G.nnz : b);
    e = e < b ? b : (e > G.nnz ? G.nnz : e);
}

// Sum over entries b + first, b + first + step, ... of w * z[source]; z was written
// earlier in this kernel, so it is read with coherent loads.
template <typename Real>
__device__ __forceinline__ Real na_sum(const SmallGraph& G, const Real* z, int64_t b, int64_t e, int first, int step) {
    Real acc = Real(0);
    constexpr int kAhead = 8;  // entries of a lane in flight
    for (int64_t p = b + first; p < e; p += kAhead * step) {
        int32_t u[kAhead];
        Real v[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const int64_t q = p + (int64_t)j * step;
            u[j] = q < e ? __ldg(G.in_col + q) : -1;
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) v[j] = u[j] >= 0 && u[j] < G.n ? z[u[j]] : Real(0);
        if (G.in_w) {
#pragma unroll
            for (int j = 0; j < kAhead; ++j) {
                const int64_t q = p + (int64_t)j * step;
                v[j] *= q < e ? (Real)__ldg(G.in_w + q) : Real(0);
            }
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) acc += v[j];
    }
    return acc;
}

// Sums over a CTA's rows.  FP32 sweep: residual, dangling mass, rank sum; FP64 sweep: the
// rank sum's two parts.
struct NaSums {
    double v[3] = {0.0, 0.0, 0.0};
};

// Finishes row r (see finish_row in sweep.cu).  jump: the dangling term, and the
// uniform teleport term where there is no teleport vector.
template <bool kFinal>
__device__ __forceinline__ void na_finish(const SmallGraph& G, int32_t r, double sum, double jump, double alpha,
                                          const float* xin, float* xout, float* zout, double* ranks, NaSums& A) {
    const double val = G.tele ? (sum + (1.0 - alpha) * (double)__ldg(G.tele + r)) + jump : sum + jump;
    if (kFinal) {
        ranks[r] = val;
        const double t = na_round50(val);
        A.v[0] += t;
        A.v[1] += na_round64(val - t);
    } else {
        const float xo = (float)val;
        A.v[0] += na_round50(fabs((double)xo - (double)xin[r]));
        xout[r] = xo;
        const double o = __ldg(G.outw + r);
        const bool dangling = o <= 1e-15;
        zout[r] = dangling ? 0.f : (float)(val * (alpha / o));  // rounded once, as in sweep.cu
        if (dangling) A.v[1] += na_round50((double)xo);
        A.v[2] += na_round50((double)xo);
    }
}

// One sweep over this CTA's rows: L lanes per row; units of 32 / L rows are dealt to
// the CTAs in turn.  Rows of more than kWideRow entries follow, a warp each, and
// those of more than huge_row, one at a time by the whole CTA.
template <bool kFinal, int L>
__device__ NaSums na_rows(const SmallGraph& G, int32_t huge_row, const typename std::conditional<kFinal, double, float>::type* z,
                          double jump, double alpha, const float* xin, float* xout, float* zout, double* ranks) {
    using Real = typename std::conditional<kFinal, double, float>::type;
    __shared__ unsigned s_wide[kWarpsNa], s_huge[kWarpsNa];
    __shared__ Real s_part[kWarpsNa];
    constexpr int kRows = 32 / L;
    const int32_t wide_row = L == 32 ? huge_row : kWideRow;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % L, grp = lane / L;
    const int64_t stride = (int64_t)gridDim.x * kWarpsNa;  // units of all CTAs together
    const int64_t units = ((int64_t)G.n + kRows - 1) / kRows;
    NaSums A;
    for (int64_t u = (int64_t)warp * gridDim.x + blockIdx.x; u < units; u += stride) {
        const int64_t r = u * kRows + grp;
        int64_t b = 0, e = 0;
        if (r < G.n) na_range(G, (int32_t)r, b, e);
        const bool mine = r < G.n && e - b <= wide_row;
        Real acc = mine ? na_sum<Real>(G, z, b, e, sub, L) : Real(0);
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(kFullNa, acc, o);
        if (mine && sub == 0) na_finish<kFinal>(G, (int32_t)r, (double)acc, jump, alpha, xin, xout, zout, ranks, A);
    }
    // the longer rows: thread t looks at the CTA's row t of each 1024
    const int64_t rounds = (units + stride - 1) / stride;  // a round: one unit per warp
    auto row_at = [&](int64_t j) {
        const int64_t u = (j / kRows) / kWarpsNa * stride + (j / kRows) % kWarpsNa * gridDim.x + blockIdx.x;
        return j < rounds * kWarpsNa * kRows && u < units ? u * kRows + j % kRows : (int64_t)G.n;
    };
    for (int64_t t0 = 0; t0 < rounds * kWarpsNa * kRows; t0 += kThreadsNa) {
        const int64_t r = row_at(t0 + threadIdx.x);
        int64_t b = 0, e = 0;
        if (r < G.n) na_range(G, (int32_t)r, b, e);
        const unsigned wide = __ballot_sync(kFullNa, e - b > wide_row && e - b <= huge_row);
        const unsigned huge = __ballot_sync(kFullNa, e - b > huge_row);
        if (lane == 0) {
            s_wide[warp] = wide;
            s_huge[warp] = huge;
        }
        if (!__syncthreads_or((wide | huge) != 0u)) continue;
        int turn = 0;  // the wide rows go to the warps in order
        for (int w = 0; w < kWarpsNa; ++w)
            for (unsigned bits = s_wide[w]; bits; bits &= bits - 1u) {
                if ((turn++ & (kWarpsNa - 1)) != warp) continue;
                const int64_t q = row_at(t0 + 32 * w + __ffs(bits) - 1);
                na_range(G, (int32_t)q, b, e);
                Real acc = na_sum<Real>(G, z, b, e, lane, 32);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFullNa, acc, o);
                if (lane == 0) na_finish<kFinal>(G, (int32_t)q, (double)acc, jump, alpha, xin, xout, zout, ranks, A);
            }
        for (int w = 0; w < kWarpsNa; ++w)
            for (unsigned bits = s_huge[w]; bits; bits &= bits - 1u) {
                const int64_t q = row_at(t0 + 32 * w + __ffs(bits) - 1);
                na_range(G, (int32_t)q, b, e);
                Real acc = na_sum<Real>(G, z, b, e, (int)threadIdx.x, kThreadsNa);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFullNa, acc, o);
                if (lane == 0) s_part[warp] = acc;
                __syncthreads();
                if (warp == 0) {
                    Real s = s_part[lane];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFullNa, s, o);
                    if (lane == 0) na_finish<kFinal>(G, (int32_t)q, (double)s, jump, alpha, xin, xout, zout, ranks, A);
                }
                __syncthreads();
            }
        __syncthreads();  // s_wide and s_huge are read
    }
    return A;
}

// Adds the CTA's sums to the accumulator words.
__device__ void na_reduce(unsigned long long* acc, NaSums A) {
    __shared__ double red[kWarpsNa][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 3; ++i) A.v[i] += __shfl_xor_sync(kFullNa, A.v[i], o);
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < 3; ++i) red[warp][i] = A.v[i];
    __syncthreads();
    if (threadIdx.x < 3) {
        double s = 0.0;
        for (int w = 0; w < kWarpsNa; ++w) s += red[w][threadIdx.x];
        na_fx_add(acc + 2 * threadIdx.x, s);
        __threadfence();
    }
}

// The whole solve.  All CTAs are resident (cooperative launch).
template <int L>
__global__ void __launch_bounds__(kThreadsNa, 1)
k_na_solve(SmallGraph G, SmallWork V, double alpha, double tol, int32_t max_iter, int32_t correction,
           int32_t huge_row, double* ranks) {
    SmallState* st = V.st;
    const int32_t n = G.n;
    const int64_t tid = (int64_t)blockIdx.x * kThreadsNa + threadIdx.x, nthreads = (int64_t)gridDim.x * kThreadsNa;
    const double c1 = G.tele ? 0.0 : (1.0 - alpha) / (double)n, tol_n = tol * (double)n;
    uint32_t barrier = 0;
    bool ok = true;
    // x0 = 1/n; z0 = x0 * alpha/outw (0 for a dangling source, outw <= 1e-15,
    // pagerank.py:118); count of dangling vertices
    const float x0 = (float)(1.0 / (double)n);
    int32_t dang = 0;
    for (int64_t v = tid; v < n; v += nthreads) {
        const double o = __ldg(G.outw + v);
        const bool dangling = o <= 1e-15;
        V.x[0][v] = x0;
        V.z[0][v] = dangling ? 0.f : (float)(alpha / o / (double)n);
        dang += dangling ? 1 : 0;
    }
    for (int o = 16; o > 0; o >>= 1) dang += __shfl_down_sync(kFullNa, dang, o);
    if ((threadIdx.x & 31) == 0 && dang) atomicAdd(&st->ndang, dang);
    ok = na_barrier(st, ++barrier);
    double dmass = alpha * ((double)__ldcg(&st->ndang) * (double)x0) / (double)n, dmass_prev = dmass;
    double residual = 0.0, xsum = 0.0;
    int32_t iter = 0;
    bool conv = false;
    // every CTA reads the same sums after a barrier and takes the same decision
    while (ok && !conv && iter < max_iter) {
        unsigned long long* acc = st->acc[iter % 3];
        const int par = iter & 1;
        na_reduce(acc, na_rows<false, L>(G, huge_row, V.z[par], c1 + dmass, alpha, V.x[par], V.x[par ^ 1], V.z[par ^ 1], nullptr));
        ok = na_barrier(st, ++barrier);
        unsigned long long w[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) w[i] = __ldcg(acc + i);
        // the set of the sweep before: every CTA has read it, the sweep after next adds to it
        if (blockIdx.x == 0 && threadIdx.x < 6) st->acc[(iter + 2) % 3][threadIdx.x] = 0ull;
        residual = na_fx_join(w[0], w[1]);
        xsum = na_fx_join(w[4], w[5]);
        dmass_prev = dmass;
        dmass = alpha * na_fx_join(w[2], w[3]) / (double)n;
        ++iter;
        conv = residual < tol_n;
    }
    if (tid == 0) {
        st->residual = residual;
        st->iter = iter;
        st->converged = conv ? 1 : 0;
    }
    if (ok && correction) {
        // the last sweep again in FP64, from x_{k-1}
        const float* xp = V.x[(iter - 1) & 1];
        for (int64_t u = tid; u < n; u += nthreads) {
            const double o = __ldg(G.outw + u);
            V.z64[u] = o <= 1e-15 ? 0.0 : alpha * (double)xp[u] / o;
        }
        ok = na_barrier(st, ++barrier);
        if (ok) {
            unsigned long long* acc = st->acc[iter % 3];
            na_reduce(acc, na_rows<true, L>(G, huge_row, V.z64, c1 + dmass_prev, alpha, xp, nullptr, nullptr, ranks));
            ok = na_barrier(st, ++barrier);
            xsum = na_fx_join(__ldcg(acc), __ldcg(acc + 1)) + na_fx_join(__ldcg(acc + 2), __ldcg(acc + 3));
        }
    }
    if (ok && __ldcg(&st->error) == 0) {  // final normalisation (pagerank.py:134-139)
        const float* xl = V.x[iter & 1];
        const double inv = xsum > 0.0 ? 1.0 / xsum : 0.0;
        for (int64_t v = tid; v < n; v += nthreads) {
            const double val = correction ? __ldcg(ranks + v) : (double)xl[v];
            ranks[v] = xsum > 0.0 ? val * inv : 1.0 / (double)n;
        }
    } else {  // a barrier ran out of time: no unfinished rank is taken for a result
        for (int64_t v = tid; v < n; v += nthreads) ranks[v] = __longlong_as_double(0x7ff8000000000000ll);
    }
    if (threadIdx.x == 0) atomicMax(&st->t_end, na_global_ns());
}

}  // namespace

// Prepared graphs whose single-vector solves run here: up to 2^18 entries.  Whole calls
// of 20 sweeps, here and in the blocked sweep: R-MAT with 111, 228, 468, 955 and 1,942 K
// entries 410 and 554, 484 and 575, 539 and 596, 687 and 642, 846 and 724 us; uniform
// with 131, 262, 524, 1,048 and 2,097 K entries 247 and 595, 311 and 584, 341 and 645,
// 421 and 676, 549 and 810 us.  So the limit keeps to sizes where it wins on both
// kinds.  EGPR_SMALL_NNZ sets it (0: none).
bool small_wanted(int32_t n, int64_t nnz) {
    const char* e = std::getenv("EGPR_SMALL_NNZ");
    const int64_t most = e ? std::atoll(e) : (int64_t)1 << 18;
    return nnz <= most && n <= most;
}

std::atomic<int32_t>& small_in_flight(int device) {
    static std::atomic<int32_t> count[64];
    return count[device >= 0 && device < 64 ? device : 0];
}

// Sets the state up and enqueues the solve.
int small_solve(const SmallGraph& graph, const SmallWork& work, double alpha, double tol, int32_t max_iter,
                bool with_correction, double* ranks, int32_t others, cudaStream_t s) {
    SmallGraph G = graph;
    SmallWork V = work;
    int32_t correction = with_correction ? 1 : 0;
    // lanes per row by the mean degree; one CTA per SM at most, fewer where there are
    // neither rows nor entries for all warps.  A warp per row: with 16 lanes, rows above
    // kWideRow would take the second pass of na_rows, 5 us per sweep (8,192 vertices of
    // degree 96 and 130, 20 sweeps: 0.40 and 0.49 ms with 16 lanes, 0.31 and 0.31 with 32;
    // many rows hide it: 131,072 of degree 96, 1.52 and 1.64 ms)
    const int64_t degree = G.nnz / G.n;
    const int lanes = degree <= 6 ? 4 : degree <= 20 ? 8 : degree <= (G.n <= 65536 ? 90 : 110) ? 16 : 32;
    const void* kernel = lanes == 4    ? (const void*)k_na_solve<4>
                         : lanes == 8  ? (const void*)k_na_solve<8>
                         : lanes == 16 ? (const void*)k_na_solve<16>
                                       : (const void*)k_na_solve<32>;
    const int64_t units = ((int64_t)G.n + 32 / lanes - 1) / (32 / lanes);
    const int64_t want = std::min(units, std::max((units + kWarpsNa - 1) / kWarpsNa, G.nnz / kCtaEntries));
    // A solve alone takes all SMs; beside others it takes its share, so that they run at
    // the same time (a cooperative launch waits until all its CTAs fit).  The results
    // do not depend on the number of CTAs.  R-MAT scale 14, 20 sweeps, solves per second
    // with 1, 4, 8 and 16 threads: 2,052, 7,277, 6,026 and 5,950; 2,051, 2,324, 2,332 and
    // 2,306 where every solve takes all SMs
    const int most = std::max(1, sweep_grid() / (1 + std::min(others, kShares - 1)));
    int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, most));
    // an odd number of CTAs: dealt by a power of two, the heavy rows of an R-MAT graph
    // (ids with few bits set) would all fall to the first CTAs
    if (grid > 1 && grid % 2 == 0) --grid;
    // Where rows are long on average and every CTA has several, the warps take them up to
    // four times the mean, one each; the whole CTA on one row after another leaves most
    // warps waiting (2,048 vertices with 4 M entries, 20 sweeps: 2.87 ms, 0.45 so)
    int32_t huge_row = kHugeRow;
    if (G.n >= kCtaRows * std::min<int64_t>(want, sweep_grid()))
        huge_row = (int32_t)std::max<int64_t>(kHugeRow, std::min<int64_t>(4 * degree, INT32_MAX));
    void* args[] = {&G, &V, &alpha, &tol, &max_iter, &correction, &huge_row, &ranks};
    k_na_reset<<<1, 1, 0, s>>>(V.st);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaLaunchCooperativeKernel(kernel, dim3((unsigned)grid), dim3(kThreadsNa), args, 0, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_cuda_error(e, "small solve launch");
    }
    return EGPR_SUCC;
}

}  // namespace egpr
