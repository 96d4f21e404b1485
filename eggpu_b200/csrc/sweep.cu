// The power iteration of the single-vector solve, for one or many graphs.
//
// A sweep computes, for every vertex v (one "row" of the inbound CSR),
//     x_new[v] = sum_{u -> v} w_uv * z[u]  +  jump
// with z[u] = alpha * x[u] / outw[u] (0 for dangling u) and
// jump = (1-alpha)/n + alpha * (dangling mass)/n — the arithmetic of the
// reference's _pagerank_power_iteration (easygraph/functions/centrality/
// pagerank.py:112-132) evaluated as a pull — and with it:
//   * the FP64 L1 residual sum |x_new - x| (pagerank.py:127-130),
//   * the FP64 dangling mass of x_new for the next sweep (pagerank.py:117-120),
//   * z_new = x_new * alpha / outw for the next sweep,
//   * the FP64 sum of x_new (final normalisation, pagerank.py:134-139),
//   * the stop decision err < tol*n (pagerank.py:131) and, through a CUDA
//     graph conditional node, whether the next sweep runs at all.
// This replaces, per iteration, the reference GPU path's cuSPARSE SpMV, cuBLAS
// Sdot, two memsets, add_base_and_reduce, scale_vec and the two host round
// trips (gpu_easygraph/functions/centrality/pagerank.cu:591-664).
//
// A sweep has two phases over the blocked layout (egpr_internal.cuh):
//   1. k_gather.  A CTA owns a contiguous share of the tiles (equal cost over
//      the CTAs, so most CTAs see one or two blocks).  It stages the block's
//      carried values in shared memory (TMA bulk copies), its warps take tiles
//      of 256 entries, gather from shared memory, sum each lane's entries run by
//      run, join the runs that cross lanes with a five-step shuffle scan and
//      write the tile's pairs, which are consecutive.
//   2. k_rows.  A CTA owns a row tile.  Its warps add the row tile's pairs into
//      64-bit fixed-point sums in shared memory (integer atomics: exact, so the
//      order of the blocks does not matter and no warp waits), then the rows are
//      finished with coalesced loads and stores.  The last CTA to leave advances
//      every graph's state.
// FP64 sums (residual, dangling mass, rank sum) are added as fixed-point
// integers, so their total does not depend on the order in which row tiles
// finish.  No warp waits on another; the only wait is on the staging copies, and
// it is bounded.
//
// What bounds it.  Gathering every entry from global memory, as a single-phase sweep
// does, costs one 32-byte sector per entry that misses L1: R-MAT scale 25 weighted took
// 2.01 ms per sweep, 0.97 of what 560 M sectors take at one per clock and SM, and
// scale 22 took 0.222 ms.  Here k_gather is bound by issue and shared-memory
// wavefronts (60% each of their peaks at scale 22: 90 us for 65 M entries, 11 M
// pairs) and by HBM where there are weights (scale 25: 1.03 ms, 4.0 GB); k_rows is
// bound by the latency of its loads (78 us and 0.70 ms, 1.7 GB).  Per sweep: scale 22 0.172
// ms, scale 25 weighted 1.71 ms, Erdos-Renyi 1.5 M vertices 93 us (112 before), R-MAT
// 100 K vertices 30 us (56 before).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "egpr_internal.cuh"

namespace egpr {
namespace {

// Phase 1: independent warps per CTA, one CTA per SM.  The FP64 block leaves room
// for the run sums of 24.
template <typename Real>
constexpr int kGatherWarps = std::is_same<Real, double>::value ? 24 : 32;
constexpr int kRowWarps = 16;         // phase 2: warps per CTA
constexpr int kRowThreads = 32 * kRowWarps;
constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kCopyPiece = 32768;                 // bytes per staging copy
constexpr unsigned long long kWaitNs = 2000000000ull;  // bound of the staging wait (2 s)

__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ int ldcg(const int* p) { return __ldcg(p); }
__device__ __forceinline__ unsigned long long ldcg_u64(const unsigned long long* p) { return __ldcg(p); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    return v;  // valid in lane 0
}

// ---- PTX wrappers ------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// A lane's eight weights: one 32-byte load, read once per sweep (no L1 space, first
// out of L2).
__device__ __forceinline__ void ld_stream8(const float* p, float (&w)[kLaneItems]) {
    asm("ld.global.nc.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7])
        : "l"(p));
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---- per-graph view ------------------------------------------------------------
// What finishing a row needs of the graph a warp works on.
struct RowView {
    const float* xin;       // previous ranks
    float* xout;
    float* zout;            // by source rank
    const double* scale;
    const int32_t* rank;
    const float* tele;
    double* out;
    double jump;            // (1-alpha)/n + dangling term (uniform teleport)
    double dmass;           // dangling term alone (personalised teleport)
    double one_minus_alpha;
    int32_t personalised;
};

template <bool kFinal>
__device__ RowView make_view(const GraphDev& G, GraphState* st, int32_t iter) {
    RowView W;
    W.one_minus_alpha = 1.0 - st->alpha;
    W.personalised = st->personalised;
    W.scale = G.scale;
    W.rank = G.rank;
    W.tele = G.tele;
    W.out = G.out;
    if (!kFinal) {
        const int par = iter & 1;
        W.xin = G.x[par];
        W.xout = G.x[par ^ 1];
        W.zout = G.z[par ^ 1];
        W.dmass = ldcg(&st->dmass);
    } else {
        W.xin = G.x[(iter - 1) & 1];  // x_{k-1}: the input of the last sweep
        W.xout = nullptr;
        W.zout = nullptr;
        W.dmass = ldcg(&st->dmass_prev);
    }
    W.jump = st->c1 + W.dmass;
    return W;
}

// Finishes row v given its gathered sum; accumulates residual / dangling /
// rank sums.  FP32 sweep: writes x_new and z_new; the residual compares the
// stored FP32 iterates, so the loop can stop once they no longer change even when
// tol*n is below FP32 resolution.  z_new comes from the row's FP64 value and the
// FP64 scale and is rounded once: an FP32 scale has the same error in every sweep and
// for every source of one out-degree, and such errors do not average out over a row
// (R-MAT, 20 sweeps, mean relative error over 8 draws: scale 21 9.9e-9 -> 1.9e-9, scale 22
// 6.3e-9 -> 3.1e-9; a sweep of scale 22 takes 172 us instead of 168).  FP64 correction sweep: writes the FP64 result.
template <bool kFinal>
__device__ __forceinline__ void finish_row(const RowView& W, int32_t v, double acc, float xin, double scale,
                                           int32_t rank, double& err, double& dsum, double& xsum) {
    double val;
    if (W.personalised) val = (acc + W.one_minus_alpha * (double)__ldg(W.tele + v)) + W.dmass;
    else val = acc + W.jump;
    if (!kFinal) {
        const float xo = (float)val;
        err += (double)fabsf(xo - xin);
        W.xout[v] = xo;
        if (rank >= 0) W.zout[rank] = (float)(val * scale);
        if (scale == 0.0) dsum += (double)xo;
        xsum += (double)xo;
    } else {
        err += fabs(val - (double)xin);
        W.out[v] = val;
        xsum += val;
    }
}

// ---- order-free FP64 sums ---------------------------------------------------------
// A value is split into two's-complement words in units of 2^-32 and of 2^-64
// (the remainder, rounded) and added as integers, so the total does not depend
// on the order in which row tiles finish.  Partial sums here are far below 2^31
// and there are far fewer than 2^20 terms per word, so no word overflows and
// both convert to double exactly.
// Adds v to two words that only the calling thread touches.
__device__ __forceinline__ void fx_add_own(unsigned long long* a, double v) {
    const double t = v * 4294967296.0;  // exact
    const double f = floor(t);
    a[0] += (unsigned long long)(long long)f;
    a[1] += (unsigned long long)rint((t - f) * 4294967296.0);
}

__device__ __forceinline__ double fx_join(unsigned long long hi, unsigned long long lo) {
    return (double)(long long)hi * (1.0 / 4294967296.0) + (double)lo * (1.0 / 18446744073709551616.0);
}

// Accumulator slot of (graph, k): each graph has acc_sub slots so that
// concurrent warps rarely add to the same address.
__device__ __forceinline__ unsigned long long* acc_slot(const SweepParams& P, int32_t gi, int32_t k) {
    return P.acc + (size_t)kAccWords * ((size_t)gi * (size_t)P.acc_sub + (size_t)(k % P.acc_sub));
}

// End of a sweep, run by the whole last CTA to leave phase 2: per graph,
// turns the accumulators into the residual, dangling mass and rank sum, clears
// them, and advances the graph's state (pagerank.py:117-131).
template <bool kFinal>
__device__ void launch_tail(const SweepParams& P) {
    const int tid = threadIdx.x;
    __threadfence();
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    for (int32_t gi = warp; gi < P.ngraphs; gi += (int32_t)(blockDim.x >> 5)) {
        GraphState* st = P.states + gi;
        if (!kFinal && ldcg(&st->done)) continue;
        // all of a lane's loads first (they are independent), then the clears
        unsigned long long w[6] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
        for (int32_t k0 = 0; k0 < P.acc_sub; k0 += 64) {
            unsigned long long* a = P.acc + (size_t)kAccWords * ((size_t)gi * (size_t)P.acc_sub + (size_t)(k0 + lane));
            unsigned long long* b = a + (size_t)kAccWords * 32;
            const bool ha = k0 + lane < P.acc_sub, hb = k0 + 32 + lane < P.acc_sub;
            unsigned long long ra[6], rb[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                ra[i] = ha ? ldcg_u64(a + i) : 0ull;
                rb[i] = hb ? ldcg_u64(b + i) : 0ull;
            }
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                w[i] += ra[i] + rb[i];
                if (ha) a[i] = 0ull;
                if (hb) b[i] = 0ull;
            }
        }
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) w[i] += __shfl_down_sync(kFull, w[i], o);
        if (lane == 0) {
            const double e = fx_join(w[0], w[1]), d = fx_join(w[2], w[3]), x = fx_join(w[4], w[5]);
            if (!kFinal) {
                st->residual = e;
                st->dsum = d;
                st->xsum = x;
                st->dmass_prev = st->dmass;
                st->dmass = st->alpha * d / (double)P.graphs[gi].n;
                const int32_t it = st->iter + 1;
                st->iter = it;
                const bool conv = e < st->tol_n;
                if (conv || it >= st->max_iter) {
                    st->done = 1;
                    st->converged = conv ? 1 : 0;
                    atomicSub(&P.ctl->active, 1);
                }
            } else {
                st->residual64 = e;
                st->xsum = x;
            }
        }
    }
    __threadfence();
    __syncthreads();
}

// ---- phase 1: entries to pairs ----------------------------------------------------
template <typename Real>
struct GatherSmem {
    Real z[kBlockSrc + 8];                    // the block's carried values; z[kBlockSrc] = 0 (padding entries)
    Real runs[kGatherWarps<Real>][kTileItems];  // run sums of each warp's tile
};

template <typename Real>
__global__ void __launch_bounds__(32 * kGatherWarps<Real>, 1) k_gather(SweepParams P) {
    constexpr bool kFinal = std::is_same<Real, double>::value;
    constexpr int kWarps = kGatherWarps<Real>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    GatherSmem<Real>& S = *reinterpret_cast<GatherSmem<Real>*>(smem_raw);
    __shared__ __align__(8) uint64_t bar;
    __shared__ int32_t s_idle;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        s_idle = (!kFinal && ldcg(&P.ctl->active) <= 0) ? 1 : 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        S.z[kBlockSrc] = Real(0);
    }
    __syncthreads();
    if (s_idle) return;
    const int32_t u1 = P.cta_unit[blockIdx.x + 1];
    uint32_t parity = 0;
    for (int32_t u = P.cta_unit[blockIdx.x]; u < u1; ++u) {
        const GatherUnit U = P.units[u];
        const GraphDev& G = P.graphs[U.graph];
        const GraphState* st = P.states + U.graph;
        if (!kFinal && ldcg(&st->done)) continue;  // converged before this sweep: the same for the whole CTA
        const Real* z = kFinal ? reinterpret_cast<const Real*>(G.z64)
                               : reinterpret_cast<const Real*>(G.z[ldcg(&st->iter) & 1]);
        const bool staged = G.idx32 == nullptr;
        if (staged) {
            z += (size_t)U.block * kBlockSrc;
            __syncthreads();  // every warp is done with the previous block
            if (threadIdx.x == 0) {
                const int32_t nz = min(kBlockSrc, G.nsrc - U.block * kBlockSrc);
                const uint32_t bytes = ((uint32_t)nz * (uint32_t)sizeof(Real) + 15u) & ~15u;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads before the copies' writes
                mbar_arrive_tx(&bar, bytes);
                for (uint32_t off = 0; off < bytes; off += kCopyPiece)
                    bulk_load(reinterpret_cast<unsigned char*>(S.z) + off, reinterpret_cast<const unsigned char*>(z) + off,
                              min(kCopyPiece, bytes - off), &bar);
            }
            bool ok = mbar_try(&bar, parity);
            if (!ok) {
                const unsigned long long t0 = global_ns();
                while (!(ok = mbar_try(&bar, parity)) && global_ns() - t0 < kWaitNs) {
                }
            }
            parity ^= 1u;
            if (__syncthreads_or(!ok)) {
                // The copies did not arrive in time: report it, wait (again with a
                // limit) so that none is in flight into this CTA, and leave.
                if (threadIdx.x == 0) {
                    atomicExch(&P.ctl->error, EGPR_TIMEOUT);
                    const unsigned long long t0 = global_ns();
                    while (!mbar_try(&bar, parity ^ 1u) && global_ns() - t0 < kWaitNs) {
                    }
                }
                return;
            }
        }
        const uint4* idx = reinterpret_cast<const uint4*>(G.idx) + lane;
        const uint4* idx32 = reinterpret_cast<const uint4*>(G.idx32) + 2 * lane;
        const unsigned short* bits = reinterpret_cast<const unsigned short*>(G.tile_bits) + lane;
        const float* wts = G.w ? G.w + kLaneItems * lane : nullptr;
        const int32_t* tpair = G.tile_pair;
        Real* pairs = static_cast<Real*>(G.pairs);
        Real* const scr = S.runs[warp];
        // A tile's indices, marks and pair range; two tiles are in flight, each in
        // registers of its own (moving a value between registers would wait for it).
        struct Ahead {
            uint4 ix;
            uint32_t mw;
            int32_t p0, p1;
        };
        // Chunks are dealt to the warps in turn: the tile after `at` of this warp.
        const int32_t cs = G.chunk_shift, in_chunk = (1 << cs) - 1, skip = (kWarps - 1) << cs;
        auto after = [&](int32_t at) { return ((at + 1 - U.tile0) & in_chunk) ? at + 1 : at + 1 + skip; };
        auto fetch = [&](int32_t at, Ahead& f) {
            if (at >= U.tile1) return;
            if (staged) f.ix = __ldcs(idx + (size_t)at * 32);
            f.mw = __ldcs(bits + (size_t)at * (2 * kTileWords));
            f.p0 = __ldg(tpair + at);
            f.p1 = __ldg(tpair + at + 1);
        };
        Real carry = Real(0);  // the run still open at the end of the previous tile of the chunk
        auto tile = [&](int32_t t, int32_t ahead, Ahead& f) {
            Real v[kLaneItems];
            if (staged) {
                v[0] = S.z[f.ix.x & 0xffffu];
                v[1] = S.z[f.ix.x >> 16];
                v[2] = S.z[f.ix.y & 0xffffu];
                v[3] = S.z[f.ix.y >> 16];
                v[4] = S.z[f.ix.z & 0xffffu];
                v[5] = S.z[f.ix.z >> 16];
                v[6] = S.z[f.ix.w & 0xffffu];
                v[7] = S.z[f.ix.w >> 16];
            } else {
                const uint4 a = __ldcs(idx32 + (size_t)t * 64), b = __ldcs(idx32 + (size_t)t * 64 + 1);
                const uint32_t r[kLaneItems] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int u = 0; u < kLaneItems; ++u) v[u] = (int32_t)r[u] >= 0 ? __ldg(z + r[u]) : Real(0);
            }
            if (wts) {
                float w[kLaneItems];
                ld_stream8(wts + (size_t)t * kTileItems, w);
#pragma unroll
                for (int u = 0; u < kLaneItems; ++u) v[u] *= (Real)w[u];
            }
            const uint32_t m = f.mw;
            const int32_t pair = f.p0, nm = f.p1 - f.p0;
            fetch(ahead, f);
            if (nm == 0) {  // the inside of a long run
                Real part = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(kFull, part, o);
                carry += part;
                return;
            }
            // per-lane run sums, stored by mark ordinal without branches; the
            // lane's first one still lacks the open sums of the lanes below
            Real* const first = scr + (m >> 8);
            Real* k = first;
            Real acc = Real(0);
#pragma unroll
            for (int u = 0; u < kLaneItems; ++u) {
                acc += v[u];
                if (m & (1u << u)) {
                    *k++ = acc;
                    acc = Real(0);
                }
            }
            // segmented inclusive scan of the open sums; a lane's segment starts
            // at the nearest marked lane at or below it
            const bool marked = (m & 0xffu) != 0u;
            const unsigned le = __ballot_sync(kFull, marked) & (0xffffffffu >> (31 - lane));
            const int span = lane - (le ? 31 - __clz(le) : 0);  // lanes below that belong to the segment
            Real open = lane == 0 && !marked ? carry + acc : acc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const Real up = __shfl_up_sync(kFull, open, o);
                if (o <= span) open += up;
            }
            Real below = __shfl_up_sync(kFull, open, 1);
            if (lane == 0) below = carry;
            if (marked) *first += below;
            carry = __shfl_sync(kFull, open, 31);  // 0 at a chunk's end: its last entry ends a run
            __syncwarp();
            for (int32_t j = lane; j < nm; j += 32) pairs[pair + j] = scr[j];
            __syncwarp();
        };
        Ahead f0 = {}, f1 = {};
        int32_t t0 = U.tile0 + (warp << cs), t1 = after(t0);
        fetch(t0, f0);
        fetch(t1, f1);
        while (t0 < U.tile1) {
            int32_t t2 = after(t1);
            tile(t0, t2, f0);
            if (t1 >= U.tile1) break;
            t0 = t2;
            t2 = after(t2);
            tile(t1, t2, f1);
            t1 = t2;
        }
    }
}

// ---- phase 2: pairs to rows ---------------------------------------------------------
// A row's sum is a 64-bit integer in units of 2^-62 (alpha lies in [0, 1] here and ranks
// sum to 1, so a row's sum stays below 2).  It is held as two words, added
// with native 32-bit shared-memory atomics and a carry (4 to 6 per clock per SM
// measured; a 64-bit shared atomicAdd is a compare-and-swap loop, 2 to 5).  The FP64
// sweep adds what is left below the unit in a second such integer, in units 2^-44
// smaller: 106 bits.
//
// A sum of at least 2^-36 (FP64: 2^-50) keeps 26 (56) bits, and so does every pair of that
// size: less error than a chain of FP32 (FP64) adds has.  Smaller sums lose bits; they
// matter only where a row gets nothing else, that is in a personalised solve on a
// graph without dangling mass, far from the seeds.  There row tiles with small pairs
// add their smallest rows again in finer units (refine_rows).  The looking out is in a
// variant of the kernel for such solves: 50 personalised sweeps on 100 K vertices with
// dangling ones 1.59 ms on the device instead of 1.58, on 1 M vertices without 3.90
// instead of 3.82 (in every solve it would cost the plain ones 3%).
constexpr double kUnit = 4611686018427387904.0;    // 2^62 units per 1
constexpr double kFine = 68719476736.0;            // 2^36 between one unit and the next finer
template <typename Real>
constexpr int kRowBits = std::is_same<Real, double>::value ? 12 : 26;  // log2 of the units a sum has at least
template <typename Real>
constexpr int kFineLevels = std::is_same<Real, double>::value ? 4 : 3;  // FP32: to its smallest number, 2^-149
// A term of every row of at least this much makes the bits below the unit immaterial.
template <typename Real>
constexpr double kRowFloor = std::is_same<Real, double>::value ? 1.0 / 4503599627370496.0 : 1.0 / 274877906944.0;  // 2^-52, 2^-38
// Returns whether the upper word was left alone.
__device__ __forceinline__ bool add_word(uint32_t* lo, uint32_t* hi, unsigned long long q) {
    const uint32_t ql = (uint32_t)q;
    uint32_t qh = (uint32_t)(q >> 32);
    if (ql) {
        const uint32_t old = atomicAdd(lo, ql);
        qh += old + ql < ql ? 1u : 0u;
    }
    if (qh) {
        atomicAdd(hi, qh);
        return false;
    }
    return true;
}

template <typename Real>
struct RowSums {
    uint32_t* w;  // lo words, hi words (FP64: then the same of the remainders)
    int32_t rows;
    __device__ __forceinline__ void clear(int32_t i) {
#pragma unroll
        for (int k = 0; k < (int)(sizeof(Real) / 2); ++k) w[i + k * rows] = 0u;
    }
    __device__ __forceinline__ bool add_units(int32_t i, double t) {  // t: in units, exact
        const double f = floor(t);
        const bool low = add_word(w + i, w + i + rows, (unsigned long long)__double2ll_rn(f));
        add_word(w + i + 2 * rows, w + i + 3 * rows, (unsigned long long)__double2ll_rn((t - f) * 17592186044416.0));
        return low;
    }
    // Returns false for a pair of 2^-30 and more.
    __device__ __forceinline__ bool add(int32_t i, Real v) {
        if constexpr (sizeof(Real) == 4)
            return add_word(w + i, w + i + rows, (unsigned long long)__float2ll_rn(v * (float)kUnit));
        else return add_units(i, v * kUnit);
    }
    __device__ __forceinline__ void add_fine(int32_t i, Real v, double unit) {
        if constexpr (sizeof(Real) == 4) add_word(w + i, w + i + rows, (unsigned long long)__double2ll_rn((double)v * unit));
        else add_units(i, v * unit);
    }
    __device__ __forceinline__ unsigned long long units(int32_t i) const {
        return (unsigned long long)w[i] | (unsigned long long)w[i + rows] << 32;
    }
    __device__ __forceinline__ double get(int32_t i, double unit = kUnit) const {
        const double inv = 1.0 / unit;
        double r = (double)(long long)units(i) * inv;
        if constexpr (sizeof(Real) == 8) {
            const unsigned long long p = (unsigned long long)w[i + 2 * rows] | (unsigned long long)w[i + 3 * rows] << 32;
            r += (double)p * (inv * (1.0 / 17592186044416.0));
        }
        return r;
    }
    // After a refinement: the sum as a double instead.
    __device__ __forceinline__ void set_double(int32_t i, double v) {
        w[i] = (uint32_t)__double2loint(v);
        w[i + rows] = (uint32_t)__double2hiint(v);
    }
    __device__ __forceinline__ double get_double(int32_t i) const {
        return __hiloint2double((int)w[i + rows], (int)w[i]);
    }
};

// Adds the rows of a row tile whose sums have too few units again, in units 2^36 times
// finer at each level, until they have enough or no pair is left that is too small for the
// level, and leaves every row's sum as a double.  What is added again stayed below
// 2^kRowBits units of the level before, so nothing overflows.  `todo`: a bit per row that
// still lacks units.  Called by the whole CTA, after a barrier, and ends with one.  Rare (see
// above): it reads the row tile's pairs once more per level.
template <typename Real>
__device__ void refine_rows(RowSums<Real> R, uint32_t* todo, const GraphDev& G, int32_t tile) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int32_t nr = __ldg(G.row_tile + tile + 1) - __ldg(G.row_tile + tile);
    const int32_t k0 = __ldg(G.row_step + tile), k1 = __ldg(G.row_step + tile + 1);
    const Real* pairs = static_cast<const Real*>(G.pairs);
    constexpr unsigned long long enough = 1ull << kRowBits<Real>;
    double unit = kUnit;
    bool more = true;
    for (int level = 0;; ++level) {
        bool any = false;
        for (int32_t i = tid; i < ((nr + 31) & ~31); i += kRowThreads) {  // whole warps: 32 rows, one word
            const bool mine = i < nr && (level == 0 || (todo[i >> 5] >> (i & 31)) & 1u);
            const bool again = mine && more && R.units(i) < enough;
            const unsigned word = __ballot_sync(kFull, again);
            if (again) R.clear(i);
            else if (mine) R.set_double(i, R.get(i, unit));
            if (lane == 0) todo[i >> 5] = word;
            any |= again;
        }
        if (!__syncthreads_or(any)) return;
        unit *= kFine;
        const double least = (double)enough / unit;
        bool small = false;  // a pair that the next level holds better
        for (int32_t k = k0 + warp; k < k1; k += kRowWarps) {
            const int2 st = __ldg(G.steps + k);
            for (int32_t j = lane; j < st.y; j += 32) {
                const int32_t i = __ldg(G.pair_row + st.x + j);
                if (!((todo[i >> 5] >> (i & 31)) & 1u)) continue;
                const Real v = __ldcg(pairs + st.x + j);
                R.add_fine(i, v, unit);
                small |= v != Real(0) && (double)v < least;
            }
        }
        more = __syncthreads_or(small) && level + 1 < kFineLevels<Real>;
    }
}

// kWatch: rows may get nothing but their sum (see refine_rows).
template <typename Real, bool kWatch>
__global__ void __launch_bounds__(kRowThreads, kRowTilesPerSm) k_rows(SweepParams P) {
    constexpr bool kFinal = std::is_same<Real, double>::value;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ RowView W;
    __shared__ double part[kRowWarps][3];
    __shared__ unsigned long long words[6];          // fixed-point sums of the row tiles of `graph` finished here
    __shared__ int32_t s_idle, s_last, s_next;
    __shared__ uint32_t todo[kWatch ? kMaxTileRows / 32 : 1];  // refine_rows
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    RowSums<Real> R{reinterpret_cast<uint32_t*>(smem_raw), P.max_rows};
    if (tid == 0) {
        s_idle = (!kFinal && ldcg(&P.ctl->active) <= 0) ? 1 : 0;  // one reading for the whole CTA
        s_next = s_idle ? P.nrow_tiles : (int32_t)atomicAdd(&P.ctl->queue, 1u);
    }
    if (tid < 6) words[tid] = 0ull;
    __syncthreads();
    int32_t graph = -1;
    auto flush = [&]() {  // threads 0..5
        unsigned long long* a = acc_slot(P, graph, (int32_t)blockIdx.x);
        if (words[tid]) atomicAdd(a + tid, words[tid]);
        words[tid] = 0ull;
    };
    for (;;) {
        const int32_t c = s_next;
        __syncthreads();
        if (c >= P.nrow_tiles) break;
        const int2 rt = __ldg(P.row_tiles + c);
        const GraphDev& G = P.graphs[rt.x];
        GraphState* st = P.states + rt.x;
        if (rt.x != graph) {
            if (graph >= 0 && tid < 6) flush();
            if (tid == 0) W = make_view<kFinal>(G, st, ldcg(&st->iter));
            graph = rt.x;
        }
        if (tid == 0) s_next = (int32_t)atomicAdd(&P.ctl->queue, 1u);
        if (!kFinal && ldcg(&st->done)) {  // a frozen graph: the same for the whole CTA
            __syncthreads();
            continue;
        }
        const int32_t v0 = __ldg(G.row_tile + rt.y), nr = __ldg(G.row_tile + rt.y + 1) - v0;
        const int32_t k1 = __ldg(G.row_step + rt.y + 1);
        int32_t k = __ldg(G.row_step + rt.y) + warp;
        for (int32_t i = tid; i < nr; i += kRowThreads) R.clear(i);
        __syncthreads();  // the sums are clear, the view is set
        [[maybe_unused]] uint32_t lost = 0u;  // 1: a small pair was added, 2: one that left no unit
        const Real* pairs = static_cast<const Real*>(G.pairs) + lane;
        const uint16_t* prow = G.pair_row + lane;
        // a step's pairs are requested before the previous step's are added
        struct Step {
            Real v[kStepPairs / 32];
            uint32_t row[kStepPairs / 32];
            int32_t len;
        };
        int2 sp = k < k1 ? __ldg(G.steps + k) : make_int2(0, 0);
        auto load = [&](Step& f) {
            f.len = sp.y - lane;
#pragma unroll
            for (int j = 0; j < kStepPairs / 32; ++j)
                if (32 * j < f.len) {
                    f.v[j] = __ldcg(pairs + sp.x + 32 * j);
                    f.row[j] = __ldg(prow + sp.x + 32 * j);
                }
            k += kRowWarps;
            sp = k < k1 ? __ldg(G.steps + k) : make_int2(0, 0);
        };
        auto add = [&](const Step& f) {
#pragma unroll
            for (int j = 0; j < kStepPairs / 32; ++j)
                if (32 * j < f.len) {
                    const bool low = R.add((int32_t)f.row[j], f.v[j]);
                    if (kWatch && low && f.v[j] != Real(0)) lost |= f.v[j] < Real(1.0 / kUnit) ? 3u : 1u;
                }
        };
        Step fa, fb;
        load(fa);
        for (int32_t q = k - kRowWarps; q < k1; q += 2 * kRowWarps) {
            load(fb);
            add(fa);
            load(fa);
            add(fb);
        }
        [[maybe_unused]] bool refined = false;
        if constexpr (kWatch) {
            // small sums matter unless every row gets enough besides
            if ((W.personalised ? W.dmass : W.jump) >= kRowFloor<Real>) lost = 0u;
            if (__syncthreads_or(lost != 0u)) {
                const bool gone = __syncthreads_or(lost & 2u);  // else a sum of no units is 0
                bool low = false;
                for (int32_t i = tid; i < nr; i += kRowThreads)
                    low |= R.units(i) < (1ull << kRowBits<Real>) && (gone || R.units(i) != 0ull);
                refined = __syncthreads_or(low);
                if (refined) refine_rows<Real>(R, todo, G, rt.y);
            }
        } else {
            __syncthreads();
        }
        double err = 0.0, dsum = 0.0, xsum = 0.0;
        // three rows of a thread at a time, their loads together (four, or two with the watch,
        // need more registers than two CTAs per SM leave; two without: 1% slower at scale 25)
        constexpr int kRowsAhead = kWatch ? 1 : 3;
        for (int32_t i0 = tid; i0 < nr; i0 += kRowsAhead * kRowThreads) {
            float xin[kRowsAhead];
            double scale[kRowsAhead];
            int32_t rank[kRowsAhead];
#pragma unroll
            for (int j = 0; j < kRowsAhead; ++j) {
                const int32_t i = i0 + j * kRowThreads;
                if (i < nr) {
                    xin[j] = W.xin[v0 + i];
                    scale[j] = kFinal ? 0.0 : W.scale[v0 + i];
                    rank[j] = kFinal ? -1 : __ldg(W.rank + v0 + i);
                }
            }
#pragma unroll
            for (int j = 0; j < kRowsAhead; ++j) {
                const int32_t i = i0 + j * kRowThreads;
                if (i < nr) {
                    const double sum = kWatch && refined ? R.get_double(i) : R.get(i);
                    finish_row<kFinal>(W, v0 + i, sum, xin[j], scale[j], rank[j], err, dsum, xsum);
                }
            }
        }
        err = warp_sum(err);
        dsum = warp_sum(dsum);
        xsum = warp_sum(xsum);
        if (lane == 0) {
            part[warp][0] = err;
            part[warp][1] = dsum;
            part[warp][2] = xsum;
        }
        __syncthreads();
        if (tid < 3) {  // the row tile's sums, in a fixed order
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kRowWarps; ++w) s += part[w][tid];
            fx_add_own(words + 2 * tid, s);
        }
        __syncthreads();
    }
    if (graph >= 0 && tid < 6) flush();
    __threadfence();  // this CTA's accumulator updates before its exit is counted
    __syncthreads();
    if (tid == 0) {
        const uint32_t prev = atomicAdd(&P.ctl->exited, 1u);
        s_last = prev == gridDim.x - 1 ? 1 : 0;
    }
    __syncthreads();
    if (!s_last) return;
    // Last CTA out: every row tile of this sweep is done.
    __threadfence();
    launch_tail<kFinal>(P);
    if (tid == 0) {
        P.ctl->queue = 0u;
        P.ctl->exited = 0u;
        if (!kFinal) {
            const int32_t launches = P.ctl->launches + 1;
            P.ctl->launches = launches;
            const int32_t active = ldcg(&P.ctl->active);
            const bool more = active > 0 && launches < P.ctl->cap && ldcg(&P.ctl->error) == 0;
            if (active > 0 && launches >= P.ctl->cap) P.ctl->error = EGPR_TIMEOUT;
            if (P.use_cond) cudaGraphSetConditional(P.cond, more ? 1u : 0u);
        }
        __threadfence();
    }
}

// ---- per-solve set-up and finishing kernels --------------------------------

// scale = alpha / outw, 0 for a dangling vertex (outw <= 1e-15, pagerank.py:118; with
// alpha = 0, where every scale is 0, the dangling term is 0 too); x0 = 1/n;
// z0 = scale / n, by source rank.
__global__ void k_init_vertices(const GraphDev* graphs, int32_t count, double alpha) {
    const int32_t gi = blockIdx.y;
    if (gi >= count) return;
    const GraphDev G = graphs[gi];
    const double x0 = 1.0 / (double)G.n;
    double* scale = const_cast<double*>(G.scale);
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < G.n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const double o = G.outw[v];
        const double sc = o <= 1e-15 ? 0.0 : alpha / o;
        const int32_t rank = G.rank[v];
        scale[v] = sc;
        G.x[0][v] = (float)x0;
        if (rank >= 0) G.z[0][rank] = (float)(x0 * sc);
    }
}

__global__ void k_init_states(GraphState* states, const GraphDev* graphs, const int32_t* ndang,
                              int32_t count, double alpha, double tol, int32_t max_iter,
                              int32_t personalised) {
    const int32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= count) return;
    const int32_t n = graphs[gi].n;
    const double x0 = (double)(float)(1.0 / (double)n);
    GraphState s;
    s.alpha = alpha;
    s.c1 = (1.0 - alpha) / (double)n;
    s.tol_n = tol * (double)n;
    s.dsum = (double)ndang[gi] * x0;
    s.dmass = alpha * s.dsum / (double)n;
    s.dmass_prev = s.dmass;
    s.residual = 0.0;
    s.residual64 = 0.0;
    s.xsum = 0.0;
    s.iter = 0;
    s.max_iter = max_iter;
    s.done = 0;
    s.converged = 0;
    s.personalised = personalised;
    states[gi] = s;
}

__global__ void k_init_ctl(Ctl* ctl, int32_t active, int32_t cap) {
    Ctl c;
    c.queue = 0u;
    c.exited = 0u;
    c.active = active;
    c.launches = 0;
    c.cap = cap;
    c.error = 0;
    *ctl = c;
}

// FP64 carried values of x_{k-1} for the correction sweep.
__global__ void k_prep_z64(const GraphDev* graphs, const GraphState* states, int32_t count) {
    const int32_t gi = blockIdx.y;
    if (gi >= count) return;
    const GraphDev G = graphs[gi];
    const GraphState* st = states + gi;
    const float* xp = G.x[(st->iter - 1) & 1];
    const double alpha = st->alpha;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < G.n;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int32_t rank = G.rank[u];
        if (rank < 0) continue;
        const double o = G.outw[u];
        G.z64[rank] = o <= 1e-15 ? 0.0 : alpha * (double)xp[u] / o;
    }
}

// Final normalisation (pagerank.py:134-139).  from_fp32: ranks come from the
// last FP32 sweep; otherwise the correction sweep wrote G.out already.
__global__ void k_normalize(const GraphDev* graphs, const GraphState* states, int32_t count,
                            int32_t from_fp32) {
    const int32_t gi = blockIdx.y;
    if (gi >= count) return;
    const GraphDev G = graphs[gi];
    const GraphState* st = states + gi;
    const double norm = st->xsum;
    const float* xl = G.x[st->iter & 1];
    const double inv = norm > 0.0 ? 1.0 / norm : 0.0;
    const double uni = 1.0 / (double)G.n;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < G.n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const double val = from_fp32 ? (double)xl[v] : G.out[v];
        G.out[v] = norm > 0.0 ? val * inv : uni;
    }
}

int cuda_ok(cudaError_t e, const char* what) { return e == cudaSuccess ? EGPR_SUCC : set_cuda_error(e, what); }

// Opts the sweep kernels in to the device's shared memory, once per device.
int smem_optin() {
    static std::atomic<int> cache[64];  // per device; host threads may race to fill it with the same value
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    const int have = cache[dev].load(std::memory_order_acquire);
    if (have > 0) return have;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (optin <= 0) optin = 232448;
    cudaFuncSetAttribute(k_gather<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GatherSmem<float>));
    cudaFuncSetAttribute(k_gather<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GatherSmem<double>));
    constexpr int rows = kMaxTileRows * 2 * (int)sizeof(uint32_t);
    cudaFuncSetAttribute(k_rows<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows);
    cudaFuncSetAttribute(k_rows<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows);
    cudaFuncSetAttribute(k_rows<double, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * rows);
    cudaFuncSetAttribute(k_rows<double, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * rows);
    cudaGetLastError();
    cache[dev].store(optin, std::memory_order_release);
    return optin;
}

size_t gather_smem(bool final) { return final ? sizeof(GatherSmem<double>) : sizeof(GatherSmem<float>); }

size_t row_smem(const Plan& plan, bool final) {
    return (size_t)plan.max_rows * (final ? 4 : 2) * sizeof(uint32_t);
}

SweepParams make_params(Plan& plan, int use_cond) {
    SweepParams P;
    P.units = plan.d_units.as<GatherUnit>();
    P.cta_unit = plan.d_cta_unit.as<int32_t>();
    P.row_tiles = plan.d_row_tiles.as<int2>();
    P.nrow_tiles = plan.nrow_tiles;
    P.max_rows = plan.max_rows;
    P.graphs = plan.d_graphs.as<GraphDev>();
    P.states = plan.d_states.as<GraphState>();
    P.acc = plan.d_acc.as<unsigned long long>();
    P.acc_sub = plan.nacc / std::max(1, plan.ngraphs);
    P.ctl = plan.d_ctl.as<Ctl>();
    P.cond = 0;
    P.use_cond = use_cond;
    P.ngraphs = plan.ngraphs;
    smem_optin();
    return P;
}

int vertex_grid(int32_t max_n) {
    int64_t b = ((int64_t)max_n + kThreads - 1) / kThreads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 8));
}

}  // namespace

// A block is staged in 16-byte units: room for the last block's rounding.
int64_t z_stride(int32_t nsrc) { return ((int64_t)nsrc + 31) & ~(int64_t)31; }

int sweep_resident_warps() { return sweep_grid() * kGatherWarps<float>; }

// CTAs of the sweep's first phase and of the batched solve over `entries` inbound
// entries: one per EGPR_CTA_ENTRIES entries (default 32768), at most `full`.  A small
// graph then holds a few SMs instead of all of them, so solves of other graphs on
// other streams run beside it (0: always the full grid).  The second phase takes a CTA
// per row tile, two per SM at most: its CTAs wait for nothing and leave after a few
// microseconds.  Eight threads solving graphs of 0.8 M and 2 M entries: 6,083 and 3,619
// solves/s, 4,798 and 2,497 with the single-phase sweep.
int work_grid(int64_t entries, int full) {
    static const int64_t per = [] {
        const char* e = std::getenv("EGPR_CTA_ENTRIES");
        const long long x = e ? std::atoll(e) : 32768;
        return (int64_t)(x >= 0 ? x : 32768);
    }();
    if (per == 0) return std::max(1, full);
    const int64_t want = (entries + per - 1) / per;
    return (int)std::max<int64_t>(1, std::min<int64_t>(want, full));
}

// One persistent CTA per SM.
int sweep_grid() {
    static std::atomic<int> cache[64];  // per device; host threads may race to fill it with the same value
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    const int have = cache[dev].load(std::memory_order_acquire);
    if (have > 0) return have;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaGetLastError();
    const int grid = std::max(1, sms);
    cache[dev].store(grid, std::memory_order_release);
    return grid;
}

GraphDev graph_dev_view(const egpr_graph* g) {
    GraphDev d;
    d.idx = g->global_block ? nullptr : g->idx.as<uint16_t>();
    d.idx32 = g->global_block ? g->idx.as<int32_t>() : nullptr;
    d.w = g->weighted ? g->sw_w.as<float>() : nullptr;
    d.tile_bits = g->tile_bits.as<uint32_t>();
    d.tile_pair = g->tile_pair.as<int32_t>();
    d.pair_row = g->pair_row.as<uint16_t>();
    d.row_step = g->row_step.as<int32_t>();
    d.steps = g->steps.as<int2>();
    d.row_tile = g->row_tile.as<int32_t>();
    d.pairs = g->pairs.p;
    d.outw = g->outw.as<double>();
    d.rank = g->rank.as<int32_t>();
    d.scale = g->scale.as<double>();
    d.tele = g->tele.as<float>();
    d.x[0] = g->x0.as<float>();
    d.x[1] = g->x1.as<float>();
    d.z[0] = g->z0.as<float>();
    d.z[1] = g->z0.as<float>() + z_stride(g->nsrc);
    d.out = g->out.as<double>();
    d.z64 = g->z64.as<double>();
    d.n = g->n;
    d.nsrc = g->nsrc;
    d.nblocks = g->nblocks;
    d.chunk_shift = g->chunk_shift;
    return d;
}

int plan_build(Plan& plan, egpr_graph* const* graphs, int32_t count, cudaStream_t stream) {
    plan.release();
    std::vector<GraphDev> views((size_t)count);
    std::vector<int32_t> ndang((size_t)count);
    int32_t max_n = 0, max_rows = kRowGroup;
    int64_t entries = 0, nrt = 0;
    std::vector<CutGraph> cuts((size_t)count);
    for (int32_t gi = 0; gi < count; ++gi) {
        const egpr_graph* g = graphs[gi];
        views[(size_t)gi] = graph_dev_view(g);
        ndang[(size_t)gi] = g->n_dangling_solve;
        max_n = std::max(max_n, g->n);
        entries += g->nnz;
        nrt += g->nrow_tiles;
        max_rows = std::max(max_rows, g->max_tile_rows);
        cuts[(size_t)gi] = CutGraph{g->h_block_tile.data(), g->h_block_pair.data(), g->nblocks, g->chunk_shift, g->tune_rc};
    }
    if (nrt > INT32_MAX / 2) return EGPR_UNSUPPORTED_GRAPH;
    plan.ngraphs = count;
    plan.max_n = max_n;
    plan.max_rows = max_rows;
    plan.nrow_tiles = (int32_t)nrt;
    plan.grid = work_grid(entries, sweep_grid());
    // phase 1
    std::vector<GatherUnit> units;
    std::vector<int32_t> cta_unit;
    cut_gather_units(cuts.data(), count, plan.grid, units, cta_unit);
    if (units.empty()) units.push_back(GatherUnit{0, 0, 0, 0});
    // phase 2: row tiles in row order (their costs are about equal)
    std::vector<int2> order;
    order.reserve((size_t)std::max<int64_t>(nrt, 1));
    for (int32_t gi = 0; gi < count; ++gi)
        for (int32_t q = 0; q < graphs[gi]->nrow_tiles; ++q) order.push_back(make_int2(gi, q));
    if (order.empty()) order.push_back(make_int2(0, 0));
    smem_optin();
    plan.row_grid = (int)std::max<int64_t>(1, std::min<int64_t>(nrt, (int64_t)sweep_grid() * kRowTilesPerSm));
    // accumulator slots: 64 per graph (few for the launch's last CTA to read,
    // enough that concurrent warps rarely add to the same address), fewer
    // for many graphs
    const int32_t per_graph = std::max(1, std::min(64, 8192 / std::max(1, count)));
    plan.nacc = per_graph * count;
    int rc;
    if ((rc = plan.d_units.alloc(units.size() * sizeof(GatherUnit))) ||
        (rc = plan.d_cta_unit.alloc(cta_unit.size() * sizeof(int32_t))) ||
        (rc = plan.d_row_tiles.alloc(order.size() * sizeof(int2))) ||
        (rc = plan.d_graphs.alloc(views.size() * sizeof(GraphDev))) ||
        (rc = plan.d_states.alloc((size_t)count * sizeof(GraphState))) ||
        (rc = plan.d_ndang.alloc((size_t)count * sizeof(int32_t))) ||
        (rc = plan.d_acc.alloc((size_t)plan.nacc * kAccWords * sizeof(unsigned long long))) ||
        (rc = plan.d_ctl.alloc(sizeof(Ctl))))
        return rc;
    if ((rc = cuda_ok(cudaMemcpyAsync(plan.d_units.p, units.data(), units.size() * sizeof(GatherUnit), cudaMemcpyHostToDevice, stream), "H2D units")) ||
        (rc = cuda_ok(cudaMemcpyAsync(plan.d_cta_unit.p, cta_unit.data(), cta_unit.size() * sizeof(int32_t), cudaMemcpyHostToDevice, stream), "H2D units")) ||
        (rc = cuda_ok(cudaMemcpyAsync(plan.d_row_tiles.p, order.data(), order.size() * sizeof(int2), cudaMemcpyHostToDevice, stream), "H2D row tiles")) ||
        (rc = cuda_ok(cudaMemcpyAsync(plan.d_graphs.p, views.data(), views.size() * sizeof(GraphDev), cudaMemcpyHostToDevice, stream), "H2D graph table")) ||
        (rc = cuda_ok(cudaMemcpyAsync(plan.d_ndang.p, ndang.data(), ndang.size() * sizeof(int32_t), cudaMemcpyHostToDevice, stream), "H2D counts")) ||
        (rc = cuda_ok(cudaStreamSynchronize(stream), "plan upload")))
        return rc;
    return EGPR_SUCC;
}

// The sweeps as a CUDA graph: a while node whose body is the two phases.
static int plan_capture_loop(Plan& plan, bool watch) {
    Plan::Loop& L = plan.loops[watch];
    if (L.exec) return EGPR_SUCC;
    if (L.failed) return EGPR_DEVICE_ERR;
    cudaGraph_t cg = nullptr;
    cudaGraphExec_t ex = nullptr;
    cudaGraphConditionalHandle h = 0;
    cudaGraphNode_t cnode = nullptr, gnode = nullptr, rnode = nullptr;
    cudaGraphNodeParams cp = {};
    cudaKernelNodeParams kp = {};
    SweepParams P;
    void* args[1];
    cudaError_t e = cudaGraphCreate(&cg, 0);
    if (e != cudaSuccess) goto fail;
    e = cudaGraphConditionalHandleCreate(&h, cg, 1u, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) goto fail;
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    e = cudaGraphAddNode(&cnode, cg, nullptr, 0, &cp);
    if (e != cudaSuccess) goto fail;
    P = make_params(plan, 1);
    P.cond = h;
    args[0] = &P;
    kp.func = (void*)k_gather<float>;
    kp.gridDim = dim3((unsigned)plan.grid);
    kp.blockDim = dim3(32 * kGatherWarps<float>);
    kp.sharedMemBytes = (unsigned)gather_smem(false);
    kp.kernelParams = args;
    e = cudaGraphAddKernelNode(&gnode, cp.conditional.phGraph_out[0], nullptr, 0, &kp);
    if (e != cudaSuccess) goto fail;
    kp.func = watch ? (void*)k_rows<float, true> : (void*)k_rows<float, false>;
    kp.gridDim = dim3((unsigned)plan.row_grid);
    kp.blockDim = dim3(kRowThreads);
    kp.sharedMemBytes = (unsigned)row_smem(plan, false);
    e = cudaGraphAddKernelNode(&rnode, cp.conditional.phGraph_out[0], &gnode, 1, &kp);
    if (e != cudaSuccess) goto fail;
    e = cudaGraphInstantiate(&ex, cg, 0);
    if (e != cudaSuccess) goto fail;
    L.graph = cg;
    L.exec = ex;
    return EGPR_SUCC;
fail:
    cudaGetLastError();
    if (cg) cudaGraphDestroy(cg);
    L.failed = true;
    return EGPR_DEVICE_ERR;
}

int launch_init(Plan& plan, double alpha, int32_t max_iter, double tol, bool personalised,
                cudaStream_t stream) {
    dim3 grid((unsigned)vertex_grid(plan.max_n), (unsigned)plan.ngraphs);
    k_init_vertices<<<grid, kThreads, 0, stream>>>(plan.d_graphs.as<GraphDev>(), plan.ngraphs, alpha);
    k_init_states<<<(plan.ngraphs + 127) / 128, 128, 0, stream>>>(plan.d_states.as<GraphState>(),
                                                                 plan.d_graphs.as<GraphDev>(),
                                                                 plan.d_ndang.as<int32_t>(), plan.ngraphs,
                                                                 alpha, tol, max_iter, personalised ? 1 : 0);
    k_init_ctl<<<1, 1, 0, stream>>>(plan.d_ctl.as<Ctl>(), plan.ngraphs, max_iter + 1);
    cudaMemsetAsync(plan.d_acc.p, 0, plan.d_acc.bytes, stream);
    return cuda_ok(cudaGetLastError(), "init launch");
}

bool rows_need_watch(const Plan& plan, double alpha, bool personalised) {
    return personalised || !((1.0 - alpha) / (double)plan.max_n >= kRowFloor<float>);
}

int launch_loop(Plan& plan, int32_t max_iter, bool watch, cudaStream_t stream, int32_t* launches) {
    *launches = -1;  // counted on the device (Ctl::launches, sweeps)
    if (graph_loop_enabled() && plan_capture_loop(plan, watch) == EGPR_SUCC)
        return cuda_ok(cudaGraphLaunch(plan.loops[watch].exec, stream), "graph launch");
    // Plain launches; a sweep with no active graph returns at once.
    SweepParams P = make_params(plan, 0);
    for (int32_t it = 0; it < max_iter; ++it) {
        k_gather<float><<<plan.grid, 32 * kGatherWarps<float>, gather_smem(false), stream>>>(P);
        if (watch) k_rows<float, true><<<plan.row_grid, kRowThreads, row_smem(plan, false), stream>>>(P);
        else k_rows<float, false><<<plan.row_grid, kRowThreads, row_smem(plan, false), stream>>>(P);
    }
    return cuda_ok(cudaGetLastError(), "sweep launch");
}

int launch_finish(Plan& plan, bool correction, bool watch, cudaStream_t stream, int32_t* launches) {
    dim3 grid((unsigned)vertex_grid(plan.max_n), (unsigned)plan.ngraphs);
    int32_t l = 0;
    if (correction) {
        k_prep_z64<<<grid, kThreads, 0, stream>>>(plan.d_graphs.as<GraphDev>(), plan.d_states.as<GraphState>(),
                                                  plan.ngraphs);
        // The loop's last CTA left the queue reset; the control block keeps the sweep count.
        SweepParams P = make_params(plan, 0);
        k_gather<double><<<plan.grid, 32 * kGatherWarps<double>, gather_smem(true), stream>>>(P);
        if (watch) k_rows<double, true><<<plan.row_grid, kRowThreads, row_smem(plan, true), stream>>>(P);
        else k_rows<double, false><<<plan.row_grid, kRowThreads, row_smem(plan, true), stream>>>(P);
        l += 3;
    }
    k_normalize<<<grid, kThreads, 0, stream>>>(plan.d_graphs.as<GraphDev>(), plan.d_states.as<GraphState>(),
                                               plan.ngraphs, correction ? 0 : 1);
    l += 1;
    *launches = l;
    return cuda_ok(cudaGetLastError(), "finish launch");
}

}  // namespace egpr
