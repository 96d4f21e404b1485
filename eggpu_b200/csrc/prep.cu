// Device-side graph preparation.
//
// Replaces the reference's single-threaded host pass build_inbound_from_csr
// (gpu_easygraph/functions/centrality/pagerank.cu:286-347) and its H2D of the
// result (:472-518) with GPU kernels over the uploaded out-edge CSR:
//
//   k_out_weight_exact  FP64 out-weight sum per source after sanitising each
//                    weight, bit-identical to the sequential sum in row order
//                    (pagerank.cu:301-316): four lanes per source (a warp for
//                    sources of more than 64 entries, 4096-entry segments on
//                    several warps for more than 16384) where the sum is
//                    provably order-free, one thread per source otherwise
//   k_in_degree      in-degree histogram over valid endpoints (:315)
//   exclusive scan   in_row (:319-320)
//   radix sort       stable LSD sort of the entries by destination: entries of
//                    one destination keep ascending entry order, i.e. the
//                    ascending-source order of the reference's sequential
//                    scatter (:328-346); the sorted pairs carry each entry's
//                    source and, when weighted, its FP32 weight, so the sorted
//                    values are in_col and in_w
//   k_dangling       dangling mask outw <= 0 (:323-326) and the counts used by
//                    the solver
//
// The results are bit-identical to build_inbound_from_csr for in_row, in_col,
// the dangling mask and the FP64 out-weight sums.  The engine stores raw
// (sanitised) FP32 weights instead of the alpha-scaled in_val, so a prepared
// graph does not depend on alpha.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cctype>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "egpr_internal.cuh"

namespace egpr {
namespace {

constexpr int kScanPerThread = 8;
constexpr int kScanTile = kThreads * kScanPerThread;
constexpr int kSortPerLane = 16;
constexpr int kWarps = kThreads / 32;
constexpr int kSortTile = kThreads * kSortPerLane;

// ---------------------------------------------------------------- scan -----
// Exclusive scan of uint32 values, tile by tile; tile totals go to tile_sums.
__global__ void __launch_bounds__(kThreads)
k_scan_tiles(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int64_t len,
             uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t s[kScanTile];
    __shared__ uint32_t warp_tot[kWarps];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    const int tid = threadIdx.x;
#pragma unroll
    for (int i = 0; i < kScanPerThread; ++i) {
        int64_t idx = base + tid + (int64_t)i * kThreads;
        s[tid + i * kThreads] = idx < len ? in[idx] : 0u;
    }
    __syncthreads();
    uint32_t v[kScanPerThread];
    uint32_t run = 0;
#pragma unroll
    for (int i = 0; i < kScanPerThread; ++i) {
        v[i] = run;
        run += s[tid * kScanPerThread + i];
    }
    // inclusive warp scan of the thread totals
    const int lane = tid & 31, warp = tid >> 5;
    uint32_t inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    uint32_t warp_off = 0, block_tot = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        if (w < warp) warp_off += warp_tot[w];
        block_tot += warp_tot[w];
    }
    const uint32_t excl = warp_off + inc - run;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanPerThread; ++i) s[tid * kScanPerThread + i] = v[i] + excl;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanPerThread; ++i) {
        int64_t idx = base + tid + (int64_t)i * kThreads;
        if (idx < len) out[idx] = s[tid + i * kThreads];
    }
    if (tid == 0 && tile_sums) tile_sums[blockIdx.x] = block_tot;
}

__global__ void k_scan_add(uint32_t* __restrict__ out, int64_t len, const uint32_t* __restrict__ tile_off) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < len) out[i] += tile_off[i / kScanTile];
}

// -------------------------------------------------------------- radix ------
// LSD radix sort of (key, value) pairs with digits of kBits bits (8 to 10).
template <int kBits>
__global__ void __launch_bounds__(kThreads)
k_radix_hist(const uint32_t* __restrict__ keys, int64_t len, int shift, int64_t ntiles,
             uint32_t* __restrict__ hist) {
    constexpr int kD = 1 << kBits;
    __shared__ uint32_t h[kD];
    for (int d = threadIdx.x; d < kD; d += kThreads) h[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    for (int i = threadIdx.x; i < kSortTile; i += kThreads) {
        int64_t idx = base + i;
        if (idx < len) atomicAdd(&h[(keys[idx] >> shift) & (kD - 1)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kD; d += kThreads) hist[(int64_t)d * ntiles + blockIdx.x] = h[d];
}

// Stable scatter: within a tile, warp w owns items [w*32*kSortPerLane, ...) in
// order; inside a warp, rounds of 32 consecutive items rank equal digits by
// lane order.  Global order = tile order (digit-major scanned histogram),
// then warp order, then item order.  keys_out may be NULL (last pass: only
// the values are needed).  kTwo: a second value array moves with the first.
// The arrays go through one staging buffer in turn, and a value is loaded when its turn
// comes, so four CTAs fit an SM (three with a buffer per array); every thread scans its
// digits.  Preparation of R-MAT scale 25 weighted, page-locked input: 173 -> 159 ms with
// the single 10-bit pass, scale 22 11.2 -> 10.2 ms.
template <int kBits>
struct RadixSmem {
    static constexpr int kD = 1 << kBits;
    uint32_t stage[kSortTile];    // the tile in digit order, one array at a time
    uint32_t out[kD];             // where the digit's first item of the tile goes, minus its place in the tile
    uint16_t hist[kWarps][kD];    // per warp: count of the digit, then the place of its first item in the tile
    uint32_t warp_tot[kWarps];
};

template <int kBits, bool kTwo>
__global__ void __launch_bounds__(kThreads, 4)
k_radix_scatter(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int64_t len,
                int shift, int64_t ntiles, const uint32_t* __restrict__ offsets,
                const uint32_t* __restrict__ vals2_in, uint32_t* __restrict__ vals2_out) {
    constexpr int kD = 1 << kBits, kOwn = kD / kThreads;  // digits of a thread in the tile's scan
    extern __shared__ __align__(16) unsigned char radix_smem[];
    RadixSmem<kBits>& S = *reinterpret_cast<RadixSmem<kBits>*>(radix_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kWarps * kD / 2; i += kThreads) reinterpret_cast<uint32_t*>(&S.hist[0][0])[i] = 0u;
    const int64_t wbase = (int64_t)blockIdx.x * kSortTile + (int64_t)warp * 32 * kSortPerLane;
    uint32_t key[kSortPerLane], place[kSortPerLane];
#pragma unroll
    for (int r = 0; r < kSortPerLane; ++r) {
        const int64_t idx = wbase + (int64_t)r * 32 + lane;
        key[r] = idx < len ? keys_in[idx] : 0u;
    }
    __syncthreads();
    const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < kSortPerLane; ++r) {
        const bool valid = wbase + (int64_t)r * 32 + lane < len;
        const uint32_t d = (key[r] >> shift) & (kD - 1);
        const uint32_t tag = valid ? d : (uint32_t)(kD + lane);
        const uint32_t peers = __match_any_sync(0xffffffffu, tag);
        const uint32_t before = valid ? S.hist[warp][d] : 0u;
        __syncwarp();
        if (valid && (peers & lt_mask) == 0u) S.hist[warp][d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        place[r] = before + __popc(peers & lt_mask);
    }
    __syncthreads();
    // the tile's counts per digit, scanned: each thread a run of digits
    uint32_t cnt[kOwn], run = 0;
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
        cnt[k] = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) cnt[k] += S.hist[w][tid * kOwn + k];
        run += cnt[k];
    }
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) S.warp_tot[warp] = incl;
    __syncthreads();
    uint32_t at = incl - run;  // of the thread's first digit
    for (int w = 0; w < warp; ++w) at += S.warp_tot[w];
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
        const int d = tid * kOwn + k;
        S.out[d] = offsets[(int64_t)d * ntiles + blockIdx.x] - at;
        uint32_t p = at;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = S.hist[w][d];
            S.hist[w][d] = (uint16_t)p;
            p += c;
        }
        at += cnt[k];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortPerLane; ++r) {
        if (wbase + (int64_t)r * 32 + lane < len) {
            place[r] += S.hist[warp][(key[r] >> shift) & (kD - 1)];
            S.stage[place[r]] = key[r];
        }
    }
    __syncthreads();
    // item i of the tile in digit order goes to dst: each digit's run is contiguous
    const int64_t tbase = (int64_t)blockIdx.x * kSortTile;
    const int nvalid = (int)(len - tbase < (int64_t)kSortTile ? len - tbase : (int64_t)kSortTile);
    uint32_t dst[kSortPerLane];
#pragma unroll
    for (int r = 0; r < kSortPerLane; ++r) {
        const int i = tid + r * kThreads;
        if (i < nvalid) {
            const uint32_t k = S.stage[i];
            dst[r] = S.out[(k >> shift) & (kD - 1)] + (uint32_t)i;
            if (keys_out) keys_out[dst[r]] = k;
        }
    }
    auto move = [&](const uint32_t* __restrict__ in, uint32_t* __restrict__ out) {
        uint32_t v[kSortPerLane];
#pragma unroll
        for (int r = 0; r < kSortPerLane; ++r) {
            const int64_t idx = wbase + (int64_t)r * 32 + lane;
            v[r] = idx < len ? in[idx] : 0u;
        }
        __syncthreads();  // the array before is read
#pragma unroll
        for (int r = 0; r < kSortPerLane; ++r)
            if (wbase + (int64_t)r * 32 + lane < len) S.stage[place[r]] = v[r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortPerLane; ++r) {
            const int i = tid + r * kThreads;
            if (i < nvalid) out[dst[r]] = S.stage[i];
        }
    };
    move(vals_in, vals_out);
    if (kTwo) move(vals2_in, vals2_out);
}

// -------------------------------------------------------------- graph ------
__device__ __forceinline__ double sanitize_w(double w) {
    return (!isfinite(w) || w < 0.0) ? 0.0 : w;
}

// Exponent of the lowest set bit of a finite w > 0: w = M * 2^q with M odd.
__device__ __forceinline__ int lsb_exponent(double w) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(w);
    const int ef = (int)((b >> 52) & 0x7ffull);
    unsigned long long m = b & 0xfffffffffffffull;
    int e = -1074;  // subnormal: w = m * 2^-1074
    if (ef != 0) {
        m |= 1ull << 52;
        e = ef - 1075;
    }
    return e + __ffsll((long long)m) - 1;
}

// Ranking key of a source with c valid out-edges: descending classes of an
// eighth of an octave, 255 for none.  Classes instead of exact degrees: one
// 8-bit sort pass ranks the vertices, and inside a class the order stays that
// of the vertices, so neighbouring rows of similar degree have neighbouring
// ranks and their carried values are written in few sectors.
constexpr uint32_t kNoRank = 255u;
__device__ __forceinline__ uint32_t rank_class(int32_t c) {
    if (c <= 0) return kNoRank;
    const int e = 31 - __clz(c);                                       // octave
    const int f = e >= 3 ? (c >> (e - 3)) & 7 : (c << (3 - e)) & 7;    // eighth of it
    return (uint32_t)(254 - (8 * e + f));                              // 8 * 30 + 7 at most
}

// FP64 out-weight sums, one warp per source, bit-identical to the sequential
// sum in entry order (pagerank.cu:301-316) without summing sequentially.
// Sanitised weights are >= 0; let 2^q be the lowest set bit among a row's
// nonzero weights.  Every partial sum, in any order, is then a multiple of
// 2^q no larger than the row's total T, so when T < 2^(q+53) every partial sum
// is an exact double and the lanes' sums and the shuffle tree give T, which
// is also what the sequential loop gives.  The computed sum s is within a few
// ulps of T, so s < 2^(q+52) proves T < 2^(q+53).  A row that fails the test
// (weights of very different scales) is listed and summed sequentially by
// k_out_weight_serial.  Weights drawn as FP32 values, as in the synthetic
// workloads, always pass.
// One source's sums over G lanes (lanes sub = 0..G-1 of a G-lane group).
template <int G>
__device__ __forceinline__ void out_weight_row(const int32_t* __restrict__ E, const double* __restrict__ W,
                                               int32_t n, int32_t b, int32_t e, int sub, double& s, int32_t& c,
                                               int& q) {
    s = 0.0;
    c = 0;
    q = 4096;  // no nonzero weight yet
    for (int32_t p = b + sub; p < e; p += G) {
        const int32_t v = E[p];
        if (v >= 0 && v < n) {
            const double w = W ? sanitize_w(W[p]) : 1.0;  // unit weights: q = 0, every sum exact
            s += w;
            ++c;
            if (w > 0.0) q = min(q, lsb_exponent(w));
        }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
        q = min(q, __shfl_xor_sync(0xffffffffu, q, o));
    }
}

// The sum s of a source's weights is its sequential sum when every partial sum
// is provably exact (see above); otherwise the source is listed for the
// sequential kernel.
__device__ __forceinline__ void out_weight_store(int64_t u, double s, int32_t c, int q, double* __restrict__ outw,
                                                 uint32_t* __restrict__ rank_key, uint32_t* __restrict__ rank_val,
                                                 int32_t* __restrict__ serial_rows,
                                                 uint32_t* __restrict__ serial_count) {
    bool exact;
    if (q == 4096) exact = true;             // only zero weights: the sum is 0
    else if (q + 52 >= 1024) exact = false;  // 2^(q+52) would overflow: sum sequentially
    else exact = s < ldexp(1.0, q + 52);
    if (exact) outw[u] = s;
    else serial_rows[atomicAdd(serial_count, 1u)] = (int32_t)u;
    rank_key[u] = rank_class(c);
    rank_val[u] = (uint32_t)u;
}

constexpr int32_t kOutWeightShort = 64;  // sources with more entries are summed by a whole warp
// Sources with more than kOutWeightHuge entries are summed in segments of
// kOutWeightSeg entries by several warps; each segment's sums go into the
// source's accumulator and the last segment to arrive finishes the source.
// A segment's sum is one of the source's partial sums, so the exactness test
// above covers the segments and their FP64 atomic adds, in any order.
constexpr int32_t kOutWeightHuge = 16384;
constexpr int32_t kOutWeightSeg = 4096;

struct HugeAcc {
    double s;          // sum of the segments' sums
    int32_t c;         // valid entries
    int32_t q;         // lowest set bit exponent of the nonzero weights
    uint32_t arrived;  // segments added so far
    int32_t pad;
};

struct OutSegs {
    int4* seg;           // (source, segment, accumulator, segments of the source)
    uint32_t* seg_count;
    HugeAcc* acc;
    uint32_t* acc_count;
};

// Lists the segments of source u (called by one thread for a huge source).
__device__ __forceinline__ void list_segments(const OutSegs& H, int32_t u, int32_t len) {
    const int32_t nseg = (len + kOutWeightSeg - 1) / kOutWeightSeg;
    const uint32_t h = atomicAdd(H.acc_count, 1u);
    H.acc[h].s = 0.0;
    H.acc[h].c = 0;
    H.acc[h].q = 4096;
    H.acc[h].arrived = 0u;
    const uint32_t s0 = atomicAdd(H.seg_count, (uint32_t)nseg);
    for (int32_t j = 0; j < nseg; ++j) H.seg[s0 + (uint32_t)j] = make_int4(u, j, (int32_t)h, nseg);
}

// Sources [r0, r1), four lanes each; a source with more than kOutWeightShort
// entries is listed for k_out_weight_long instead.
__global__ void k_out_weight_exact(const int32_t* __restrict__ V, const int32_t* __restrict__ E,
                                   const double* __restrict__ W, int32_t n, int32_t r0, int32_t r1,
                                   double* __restrict__ outw, uint32_t* __restrict__ rank_key,
                                   uint32_t* __restrict__ rank_val, int32_t* __restrict__ serial_rows,
                                   uint32_t* __restrict__ serial_count, int32_t* __restrict__ long_rows,
                                   uint32_t* __restrict__ long_count, OutSegs H) {
    constexpr int G = 4;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), grp = lane / G;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t ub = r0 + warp * (32 / G); ub < r1; ub += nwarps * (32 / G)) {
        const int64_t u = ub + grp;
        int32_t b = 0, e = 0;
        if (u < r1) {
            b = V[u];
            e = V[u + 1];
            if (e - b > kOutWeightShort) {
                if (sub == 0) {
                    if (e - b > kOutWeightHuge) list_segments(H, (int32_t)u, e - b);
                    else long_rows[atomicAdd(long_count, 1u)] = (int32_t)u;
                }
                e = b;  // the group still takes part in the shuffles
            }
        }
        double s;
        int32_t c;
        int q;
        out_weight_row<G>(E, W, n, b, e, sub, s, c, q);
        if (u < r1 && sub == 0 && V[u + 1] - V[u] <= kOutWeightShort)
            out_weight_store(u, s, c, q, outw, rank_key, rank_val, serial_rows, serial_count);
    }
}

// The long sources listed by k_out_weight_exact, one warp each, then the
// segments of the huge ones (weighted or not).
__global__ void k_out_weight_long(const int32_t* __restrict__ V, const int32_t* __restrict__ E,
                                  const double* __restrict__ W, int32_t n, const int32_t* __restrict__ long_rows,
                                  const uint32_t* __restrict__ long_count, double* __restrict__ outw,
                                  uint32_t* __restrict__ rank_key, uint32_t* __restrict__ rank_val,
                                  int32_t* __restrict__ serial_rows, uint32_t* __restrict__ serial_count,
                                  OutSegs H) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const uint32_t k = long_count ? *long_count : 0u;
    for (int64_t i = warp; i < (int64_t)k; i += nwarps) {
        const int32_t u = long_rows[i];
        double s;
        int32_t c;
        int q;
        out_weight_row<32>(E, W, n, V[u], V[u + 1], lane, s, c, q);
        if (lane == 0) out_weight_store(u, s, c, q, outw, rank_key, rank_val, serial_rows, serial_count);
    }
    // segments of the huge sources: the last segment of a source to arrive finishes it
    const uint32_t ns = *H.seg_count;
    for (int64_t i = warp; i < (int64_t)ns; i += nwarps) {
        const int4 sg = H.seg[i];
        const int32_t u = sg.x, b = V[u] + sg.y * kOutWeightSeg, e = min(V[u + 1], b + kOutWeightSeg);
        double s;
        int32_t c;
        int q;
        out_weight_row<32>(E, W, n, b, e, lane, s, c, q);
        if (lane == 0) {
            HugeAcc& A = H.acc[sg.z];
            if (s != 0.0) atomicAdd(&A.s, s);
            atomicAdd(&A.c, c);
            atomicMin(&A.q, q);
            __threadfence();
            if (atomicAdd(&A.arrived, 1u) == (uint32_t)(sg.w - 1)) {
                __threadfence();
                const double ts = __ldcg(&A.s);
                const int32_t tc = __ldcg(&A.c);
                const int tq = __ldcg(&A.q);
                if (W) {
                    out_weight_store(u, ts, tc, tq, outw, rank_key, rank_val, serial_rows, serial_count);
                } else {  // unit weights: the count
                    outw[u] = (double)tc;
                    rank_key[u] = rank_class(tc);
                    rank_val[u] = (uint32_t)u;
                }
            }
        }
    }
}

// The rows k_out_weight_exact could not prove order-free: summed in entry
// order, one thread per row, exactly as pagerank.cu:301-316 does.
__global__ void k_out_weight_serial(const int32_t* __restrict__ V, const int32_t* __restrict__ E,
                                    const double* __restrict__ W, int32_t n, const int32_t* __restrict__ rows,
                                    const uint32_t* __restrict__ count, double* __restrict__ outw) {
    const uint32_t k = *count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) {
        const int32_t u = rows[i];
        double s = 0.0;
        for (int32_t p = V[u]; p < V[u + 1]; ++p) {
            const int32_t v = E[p];
            if (v >= 0 && v < n) s += sanitize_w(W[p]);
        }
        outw[u] = s;
    }
}

// Unit weights: the out-weight sum is the count of valid entries, exact in any
// order, so one warp counts a row.
__global__ void k_out_degree(const int32_t* __restrict__ V, const int32_t* __restrict__ E, int32_t n, int32_t r0,
                             int32_t r1, double* __restrict__ outw, uint32_t* __restrict__ rank_key,
                             uint32_t* __restrict__ rank_val, OutSegs H) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t u = r0 + warp; u < r1; u += nwarps) {
        const int32_t b = V[u], e = V[u + 1];
        if (e - b > kOutWeightHuge) {  // counted in segments by k_out_weight_long
            if (lane == 0) list_segments(H, (int32_t)u, e - b);
            continue;
        }
        int32_t c = 0;
        for (int32_t p = b + lane; p < e; p += 32) {
            const int32_t v = E[p];
            c += (v >= 0 && v < n) ? 1 : 0;
        }
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (lane == 0) {
            outw[u] = (double)c;
            rank_key[u] = rank_class(c);
            rank_val[u] = (uint32_t)u;
        }
    }
}

// rank[v] = position of v in the ranking (ranked[0 .. n)), -1 for a vertex
// without valid out-edges (they come last).
__global__ void k_ranks(const uint32_t* __restrict__ ranked, int32_t n, int32_t nsrc, int32_t* __restrict__ rank) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        rank[ranked[i]] = i < nsrc ? (int32_t)i : -1;
}

// In-degree histogram and the sort keys: destination, or n for an entry whose
// destination is outside [0, n) (those sort last and are dropped).
__global__ void k_in_degree_keys(const int32_t* __restrict__ E, int64_t p0, int64_t p1, int32_t n,
                                 uint32_t* __restrict__ indeg, uint32_t* __restrict__ keys) {
    for (int64_t p = p0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < p1;
         p += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = E[p];
        const bool ok = v >= 0 && v < n;
        if (ok) atomicAdd(&indeg[v], 1u);
        keys[p] = ok ? (uint32_t)v : (uint32_t)n;
    }
}

// Source id of every entry: one warp per row writes its range.
__global__ void k_expand_src(const int32_t* __restrict__ V, int32_t n, int32_t* __restrict__ src) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t u = warp; u < n; u += nwarps) {
        const int32_t b = V[u], e = V[u + 1];
        for (int32_t p = b + lane; p < e; p += 32) src[p] = (int32_t)u;
    }
}

// FP32 bits of each entry's sanitised weight (the stored in_w), for entries [p0, p1).
__global__ void k_weight_bits(const double* __restrict__ W, int64_t p0, int64_t p1, uint32_t* __restrict__ out) {
    for (int64_t p = p0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < p1;
         p += (int64_t)gridDim.x * blockDim.x)
        out[p] = __float_as_uint((float)sanitize_w(W[p]));
}

// Dangling mask, and the counts of vertices with out-weight <= 0, with out-weight
// <= 1e-15 and with a rank (valid out-edges).
__global__ void k_dangling(const double* __restrict__ outw, const uint32_t* __restrict__ rank_key, int32_t n,
                           int32_t* __restrict__ mask, unsigned long long* __restrict__ counts) {
    __shared__ unsigned long long c0, c1, c2;
    if (threadIdx.x == 0) { c0 = 0; c1 = 0; c2 = 0; }
    __syncthreads();
    unsigned long long a = 0, b = 0, c = 0;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n;
         u += (int64_t)gridDim.x * blockDim.x) {
        const double w = outw[u];
        const int d = w <= 0.0 ? 1 : 0;
        mask[u] = d;
        a += d;
        b += (w <= 1e-15) ? 1 : 0;
        c += rank_key[u] != kNoRank ? 1 : 0;
    }
    // warp sums first: one shared atomic per warp and count
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&c0, a);
        atomicAdd(&c1, b);
        atomicAdd(&c2, c);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&counts[0], c0);
        atomicAdd(&counts[1], c1);
        atomicAdd(&counts[2], c2);
    }
}

inline int grid_for(int64_t work, int per_block = kThreads) {
    int64_t g = (work + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > 148 * 32) g = 148 * 32;
    return (int)g;
}

int cuda_ok(cudaError_t e, const char* what) { return e == cudaSuccess ? EGPR_SUCC : set_cuda_error(e, what); }

// Stream-ordered scratch of the preparation comes from the library's device
// pool (device_pool), which keeps freed memory for the next preparation.
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
    cudaMemPool_t pool = device_pool();
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

struct TmpAlloc {
    cudaStream_t s;
    std::vector<void*> ptrs;
    explicit TmpAlloc(cudaStream_t st) : s(st) {}
    ~TmpAlloc() {
        for (void* p : ptrs) cudaFreeAsync(p, s);
    }
    template <typename T>
    T* get(size_t count, int* rc) {
        void* p = nullptr;
        cudaError_t e = scratch_alloc(&p, std::max<size_t>(count, 1) * sizeof(T), s);
        if (e != cudaSuccess) {
            set_cuda_error(e, "cudaMallocAsync (preparation scratch)");
            *rc = EGPR_FAILED_TO_ALLOCATE_DEVICE_MEM;
            return nullptr;
        }
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
};

template <int kBits, bool kTwo>
int radix_pass(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, int64_t len, int shift,
               bool last, int64_t ntiles, uint32_t* hist, cudaStream_t s, const uint32_t* v2in, uint32_t* v2out) {
    constexpr int kD = 1 << kBits;
    const size_t smem = sizeof(RadixSmem<kBits>);
    // The shared-memory opt-in is a per-device attribute of the function: made
    // once per device (bit d of the mask; devices past 63 repeat it, which is
    // harmless).  Atomic: several host threads prepare graphs at once.
    static std::atomic<uint64_t> attr_devices{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    const uint64_t bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
    if (!bit || !(attr_devices.load(std::memory_order_acquire) & bit)) {
        cudaFuncSetAttribute(k_radix_scatter<kBits, kTwo>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        attr_devices.fetch_or(bit, std::memory_order_release);
    }
    k_radix_hist<kBits><<<(unsigned)ntiles, kThreads, 0, s>>>(kin, len, shift, ntiles, hist);
    int rc = exclusive_scan_u32(hist, hist, ntiles * kD, s);
    if (rc) return rc;
    k_radix_scatter<kBits, kTwo><<<(unsigned)ntiles, kThreads, smem, s>>>(kin, vin, last ? nullptr : kout, vout, len,
                                                                          shift, ntiles, hist, v2in, v2out);
    return EGPR_SUCC;
}

template <int kBits>
int radix_pass_any(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, int64_t len, int shift,
                   bool last, int64_t ntiles, uint32_t* hist, cudaStream_t s, const uint32_t* v2in, uint32_t* v2out) {
    return v2in ? radix_pass<kBits, true>(kin, vin, kout, vout, len, shift, last, ntiles, hist, s, v2in, v2out)
                : radix_pass<kBits, false>(kin, vin, kout, vout, len, shift, last, ntiles, hist, s, nullptr, nullptr);
}

// Sorts (keys, vals) by `bits` bits of the keys from first_bit, stable.  After the
// call the values are in the buffer *result_in_alt names; the keys are sorted
// alongside except in the last pass, which writes values only.
int radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt,
                     int64_t len, int bits, cudaStream_t s, TmpAlloc& tmp, bool* result_in_alt,
                     bool keys_needed = true, uint32_t* vals2 = nullptr, uint32_t* vals2_alt = nullptr,
                     int first_bit = 0) {
    *result_in_alt = false;
    if (len <= 1 || bits <= 0) return EGPR_SUCC;
    int rc = EGPR_SUCC;
    // 8-bit digits: with 4096-item tiles a digit's run averages 16 items, so the
    // runs written out are 64-byte pieces.  Where digits of 9 or 10 bits save a
    // whole pass they are used (25-bit keys: 9 + 8 + 8 instead of 8 + 8 + 8 + 1; the
    // sweep layout's sort by 628 blocks at R-MAT scale 25: one pass of 10).
    int passes = (bits + 7) / 8;
    while (passes > 1 && bits <= 10 * (passes - 1)) --passes;
    const int64_t ntiles = (len + kSortTile - 1) / kSortTile;
    const int widest = std::max(8, (bits + passes - 1) / passes);
    uint32_t* hist = tmp.get<uint32_t>((size_t)ntiles << widest, &rc);
    if (!hist) return rc;
    uint32_t *kin = keys, *vin = vals, *kout = keys_alt, *vout = vals_alt, *v2in = vals2, *v2out = vals2_alt;
    int shift = first_bit;
    for (int p = 0; p < passes; ++p) {
        const bool last = p == passes - 1 && !keys_needed;
        const int left = first_bit + bits - shift;  // the wider digits first
        const int digit = std::max(8, (left + passes - p - 1) / (passes - p));
        rc = digit == 10 ? radix_pass_any<10>(kin, vin, kout, vout, len, shift, last, ntiles, hist, s, v2in, v2out)
             : digit == 9 ? radix_pass_any<9>(kin, vin, kout, vout, len, shift, last, ntiles, hist, s, v2in, v2out)
                          : radix_pass_any<8>(kin, vin, kout, vout, len, shift, last, ntiles, hist, s, v2in, v2out);
        shift += digit;
        if (rc) return rc;
        std::swap(kin, kout);
        std::swap(vin, vout);
        std::swap(v2in, v2out);
    }
    *result_in_alt = (vin == vals_alt);
    return cuda_ok(cudaGetLastError(), "radix sort");
}

}  // namespace

int exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t len, cudaStream_t s) {
    if (len <= 0) return EGPR_SUCC;
    const int64_t ntiles = (len + kScanTile - 1) / kScanTile;
    if (ntiles == 1) {
        k_scan_tiles<<<1, kThreads, 0, s>>>(in, out, len, nullptr);
        return cuda_ok(cudaGetLastError(), "scan");
    }
    uint32_t* sums = nullptr;
    cudaError_t e = scratch_alloc(reinterpret_cast<void**>(&sums), (size_t)ntiles * sizeof(uint32_t), s);
    if (e != cudaSuccess) {
        set_cuda_error(e, "cudaMallocAsync (scan)");
        return EGPR_FAILED_TO_ALLOCATE_DEVICE_MEM;
    }
    k_scan_tiles<<<(unsigned)ntiles, kThreads, 0, s>>>(in, out, len, sums);
    int rc = exclusive_scan_u32(sums, sums, ntiles, s);
    if (rc == EGPR_SUCC) {
        k_scan_add<<<(unsigned)((len + 255) / 256), 256, 0, s>>>(out, len, sums);
        rc = cuda_ok(cudaGetLastError(), "scan add");
    }
    cudaFreeAsync(sums, s);
    return rc;
}

// ---- the sweep's layout -----------------------------------------------------------
// Block and index of every inbound entry's source: (rank / kBlockSrc) in the high
// bits, rank % kBlockSrc in the low kBlockBits (one-block layout: the rank).
__global__ void k_source_codes(const int32_t* in_col, int64_t nnz, const int32_t* __restrict__ rank,
                               int32_t blocked, uint32_t* code) {  // code may be in_col
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)rank[in_col[i]];
        code[i] = blocked ? ((r / (uint32_t)kBlockSrc) << kBlockBits) | (r % (uint32_t)kBlockSrc) : r;
    }
}

// First entry of every block in the code-sorted entries (nblocks + 1 values).
__global__ void k_block_starts(const uint32_t* __restrict__ code, int32_t nnz, int32_t nblocks,
                               int32_t* __restrict__ start) {
    for (int32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= nblocks; b += gridDim.x * blockDim.x) {
        int32_t lo = 0, hi = nnz;  // first entry of a block >= b
        if (b == nblocks) lo = nnz;
        while (lo < hi) {
            const int32_t mid = lo + ((hi - lo) >> 1);
            if ((int32_t)(code[mid] >> kBlockBits) < b) lo = mid + 1;
            else hi = mid;
        }
        start[b] = lo;
    }
}

__device__ __forceinline__ int32_t block_of_tile(const int32_t* __restrict__ block_tile, int32_t nblocks, int32_t t) {
    int32_t lo = 0, hi = nblocks - 1;  // the last block whose first tile is at or before t (no block is empty)
    while (lo < hi) {
        const int32_t mid = lo + ((hi - lo + 1) >> 1);
        if (block_tile[mid] <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// One warp per tile: indices and weights of its entries (zero-slot entries past
// the block's last one), run-end marks, marks of the lanes below, mark count.
__global__ void k_tiles(const uint32_t* __restrict__ code, const uint32_t* __restrict__ dst,
                        const float* __restrict__ w_in, const int32_t* __restrict__ block_start,
                        const int32_t* __restrict__ block_tile, int32_t nblocks, int32_t ntiles, int32_t blocked,
                        int32_t chunk_shift, void* __restrict__ idx, float* __restrict__ w_out, uint32_t* __restrict__ bits,
                        uint32_t* __restrict__ count) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = warp; t < ntiles; t += nwarps) {
        const int32_t b = block_of_tile(block_tile, nblocks, (int32_t)t);
        const int32_t end = block_start[b + 1];
        // 64-bit: a tile may reach past the last of nearly 2^31 entries
        const int64_t i0 = block_start[b] + (t - block_tile[b]) * kTileItems + kLaneItems * lane;
        uint32_t code8[kLaneItems], row8[kLaneItems + 1];
        float w8[kLaneItems];
#pragma unroll
        for (int u = 0; u < kLaneItems; ++u) {
            const bool in = i0 + u < end;
            code8[u] = in ? code[i0 + u] : (blocked ? (uint32_t)kBlockSrc : 0xffffffffu);
            row8[u] = in ? dst[i0 + u] : 0xffffffffu;
            if (w_out) w8[u] = in ? w_in[i0 + u] : 0.f;
        }
        row8[kLaneItems] = i0 + kLaneItems < end ? dst[i0 + kLaneItems] : 0xffffffffu;
        // a run ends with its row and with its chunk
        const int32_t in_chunk = (1 << chunk_shift) - 1;
        const bool chunk_end = (((int32_t)t - block_tile[b]) & in_chunk) == in_chunk;
        uint32_t marks = 0u;
#pragma unroll
        for (int u = 0; u < kLaneItems; ++u)
            if (i0 + u < end && (row8[u + 1] != row8[u] || (chunk_end && lane == 31 && u == kLaneItems - 1)))
                marks |= 1u << u;
        const uint32_t mine = __popc(marks);
        uint32_t incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        reinterpret_cast<uint16_t*>(bits + (size_t)t * kTileWords)[lane] = (uint16_t)(marks | ((incl - mine) << 8));
        if (lane == 31) count[t] = incl;
        const size_t o = (size_t)t * kTileItems + (size_t)(kLaneItems * lane);
        if (blocked) {
            uint4 p;
            constexpr uint32_t m = (1u << kBlockBits) - 1u;
            p.x = (code8[0] & m) | (code8[1] & m) << 16;
            p.y = (code8[2] & m) | (code8[3] & m) << 16;
            p.z = (code8[4] & m) | (code8[5] & m) << 16;
            p.w = (code8[6] & m) | (code8[7] & m) << 16;
            *reinterpret_cast<uint4*>(static_cast<uint16_t*>(idx) + o) = p;
        } else {
            uint4* q = reinterpret_cast<uint4*>(static_cast<int32_t*>(idx) + o);
            q[0] = make_uint4(code8[0], code8[1], code8[2], code8[3]);
            q[1] = make_uint4(code8[4], code8[5], code8[6], code8[7]);
        }
        if (w_out) {
            float4* q = reinterpret_cast<float4*>(w_out + o);
            q[0] = make_float4(w8[0], w8[1], w8[2], w8[3]);
            q[1] = make_float4(w8[4], w8[5], w8[6], w8[7]);
        }
    }
}

// Row tiles.  A row costs phase 2 about its pairs (at most one per block and one
// per tile of its entries) plus its finishing (about four pairs' worth); costs are in units of four.  A
// row tile is a run of 32-row groups: group g belongs to the tile its prefix of
// the costs falls in, floor(prefix / cap), where a group counts at least
// cap / max_groups, so no tile has more groups than that.
__global__ void k_group_cost(const int32_t* __restrict__ in_row, int32_t n, int32_t nblocks, int32_t groups,
                             uint32_t* __restrict__ cost) {
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g <= groups;
         g += (int64_t)gridDim.x * blockDim.x) {
        uint32_t c = 0u;
        for (int64_t r = g * kRowGroup; r < min((g + 1) * kRowGroup, (int64_t)n); ++r) {
            const int32_t len = in_row[r + 1] - in_row[r];
            c += (uint32_t)(min(len, nblocks) + len / kTileItems + 4);
        }
        cost[g] = (c + 3u) >> 2;  // group `groups` closes the scan with 0
    }
}

__device__ __forceinline__ uint32_t row_tile_cap(const uint32_t* total, int32_t want) {
    return *total / (uint32_t)want + 1u;
}

__global__ void k_group_floor(const uint32_t* __restrict__ cost, const uint32_t* __restrict__ total, int32_t want,
                              int32_t max_groups, int32_t groups, uint32_t* __restrict__ out) {
    const uint32_t least = (row_tile_cap(total, want) + (uint32_t)max_groups - 1u) / (uint32_t)max_groups;
    for (int32_t g = blockIdx.x * blockDim.x + threadIdx.x; g <= groups; g += gridDim.x * blockDim.x)
        out[g] = g < groups ? max(cost[g], least) : 0u;
}

// 1 for a group that begins a row tile.
__global__ void k_group_flags(const uint32_t* __restrict__ prefix, const uint32_t* __restrict__ total, int32_t want,
                              int32_t groups, uint32_t* __restrict__ flag) {
    const uint32_t cap = row_tile_cap(total, want);
    for (int32_t g = blockIdx.x * blockDim.x + threadIdx.x; g <= groups; g += gridDim.x * blockDim.x)
        flag[g] = g < groups && (g == 0 || prefix[g] / cap != prefix[g - 1] / cap) ? 1u : 0u;
}

// Row tile of every group, first row of every row tile.
__global__ void k_row_tiles(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ before,
                            int32_t groups, int32_t n, int32_t* __restrict__ group_tile,
                            int32_t* __restrict__ row_tile) {
    for (int32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < groups; g += gridDim.x * blockDim.x) {
        const int32_t q = (int32_t)(before[g] + flag[g]) - 1;
        group_tile[g] = q;
        if (flag[g]) row_tile[q] = g * kRowGroup;
        if (g == groups - 1) row_tile[q + 1] = n;
    }
}

// One warp per tile: the row of each of its pairs inside the row tile, and the
// first pair of every (row tile, block) cell.  Every cell is written once: the pair
// before the cell's first one writes it, the block's first pair the cells up to
// its own row tile, the last one the rest (and the closing row of cells).
__global__ void k_pair_rows(const uint32_t* __restrict__ dst, const int32_t* __restrict__ block_start,
                            const int32_t* __restrict__ block_tile, int32_t nblocks, int32_t ntiles,
                            const int32_t* __restrict__ group_tile, const int32_t* __restrict__ row_tile,
                            int32_t nrow_tiles, const uint32_t* __restrict__ bits,
                            const int32_t* __restrict__ tile_pair, uint16_t* __restrict__ pair_row,
                            int32_t* __restrict__ cell) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = warp; t < ntiles; t += nwarps) {
        const int32_t b = block_of_tile(block_tile, nblocks, (int32_t)t);
        const int32_t end = block_start[b + 1];
        const int64_t i0 = block_start[b] + (t - block_tile[b]) * kTileItems + kLaneItems * lane;
        const uint32_t mw = reinterpret_cast<const uint16_t*>(bits + (size_t)t * kTileWords)[lane];
        int32_t k = tile_pair[t] + (int32_t)(mw >> 8);
        for (int u = 0; u < kLaneItems; ++u) {
            if (!(mw & (1u << u))) continue;
            const uint32_t r = dst[i0 + u];
            const bool last = i0 + u + 1 >= end;
            const int32_t q0 = group_tile[r / kRowGroup];
            pair_row[k] = (uint16_t)(r - (uint32_t)row_tile[q0]);
            if (k == tile_pair[block_tile[b]])
                for (int32_t q = 0; q <= q0; ++q) cell[(size_t)q * nblocks + b] = k;
            const int32_t q1 = last ? nrow_tiles : group_tile[dst[i0 + u + 1] / kRowGroup];
            for (int32_t q = q0 + 1; q <= q1; ++q) cell[(size_t)q * nblocks + b] = k + 1;
            ++k;
        }
    }
}

// Steps of every (row tile, block) cell; 0 for the closing slot.
__global__ void k_cell_steps(const int32_t* __restrict__ cell, int64_t cells, int32_t nblocks,
                             uint32_t* __restrict__ count) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c <= cells; c += (int64_t)gridDim.x * blockDim.x)
        count[c] = c < cells ? (uint32_t)((cell[c + nblocks] - cell[c] + kStepPairs - 1) / kStepPairs) : 0u;
}

__global__ void k_steps(const int32_t* __restrict__ cell, int64_t cells, int32_t nblocks,
                        const uint32_t* __restrict__ first, int2* __restrict__ steps, int32_t* __restrict__ row_step) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c <= cells; c += (int64_t)gridDim.x * blockDim.x) {
        uint32_t at = first[c];
        if (c % nblocks == 0) row_step[c / nblocks] = (int32_t)at;
        if (c == cells) continue;
        const int32_t e = cell[c + nblocks];
        for (int32_t k = cell[c]; k < e; k += kStepPairs) steps[at++] = make_int2(k, min(kStepPairs, e - k));
    }
}

__global__ void k_gather_i32(const int32_t* __restrict__ src, const int32_t* __restrict__ at, int32_t count,
                             int32_t* __restrict__ out) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) out[i] = src[at[i]];
}

void expand_rows(const int32_t* row, int32_t n, int32_t* dst, cudaStream_t s) {
    k_expand_src<<<grid_for((int64_t)n * 32), kThreads, 0, s>>>(row, n, dst);
}

// Defaults of a graph's layout parameters (egpr_graph_set_tuning and
// egpr_graph_autotune change them per graph).
int default_chunks_per_warp() {
    static const int v = [] {
        const char* e = std::getenv("EGPR_CHUNKS_PER_WARP");  // row tiles per resident warp
        const int x = e ? std::atoi(e) : 8;
        return x >= 1 && x <= 64 ? x : 8;
    }();
    return v;
}

// Cost of one pair, in entries, when phase 1 is cut into CTA shares.
int default_row_cost() {
    static const int v = [] {
        const char* e = std::getenv("EGPR_ROW_COST");
        const int x = e ? std::atoi(e) : 4;
        return x >= 0 && x <= 64 ? x : 4;
    }();
    return v;
}

// (row tile, block) cells above which the blocks are given up: graphs of more than
// about 3 * 10^8 vertices, whose cells would hold fewer pairs than a step costs.
// EGPR_MAX_CELLS lowers it (tests).
int64_t max_pair_cells() {
    const char* e = std::getenv("EGPR_MAX_CELLS");
    const long long x = e ? std::atoll(e) : 0;
    return x > 0 ? (int64_t)x : (int64_t)1 << 28;
}

// Builds the sweep's layout (see GraphDev) from the inbound entries in
// destination order: src (sources) in `code`, destinations in `dst`, weights in
// `w` (NULL: unit weights).  The three arrays and their *_alt counterparts are
// scratch of nnz entries that the sort overwrites; code may equal in_col's copy.
int build_sweep_layout(egpr_graph* g, uint32_t* code, uint32_t* dst, uint32_t* w, uint32_t* code_alt,
                       uint32_t* dst_alt, uint32_t* w_alt, TmpAlloc& tmp, cudaStream_t s) {
    const int32_t n = g->n;
    const int32_t nnz = (int32_t)g->nnz;
    int rc = EGPR_SUCC;
    if (nnz <= 0 || g->nsrc <= 0) {
        g->nblocks = 0;
        g->h_block_tile.assign(1, 0);
        g->h_block_pair.assign(1, 0);
        g->nrow_tiles = 0;
        return EGPR_SUCC;
    }
    // row tiles: a quarter of tune_cpw per resident CTA of phase 2 (fewer where they would
    // have less than kMinTileRows rows), of up to four times the mean number of rows
    const int32_t want = (int32_t)std::max<int64_t>(
        1, std::min<int64_t>((int64_t)sweep_grid() * kRowTilesPerSm * std::max(1, g->tune_cpw) / 4,
                             ((int64_t)n + kMinTileRows - 1) / kMinTileRows));
    int32_t max_rows = kMinTileRows;
    while (max_rows < kMaxTileRows && (int64_t)max_rows * want < 4 * (int64_t)n) max_rows = std::min(2 * max_rows, kMaxTileRows);
    const int32_t groups = (n + kRowGroup - 1) / kRowGroup;
    int32_t nb = (g->nsrc + kBlockSrc - 1) / kBlockSrc;
    uint32_t* d_gcost = tmp.get<uint32_t>((size_t)groups + 1, &rc);
    uint32_t* d_gpre = tmp.get<uint32_t>((size_t)groups + 1, &rc);
    uint32_t* d_gfloor = tmp.get<uint32_t>((size_t)groups + 1, &rc);
    uint32_t* d_gflag = tmp.get<uint32_t>((size_t)groups + 1, &rc);
    int32_t* d_gtile = tmp.get<int32_t>((size_t)groups, &rc);
    int32_t* d_rtile = tmp.get<int32_t>((size_t)groups + 1, &rc);
    if (rc) return rc;
    k_group_cost<<<grid_for((int64_t)groups + 1), kThreads, 0, s>>>(g->in_row.as<int32_t>(), n, nb, groups, d_gcost);
    if ((rc = exclusive_scan_u32(d_gcost, d_gpre, (int64_t)groups + 1, s))) return rc;
    k_group_floor<<<grid_for(groups + 1), kThreads, 0, s>>>(d_gcost, d_gpre + groups, want, max_rows / kRowGroup, groups,
                                                            d_gfloor);
    uint32_t* d_fpre = reinterpret_cast<uint32_t*>(d_rtile);  // free until k_row_tiles
    if ((rc = exclusive_scan_u32(d_gfloor, d_fpre, (int64_t)groups + 1, s))) return rc;
    k_group_flags<<<grid_for(groups + 1), kThreads, 0, s>>>(d_fpre, d_gpre + groups, want, groups, d_gflag);
    if ((rc = exclusive_scan_u32(d_gflag, d_gfloor, (int64_t)groups + 1, s))) return rc;
    k_row_tiles<<<grid_for(groups), kThreads, 0, s>>>(d_gflag, d_gfloor, groups, n, d_gtile, d_rtile);
    uint32_t nrt_u = 0;
    if ((rc = cuda_ok(cudaMemcpyAsync(&nrt_u, d_gfloor + groups, sizeof(nrt_u), cudaMemcpyDeviceToHost, s), "D2H row tiles")) ||
        (rc = cuda_ok(cudaStreamSynchronize(s), "sweep layout")))
        return rc;
    const int32_t nrt = (int32_t)nrt_u;
    const bool blocked = (int64_t)nb * ((int64_t)nrt + 1) <= max_pair_cells();
    if (!blocked) nb = 1;
    g->nblocks = nb;
    g->nrow_tiles = nrt;
    g->global_block = blocked ? 0 : 1;
    g->max_tile_rows = max_rows;
    // chunks of four tiles where every warp still gets several of them
    g->chunk_shift = nnz >= 2 * sweep_resident_warps() * (4 * kTileItems) ? 2 : 0;
    k_source_codes<<<grid_for(nnz), kThreads, 0, s>>>(reinterpret_cast<const int32_t*>(code), nnz,
                                                      g->rank.as<int32_t>(), blocked ? 1 : 0, code);
    int bits = 0;
    while (((nb - 1) >> bits) != 0) ++bits;
    bool alt = false;
    if ((rc = radix_sort_pairs(code, dst, code_alt, dst_alt, nnz, bits, s, tmp, &alt, true, w, w_alt, kBlockBits)))
        return rc;
    if (alt) {
        std::swap(code, code_alt);
        std::swap(dst, dst_alt);
        std::swap(w, w_alt);
    }
    int32_t* d_start = tmp.get<int32_t>((size_t)nb + 1, &rc);
    int32_t* d_btile = tmp.get<int32_t>((size_t)nb + 1, &rc);
    int32_t* d_bpair = tmp.get<int32_t>((size_t)nb + 1, &rc);
    if (rc) return rc;
    std::vector<int32_t> start((size_t)nb + 1);
    if (blocked) {
        k_block_starts<<<grid_for(nb + 1), kThreads, 0, s>>>(code, nnz, nb, d_start);
        if ((rc = cuda_ok(cudaMemcpyAsync(start.data(), d_start, start.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, s), "D2H block starts")) ||
            (rc = cuda_ok(cudaStreamSynchronize(s), "sweep layout")))
            return rc;
    } else {
        start[0] = 0;
        start[1] = nnz;
        if ((rc = cuda_ok(cudaMemcpyAsync(d_start, start.data(), start.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s), "H2D block starts")))
            return rc;
    }
    std::vector<int32_t>& btile = g->h_block_tile;
    btile.assign((size_t)nb + 1, 0);
    for (int32_t b = 0; b < nb; ++b)
        btile[(size_t)b + 1] = btile[(size_t)b] +
                               (int32_t)(((int64_t)start[(size_t)b + 1] - start[(size_t)b] + kTileItems - 1) / kTileItems);
    const int32_t ntiles = btile[(size_t)nb];
    const size_t entries = (size_t)ntiles * kTileItems;
    const int64_t cells = (int64_t)nrt * nb;
    uint32_t* d_count = tmp.get<uint32_t>((size_t)ntiles + 1, &rc);
    int32_t* d_cell = tmp.get<int32_t>((size_t)cells + (size_t)nb, &rc);  // [row tile][block], closed by a row
    uint32_t* d_first = tmp.get<uint32_t>((size_t)cells + 1, &rc);
    if (rc || (rc = g->idx.alloc(entries * (blocked ? sizeof(uint16_t) : sizeof(int32_t)))) ||
        (g->weighted && (rc = g->sw_w.alloc(entries * sizeof(float)))) ||
        (rc = g->tile_bits.alloc((size_t)ntiles * kTileWords * sizeof(uint32_t))) ||
        (rc = g->tile_pair.alloc(((size_t)ntiles + 1) * sizeof(int32_t))) ||
        (rc = g->row_tile.alloc(((size_t)nrt + 1) * sizeof(int32_t))) ||
        (rc = g->row_step.alloc(((size_t)nrt + 1) * sizeof(int32_t))))
        return rc;
    if ((rc = cuda_ok(cudaMemcpyAsync(g->row_tile.p, d_rtile, ((size_t)nrt + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, s), "row tiles")) ||
        (rc = cuda_ok(cudaMemcpyAsync(d_btile, btile.data(), btile.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s), "H2D block tiles")) ||
        (rc = cuda_ok(cudaMemsetAsync(d_count + ntiles, 0, sizeof(uint32_t), s), "memset")))
        return rc;
    k_tiles<<<grid_for((int64_t)ntiles * 32), kThreads, 0, s>>>(
        code, dst, reinterpret_cast<const float*>(w), d_start, d_btile, nb, ntiles, blocked ? 1 : 0, g->chunk_shift, g->idx.p,
        g->weighted ? g->sw_w.as<float>() : nullptr, g->tile_bits.as<uint32_t>(), d_count);
    if ((rc = exclusive_scan_u32(d_count, g->tile_pair.as<uint32_t>(), (int64_t)ntiles + 1, s))) return rc;
    k_gather_i32<<<grid_for(nb + 1), kThreads, 0, s>>>(g->tile_pair.as<int32_t>(), d_btile, nb + 1, d_bpair);
    g->h_block_pair.assign((size_t)nb + 1, 0);
    if ((rc = cuda_ok(cudaMemcpyAsync(g->h_block_pair.data(), d_bpair, ((size_t)nb + 1) * sizeof(int32_t), cudaMemcpyDeviceToHost, s), "D2H pairs")) ||
        (rc = cuda_ok(cudaStreamSynchronize(s), "sweep layout")))
        return rc;
    const size_t npairs = (size_t)g->h_block_pair[(size_t)nb];
    if ((rc = g->pair_row.alloc(npairs * sizeof(uint16_t))) || (rc = g->pairs.alloc(npairs * sizeof(double)))) return rc;
    k_pair_rows<<<grid_for((int64_t)ntiles * 32), kThreads, 0, s>>>(
        dst, d_start, d_btile, nb, ntiles, d_gtile, d_rtile, nrt, g->tile_bits.as<uint32_t>(),
        g->tile_pair.as<int32_t>(), g->pair_row.as<uint16_t>(), d_cell);
    k_cell_steps<<<grid_for(cells + 1), kThreads, 0, s>>>(d_cell, cells, nb, d_first);
    if ((rc = exclusive_scan_u32(d_first, d_first, cells + 1, s))) return rc;
    uint32_t nsteps = 0;
    if ((rc = cuda_ok(cudaMemcpyAsync(&nsteps, d_first + cells, sizeof(nsteps), cudaMemcpyDeviceToHost, s), "D2H steps")) ||
        (rc = cuda_ok(cudaStreamSynchronize(s), "sweep layout")) || (rc = g->steps.alloc((size_t)nsteps * sizeof(int2))))
        return rc;
    k_steps<<<grid_for(cells + 1), kThreads, 0, s>>>(d_cell, cells, nb, d_first, g->steps.as<int2>(), g->row_step.as<int32_t>());
    if ((rc = cuda_ok(cudaGetLastError(), "sweep layout"))) return rc;
    return cuda_ok(cudaStreamSynchronize(s), "sweep layout");
}

int rebuild_sweep_layout(egpr_graph* g, cudaStream_t s) {
    TmpAlloc tmp(s);
    int rc = EGPR_SUCC;
    const size_t nnz = (size_t)std::max<int64_t>(g->nnz, 1);
    uint32_t* code = tmp.get<uint32_t>(nnz, &rc);
    uint32_t* code2 = tmp.get<uint32_t>(nnz, &rc);
    uint32_t* dst = tmp.get<uint32_t>(nnz, &rc);
    uint32_t* dst2 = tmp.get<uint32_t>(nnz, &rc);
    uint32_t* w = g->weighted ? tmp.get<uint32_t>(nnz, &rc) : nullptr;
    uint32_t* w2 = g->weighted ? tmp.get<uint32_t>(nnz, &rc) : nullptr;
    if (rc) return rc;
    expand_rows(g->in_row.as<int32_t>(), g->n, reinterpret_cast<int32_t*>(dst), s);
    if ((rc = cuda_ok(cudaMemcpyAsync(code, g->in_col.p, (size_t)g->nnz * sizeof(int32_t), cudaMemcpyDeviceToDevice, s), "sources")) ||
        (w && (rc = cuda_ok(cudaMemcpyAsync(w, g->in_w.p, (size_t)g->nnz * sizeof(float), cudaMemcpyDeviceToDevice, s), "weights"))))
        return rc;
    return build_sweep_layout(g, code, dst, w, code2, dst2, w2, tmp, s);
}

// ---- the binned sweep's layout -------------------------------------------------
// Renumbering key of vertex v: the hub block (the first `hubs` vertices of the
// out-degree ranking) first, then everyone else; descending in-degree inside
// each block; the sort is stable, so equal keys keep ascending vertex ids.
__global__ void k_bin_keys(const int32_t* __restrict__ in_row, int32_t n, const uint8_t* __restrict__ hub_flag,
                           uint32_t* __restrict__ key, uint32_t* __restrict__ val) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t deg = (uint32_t)(in_row[v + 1] - in_row[v]);
        key[v] = (hub_flag[v] ? 0u : 0x80000000u) | (0x7fffffffu - deg);
        val[v] = (uint32_t)v;
    }
}

__global__ void k_bin_hub_flags(const uint32_t* __restrict__ ranked, int32_t hubs, uint8_t* __restrict__ flag) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < hubs; i += gridDim.x * blockDim.x) flag[ranked[i]] = 1;
}

// inv: the sorted vertex list; perm[inv[i]] = i; row lengths and FP64
// out-weights in the new order.
__global__ void k_bin_perm(const uint32_t* __restrict__ inv, int32_t n, const int32_t* __restrict__ in_row,
                           const double* __restrict__ outw, int32_t* __restrict__ perm, uint32_t* __restrict__ len,
                           double* __restrict__ outw_new) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)inv[i];
        perm[v] = (int32_t)i;
        len[i] = (uint32_t)(in_row[v + 1] - in_row[v]);
        outw_new[i] = outw[v];
    }
}

// Inbound entry e (destination dst[e], source in_col[e]) to its place in the
// renumbered CSR: same position inside its row, source renumbered.
__global__ void k_bin_entries(const uint32_t* __restrict__ dst, int64_t nnz, const int32_t* __restrict__ in_row,
                              const int32_t* __restrict__ in_col, const float* __restrict__ in_w,
                              const int32_t* __restrict__ perm, const int32_t* __restrict__ row_new,
                              int32_t* __restrict__ col_new, float* __restrict__ w_new) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)dst[e];
        const int64_t pos = (int64_t)row_new[perm[v]] + (e - (int64_t)in_row[v]);
        col_new[pos] = perm[in_col[e]];
        if (w_new) w_new[pos] = in_w[e];
    }
}

// Builds g->bins from the natural inbound CSR (in_row, plain source ids in
// in_col, in_w, outw) and the out-degree ranking of the vertices.  The work
// queue follows in bins_build_items.
int build_bin_layout(egpr_graph* g, const uint32_t* sorted_dst, const uint32_t* ranked, TmpAlloc& tmp,
                     cudaStream_t s) {
    const int32_t n = g->n;
    const int64_t nnz = g->nnz;
    BinLayout* B = new (std::nothrow) BinLayout();
    if (!B) return EGPR_FAILED_TO_ALLOCATE_HOST_MEM;
    g->bins = B;
    B->n = n;
    B->nnz = nnz;
    B->hubs = std::min<int32_t>(n, bin_hub_cap()) & ~3;  // a multiple of 4: the staging copy moves 16-byte units
    if (const char* e = std::getenv("EGPR_BIN_HUBS")) B->hubs = std::min<int32_t>(B->hubs, std::max(0, atoi(e)) & ~3);
    int rc = EGPR_SUCC;
    uint8_t* flag = tmp.get<uint8_t>((size_t)n, &rc);
    uint32_t* key = tmp.get<uint32_t>((size_t)n, &rc);
    uint32_t* val = tmp.get<uint32_t>((size_t)n, &rc);
    uint32_t* key2 = tmp.get<uint32_t>((size_t)n, &rc);
    uint32_t* val2 = tmp.get<uint32_t>((size_t)n, &rc);
    uint32_t* len = tmp.get<uint32_t>((size_t)n + 1, &rc);
    if (rc) return rc;
    // Every array the sweep reads row by row is padded by 16 entries (vector
    // loads near the end); the padding is zero.
    const size_t pad = 16;
    if ((rc = B->perm.alloc((size_t)n * sizeof(int32_t))) || (rc = B->inv.alloc((size_t)n * sizeof(int32_t))) ||
        (rc = B->row.alloc(((size_t)n + 1 + pad) * sizeof(int32_t))) ||
        (rc = B->col.alloc(((size_t)std::max<int64_t>(nnz, 1) + pad) * sizeof(int32_t))) ||
        (rc = B->outw.alloc(((size_t)n + pad) * sizeof(double))) ||
        (g->weighted && (rc = B->w.alloc(((size_t)std::max<int64_t>(nnz, 1) + pad) * sizeof(float)))))
        return rc;
    cudaMemsetAsync(flag, 0, (size_t)n, s);
    cudaMemsetAsync(len, 0, ((size_t)n + 1) * sizeof(uint32_t), s);  // len[n] = 0 closes the scan
    cudaMemsetAsync(B->row.p, 0, B->row.bytes, s);
    cudaMemsetAsync(B->col.p, 0, B->col.bytes, s);
    if (g->weighted) cudaMemsetAsync(B->w.p, 0, B->w.bytes, s);
    if (B->hubs > 0) k_bin_hub_flags<<<grid_for(B->hubs), kThreads, 0, s>>>(ranked, B->hubs, flag);
    k_bin_keys<<<grid_for(n), kThreads, 0, s>>>(g->in_row.as<int32_t>(), n, flag, key, val);
    bool alt = false;
    if ((rc = radix_sort_pairs(key, val, key2, val2, n, 32, s, tmp, &alt, false))) return rc;
    const uint32_t* inv = alt ? val2 : val;
    cudaMemcpyAsync(B->inv.p, inv, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToDevice, s);
    k_bin_perm<<<grid_for(n), kThreads, 0, s>>>(inv, n, g->in_row.as<int32_t>(), g->outw.as<double>(),
                                                B->perm.as<int32_t>(), len, B->outw.as<double>());
    if ((rc = exclusive_scan_u32(len, reinterpret_cast<uint32_t*>(B->row.as<int32_t>()), (int64_t)n + 1, s)))
        return rc;
    if (nnz > 0)
        k_bin_entries<<<grid_for(nnz), kThreads, 0, s>>>(sorted_dst, nnz, g->in_row.as<int32_t>(),
                                                         g->in_col.as<int32_t>(), g->weighted ? g->in_w.as<float>() : nullptr,
                                                         B->perm.as<int32_t>(), B->row.as<int32_t>(),
                                                         B->col.as<int32_t>(), g->weighted ? B->w.as<float>() : nullptr);
    if ((rc = cuda_ok(cudaGetLastError(), "binned layout"))) return rc;
    if ((rc = bins_build_items(g, s))) return rc;
    return bins_alloc_solve(g, s);
}

// ---- host inputs ------------------------------------------------------------
// A host input array reaches the device in one of three ways:
//  * already page-locked (torch pinned memory, cudaHostAlloc, a registered
//    range): copied by DMA directly;
//  * pageable, with EASYGRAPH_GPU_HOST_REGISTER set to 1/TRUE/ON/YES:
//    page-locked in place for the upload and released after it, as the
//    reference's prepare_h2d_source / release_h2d_source do
//    (gpu_easygraph/common/buffer_cache.h:115-176), for arrays of at least
//    EASYGRAPH_GPU_HOST_REGISTER_MIN_BYTES (default 1 MiB); read-only
//    mappings (memory-mapped bulk CSR files) are registered read-only where
//    the device supports it;
//  * pageable otherwise (the default here; the reference registers by
//    default): copied through a process-wide pool of page-locked staging
//    buffers, host threads filling one buffer while DMA drains the others.
//    Registering pages in place cost about 0.2 s per GB on B200 hosts, several
//    times the copy itself, and it is paid again on every call.
bool host_register_requested() {
    const char* v = std::getenv("EASYGRAPH_GPU_HOST_REGISTER");
    if (!v) return false;
    std::string s(v);
    for (char& c : s) c = (char)std::toupper((unsigned char)c);
    return s == "1" || s == "TRUE" || s == "ON" || s == "YES";
}

size_t host_register_min_bytes() {
    const char* v = std::getenv("EASYGRAPH_GPU_HOST_REGISTER_MIN_BYTES");
    const unsigned long long parsed = v ? std::strtoull(v, nullptr, 10) : 0ull;
    return parsed > 0ull ? (size_t)parsed : (size_t)1 << 20;
}

bool host_page_locked(const void* p) {
    cudaPointerAttributes a = {};
    const cudaError_t e = cudaPointerGetAttributes(&a, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// Page-locked staging buffers shared by every upload of the process (one
// upload at a time uses them).
constexpr int kStageSlots = 4;
constexpr size_t kStageBytes = (size_t)32 << 20;
struct StagePool {
    std::mutex mu;
    void* slot[kStageSlots] = {};
};
StagePool& stage_pool() {
    static StagePool* p = new StagePool();  // never destroyed: pinned memory outlives static teardown order
    return *p;
}

void parallel_memcpy(void* dst, const void* src, size_t bytes) {
    constexpr size_t kBlock = (size_t)1 << 20;
    const int64_t blocks = (int64_t)((bytes + kBlock - 1) / kBlock);
    if (blocks <= 1) {
        std::memcpy(dst, src, bytes);
        return;
    }
#pragma omp parallel for schedule(static) num_threads(std::min<int64_t>(blocks, 16))
    for (int64_t i = 0; i < blocks; ++i) {
        const size_t off = (size_t)i * kBlock;
        std::memcpy(static_cast<char*>(dst) + off, static_cast<const char*>(src) + off,
                    std::min(kBlock, bytes - off));
    }
}

// H2D copy of a pageable host array through the staging pool, enqueued on s.
// Returns once every byte has left the source array (later work on s sees
// the data in stream order).
int staged_h2d(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    StagePool& P = stage_pool();
    std::lock_guard<std::mutex> lk(P.mu);
    for (int k = 0; k < kStageSlots; ++k)
        if (!P.slot[k]) {
            const cudaError_t e = cudaHostAlloc(&P.slot[k], kStageBytes, cudaHostAllocPortable);
            if (e != cudaSuccess) {
                P.slot[k] = nullptr;
                cudaGetLastError();
                // no staging memory: the driver copies from pageable memory
                return cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s), "H2D (pageable)");
            }
        }
    cudaEvent_t ev[kStageSlots] = {};
    bool used[kStageSlots] = {};
    int rc = EGPR_SUCC;
    for (int k = 0; k < kStageSlots && !rc; ++k)
        rc = cuda_ok(cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming), "event");
    size_t off = 0;
    for (int i = 0; off < bytes && !rc; ++i) {
        const int k = i % kStageSlots;
        const size_t len = std::min(kStageBytes, bytes - off);
        if (used[k] && (rc = cuda_ok(cudaEventSynchronize(ev[k]), "staging"))) break;
        parallel_memcpy(P.slot[k], static_cast<const char*>(src) + off, len);
        if ((rc = cuda_ok(cudaMemcpyAsync(static_cast<char*>(dst) + off, P.slot[k], len, cudaMemcpyHostToDevice, s),
                          "H2D (staged)")))
            break;
        if ((rc = cuda_ok(cudaEventRecord(ev[k], s), "event"))) break;
        used[k] = true;
        off += len;
    }
    // the slots are free again once their last copies are done
    for (int k = 0; k < kStageSlots; ++k) {
        if (used[k]) cudaEventSynchronize(ev[k]);
        if (ev[k]) cudaEventDestroy(ev[k]);
    }
    return rc;
}

// D2H copy into a pageable host array through the staging pool, after the
// work already enqueued on s: up to kStageSlots chunk copies in flight while
// host threads move finished chunks out.  Returns once every byte is in dst.
int staged_d2h(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    // the work that produces the result finishes before the pool is taken, so
    // another thread's upload or download does not wait on this stream's kernels
    int rc0 = cuda_ok(cudaStreamSynchronize(s), "D2H (staged)");
    if (rc0) return rc0;
    StagePool& P = stage_pool();
    std::lock_guard<std::mutex> lk(P.mu);
    for (int k = 0; k < kStageSlots; ++k)
        if (!P.slot[k]) {
            const cudaError_t e = cudaHostAlloc(&P.slot[k], kStageBytes, cudaHostAllocPortable);
            if (e != cudaSuccess) {
                P.slot[k] = nullptr;
                cudaGetLastError();
                int rc = cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), "D2H (pageable)");
                return rc ? rc : cuda_ok(cudaStreamSynchronize(s), "D2H (pageable)");
            }
        }
    cudaEvent_t ev[kStageSlots] = {};
    int rc = EGPR_SUCC;
    for (int k = 0; k < kStageSlots && !rc; ++k)
        rc = cuda_ok(cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming), "event");
    const size_t chunks = (bytes + kStageBytes - 1) / kStageBytes;
    auto issue = [&](size_t i) {
        const int k = (int)(i % kStageSlots);
        const size_t off = i * kStageBytes, len = std::min(kStageBytes, bytes - off);
        int r = cuda_ok(cudaMemcpyAsync(P.slot[k], static_cast<const char*>(src) + off, len, cudaMemcpyDeviceToHost, s),
                        "D2H (staged)");
        return r ? r : cuda_ok(cudaEventRecord(ev[k], s), "event");
    };
    for (size_t i = 0; i < std::min<size_t>(chunks, kStageSlots) && !rc; ++i) rc = issue(i);
    for (size_t i = 0; i < chunks && !rc; ++i) {
        const int k = (int)(i % kStageSlots);
        const size_t off = i * kStageBytes, len = std::min(kStageBytes, bytes - off);
        if ((rc = cuda_ok(cudaEventSynchronize(ev[k]), "staging"))) break;
        parallel_memcpy(static_cast<char*>(dst) + off, P.slot[k], len);
        if (i + kStageSlots < chunks) rc = issue(i + kStageSlots);
    }
    if (rc) cudaStreamSynchronize(s);  // no copy may still write into a slot once the pool is unlocked
    for (int k = 0; k < kStageSlots; ++k)
        if (ev[k]) cudaEventDestroy(ev[k]);
    return rc;
}

struct HostInputs {
    cudaStream_t stream;            // the upload's stream: drained before unregistering
    std::vector<void*> registered;  // registered here, unregistered when the upload is done
    int registered_count = 0;
    int already_locked = 0;
    int staged = 0;
    explicit HostInputs(cudaStream_t s) : stream(s) {}
    // Decides how `p` is uploaded; true when it is (now) page-locked.
    bool prepare(const void* p, size_t bytes, int dev) {
        if (!p || bytes == 0) return true;
        if (host_page_locked(p)) {
            ++already_locked;
            return true;
        }
        if (host_register_requested() && bytes >= host_register_min_bytes()) {
            int ro = 0;
            cudaDeviceGetAttribute(&ro, cudaDevAttrHostRegisterReadOnlySupported, dev);
            const unsigned flags = cudaHostRegisterPortable | (ro ? cudaHostRegisterReadOnly : 0u);
            const cudaError_t e = cudaHostRegister(const_cast<void*>(p), bytes, flags);
            if (e == cudaSuccess) {
                registered.push_back(const_cast<void*>(p));
                ++registered_count;
                return true;
            }
            cudaGetLastError();
            if (e == cudaErrorHostMemoryAlreadyRegistered) {  // not ours to unregister
                ++already_locked;
                return true;
            }
        }
        if (bytes >= ((size_t)1 << 20)) ++staged;
        return bytes < ((size_t)1 << 20);  // small arrays: the driver's pageable copy
    }
    ~HostInputs() {
        if (registered.empty()) return;
        cudaStreamSynchronize(stream);  // no copy from these pages may still be in flight
        for (void* p : registered) cudaHostUnregister(p);
        cudaGetLastError();
    }
};

// H2D of [src, src + bytes): direct when `locked`, else through the staging pool.
int upload_h2d(void* dst, const void* src, size_t bytes, bool locked, cudaStream_t s, const char* what) {
    if (bytes == 0) return EGPR_SUCC;
    if (locked) return cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s), what);
    return staged_h2d(dst, src, bytes, s);
}

int download_d2h(void* dst, const void* src, size_t bytes, cudaStream_t s, const char* what) {
    if (bytes == 0) return EGPR_SUCC;
    if (bytes < ((size_t)1 << 20) || host_page_locked(dst))
        return cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), what);
    return staged_d2h(dst, src, bytes, s);
}

int prepare_graph(egpr_graph* g, const int32_t* V, const int32_t* E, const double* W) {
    const int32_t n = g->n;
    const int64_t m = g->m_input;
    cudaStream_t s = g->own_stream;
    int rc = EGPR_SUCC;
    const double t0 = wall_seconds();
    // declared before the scratch so that registrations outlive every copy
    // (the stream is synchronised before this function returns)
    HostInputs host(s);
    const bool v_locked = host.prepare(V, ((size_t)n + 1) * sizeof(int32_t), g->device);
    const bool e_locked = host.prepare(E, (size_t)m * sizeof(int32_t), g->device);
    const bool w_locked = host.prepare(W, W ? (size_t)m * sizeof(double) : 0, g->device);
    g->host_inputs_registered = host.registered_count;
    g->host_inputs_locked = host.already_locked;
    g->host_inputs_staged = host.staged;
    cudaEventRecord(g->ev0, s);
    {
        TmpAlloc tmp(s);
        int32_t* dV = tmp.get<int32_t>((size_t)n + 1, &rc);
        int32_t* dE = tmp.get<int32_t>((size_t)m, &rc);
        double* dW = W ? tmp.get<double>((size_t)m, &rc) : nullptr;
        uint32_t* indeg = tmp.get<uint32_t>((size_t)n + 1, &rc);
        uint32_t* keys = tmp.get<uint32_t>((size_t)m, &rc);
        uint32_t* vals = tmp.get<uint32_t>((size_t)m, &rc);
        uint32_t* keys2 = tmp.get<uint32_t>((size_t)m, &rc);
        uint32_t* vals2 = tmp.get<uint32_t>((size_t)m, &rc);
        // weighted: the FP32 weight of every entry moves through the sort with its source
        uint32_t* wbits = W ? tmp.get<uint32_t>((size_t)m, &rc) : nullptr;
        uint32_t* wbits2 = W ? tmp.get<uint32_t>((size_t)m, &rc) : nullptr;
        unsigned long long* counts = tmp.get<unsigned long long>(3, &rc);
        uint32_t* hkey = tmp.get<uint32_t>((size_t)n, &rc);
        uint32_t* hval = tmp.get<uint32_t>((size_t)n, &rc);
        uint32_t* hkey2 = tmp.get<uint32_t>((size_t)n, &rc);
        uint32_t* hval2 = tmp.get<uint32_t>((size_t)n, &rc);
        // weighted: rows whose out-weight is summed sequentially (k_out_weight_exact)
        int32_t* serial_rows = W ? tmp.get<int32_t>((size_t)n, &rc) : nullptr;
        uint32_t* serial_count = W ? tmp.get<uint32_t>(1, &rc) : nullptr;
        int32_t* long_rows = W ? tmp.get<int32_t>((size_t)n, &rc) : nullptr;  // per piece: sources of many entries
        uint32_t* long_count = W ? tmp.get<uint32_t>(1, &rc) : nullptr;
        // per piece: segments of the sources of very many entries, and their accumulators
        OutSegs segs;
        const size_t max_huge = (size_t)(m / kOutWeightHuge) + 1;
        segs.seg = tmp.get<int4>((size_t)(m / kOutWeightSeg) + max_huge, &rc);
        segs.seg_count = tmp.get<uint32_t>(1, &rc);
        segs.acc = tmp.get<HugeAcc>(max_huge, &rc);
        segs.acc_count = tmp.get<uint32_t>(1, &rc);
        if (rc) return rc;
        if (W) cudaMemsetAsync(serial_count, 0, sizeof(uint32_t), s);
        if ((rc = g->in_row.alloc(((size_t)n + 8) * sizeof(int32_t))) ||
            (rc = g->outw.alloc((size_t)n * sizeof(double))) ||
            (rc = g->dangling01.alloc((size_t)n * sizeof(int32_t))))
            return rc;
        if ((rc = upload_h2d(dV, V, ((size_t)n + 1) * sizeof(int32_t), v_locked, s, "H2D offsets"))) return rc;
        cudaMemsetAsync(indeg, 0, ((size_t)n + 1) * sizeof(uint32_t), s);
        cudaMemsetAsync(counts, 0, 3 * sizeof(unsigned long long), s);
        // the sort carries each entry's source (written from the offsets alone,
        // while E is still arriving) and, when weighted, its FP32 weight
        // (converted as each piece of W arrives), so no gather follows it
        if (m > 0)
            k_expand_src<<<grid_for((int64_t)n * 32), kThreads, 0, s>>>(dV, n, reinterpret_cast<int32_t*>(vals));
        {
            // E (and W) arrive in pieces on a copy stream; the degree passes of
            // each piece run on s while the next one is in flight.  A piece's
            // out-degree pass covers the rows whose entries have all arrived.
            const int pieces = m >= (int64_t)(8 << 20) ? 4 : 1;
            cudaStream_t sc = nullptr;
            std::vector<cudaEvent_t> ev((size_t)pieces, nullptr);
            if (pieces > 1) {
                rc = cuda_ok(cudaStreamCreateWithFlags(&sc, cudaStreamNonBlocking), "stream");
                for (int i = 0; i < pieces && !rc; ++i)
                    rc = cuda_ok(cudaEventCreateWithFlags(&ev[(size_t)i], cudaEventDisableTiming), "event");
                // the copy stream starts after the memsets and the offsets above
                cudaEvent_t start = nullptr;
                if (!rc) rc = cuda_ok(cudaEventCreateWithFlags(&start, cudaEventDisableTiming), "event");
                if (!rc) rc = cuda_ok(cudaEventRecord(start, s), "event");
                if (!rc) rc = cuda_ok(cudaStreamWaitEvent(sc, start, 0), "event");
                if (start) cudaEventDestroy(start);
            }
            int32_t r_done = 0;
            for (int i = 0; i < pieces && !rc; ++i) {
                const int64_t a = m * i / pieces, b = m * (i + 1) / pieces;
                cudaStream_t cs = pieces > 1 ? sc : s;
                if (b > a) {
                    rc = upload_h2d(dE + a, E + a, (size_t)(b - a) * sizeof(int32_t), e_locked, cs, "H2D indices");
                    if (!rc && W)
                        rc = upload_h2d(dW + a, W + a, (size_t)(b - a) * sizeof(double), w_locked, cs, "H2D weights");
                }
                if (!rc && pieces > 1) {
                    rc = cuda_ok(cudaEventRecord(ev[(size_t)i], sc), "event");
                    if (!rc) rc = cuda_ok(cudaStreamWaitEvent(s, ev[(size_t)i], 0), "event");
                }
                if (rc) break;
                // rows [r_done, r_end): V[r_end] <= b, all of them when this is the last piece
                int32_t r_end = n;
                if (i + 1 < pieces) r_end = (int32_t)(std::upper_bound(V, V + n + 1, (int32_t)b) - V) - 1;
                if (r_end > r_done) {
                    cudaMemsetAsync(segs.seg_count, 0, sizeof(uint32_t), s);
                    cudaMemsetAsync(segs.acc_count, 0, sizeof(uint32_t), s);
                    if (dW) {
                        cudaMemsetAsync(long_count, 0, sizeof(uint32_t), s);
                        k_out_weight_exact<<<grid_for((int64_t)(r_end - r_done) * 8), kThreads, 0, s>>>(
                            dV, dE, dW, n, r_done, r_end, g->outw.as<double>(), hkey, hval, serial_rows,
                            serial_count, long_rows, long_count, segs);
                    } else {
                        k_out_degree<<<grid_for((int64_t)(r_end - r_done) * 32), kThreads, 0, s>>>(
                            dV, dE, n, r_done, r_end, g->outw.as<double>(), hkey, hval, segs);
                    }
                    k_out_weight_long<<<148 * 8, kThreads, 0, s>>>(dV, dE, dW, n, long_rows, long_count,
                                                                   g->outw.as<double>(), hkey, hval, serial_rows,
                                                                   serial_count, segs);
                    r_done = r_end;
                }
                if (b > a)
                    k_in_degree_keys<<<grid_for(b - a), kThreads, 0, s>>>(dE, a, b, n, indeg, keys);
                if (b > a && W) k_weight_bits<<<grid_for(b - a), kThreads, 0, s>>>(dW, a, b, wbits);
            }
            if (sc) {
                if (rc) cudaStreamSynchronize(sc);
                cudaStreamDestroy(sc);  // released once its copies are done
            }
            for (cudaEvent_t e : ev)
                if (e) cudaEventDestroy(e);
            if (rc) return rc;
            if (dW && n > 0)
                k_out_weight_serial<<<grid_for(n), kThreads, 0, s>>>(dV, dE, dW, n, serial_rows, serial_count,
                                                                     g->outw.as<double>());
        }
        if ((rc = exclusive_scan_u32(indeg, reinterpret_cast<uint32_t*>(g->in_row.as<int32_t>()), (int64_t)n + 1, s)))
            return rc;
        k_dangling<<<grid_for(n), kThreads, 0, s>>>(g->outw.as<double>(), hkey, n, g->dangling01.as<int32_t>(), counts);
        int32_t nnz32 = 0;
        unsigned long long hc[3] = {0, 0, 0};
        if ((rc = cuda_ok(cudaMemcpyAsync(&nnz32, g->in_row.as<int32_t>() + n, sizeof(int32_t), cudaMemcpyDeviceToHost, s), "D2H nnz")) ||
            (rc = cuda_ok(cudaMemcpyAsync(hc, counts, sizeof(hc), cudaMemcpyDeviceToHost, s), "D2H counts")) ||
            (rc = cuda_ok(cudaStreamSynchronize(s), "preparation")))
            return rc;
        g->nnz = nnz32;
        g->n_dangling = (int32_t)hc[0];
        g->n_dangling_solve = (int32_t)hc[1];
        g->nsrc = (int32_t)hc[2];
        const int64_t nnz = g->nnz;
        const size_t pad = 16 * sizeof(int32_t);
        if ((rc = g->in_col.alloc((size_t)std::max<int64_t>(nnz, 1) * sizeof(int32_t) + pad)))
            return rc;
        if (W && (rc = g->in_w.alloc((size_t)std::max<int64_t>(nnz, 1) * sizeof(float) + pad)))
            return rc;
        if (m > 0) {
            // keys are destinations in [0, n), and n for an out-of-range one:
            // the key width covers n only when such an entry exists
            const uint64_t kmax = nnz < m ? (uint64_t)n : (uint64_t)n - 1;
            int bits = 0;
            while (bits < 32 && (kmax >> bits) != 0) ++bits;
            bool alt = false;
            if ((rc = radix_sort_pairs(keys, vals, keys2, vals2, m, bits, s, tmp, &alt, true, wbits, wbits2)))
                return rc;
            if (alt) {
                std::swap(keys, keys2);
                std::swap(vals, vals2);
                std::swap(wbits, wbits2);
            }
            if (nnz > 0 && (rc = cuda_ok(cudaMemcpyAsync(g->in_col.p, vals, (size_t)nnz * sizeof(int32_t),
                                                         cudaMemcpyDeviceToDevice, s), "inbound sources")))
                return rc;
            if (W && nnz > 0 &&
                (rc = cuda_ok(cudaMemcpyAsync(g->in_w.p, wbits, (size_t)nnz * sizeof(float),
                                              cudaMemcpyDeviceToDevice, s), "inbound weights")))
                return rc;
        }
        // the out-degree ranking (classes, then vertex ids)
        bool ralt = false;
        if ((rc = g->rank.alloc((size_t)n * sizeof(int32_t))) ||
            (rc = radix_sort_pairs(hkey, hval, hkey2, hval2, n, 8, s, tmp, &ralt, false)))
            return rc;
        const uint32_t* ranked = ralt ? hval2 : hval;
        k_ranks<<<grid_for(n), kThreads, 0, s>>>(ranked, n, g->nsrc, g->rank.as<int32_t>());
        // both layouts read the destination-sorted entries, the sweep's last
        // (its sort overwrites them)
        if (bins_wanted(n, nnz) && (rc = build_bin_layout(g, keys, ranked, tmp, s))) return rc;
        if ((rc = build_sweep_layout(g, vals, keys, wbits, vals2, keys2, wbits2, tmp, s))) return rc;
    }
    cudaEventRecord(g->ev1, s);
    if ((rc = cuda_ok(cudaStreamSynchronize(s), "preparation"))) return rc;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    g->prep_seconds = ms * 1e-3;
    (void)t0;
    return EGPR_SUCC;
}

int export_in_col(const egpr_graph* g, int32_t* host, cudaStream_t s) {
    if (g->nnz <= 0) return EGPR_SUCC;
    return cuda_ok(cudaMemcpyAsync(host, g->in_col.p, (size_t)g->nnz * sizeof(int32_t), cudaMemcpyDeviceToHost, s),
                   "D2H in_col");
}

}  // namespace egpr
