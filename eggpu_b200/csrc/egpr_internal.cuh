// Internal declarations shared by the CUDA translation units of libegpr.so.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/egpr.h"
#include "sweep_cut.h"

namespace egpr {

// ---------------------------------------------------------------------------
// Layout of the single-vector sweep.
//
// A random 4-byte read that misses L1 costs an SM one 32-byte sector from L2,
// and an SM receives about one sector per clock (measured on B200: 289 G such
// reads/s over all SMs, from any vector that fits L2), while shared memory
// serves 11 random reads per clock.  So no carried value is gathered from
// global memory:
//   * sources (vertices with out-edges) are ranked by out-degree and cut into
//     blocks of kBlockSrc; the carried values z are stored in rank order, so a
//     block's values are one contiguous piece that a CTA stages in shared memory;
//   * the inbound entries are ordered by (block, destination); each is a 16-bit
//     index into its block;
//   * phase 1 (k_gather) sums every run of entries of one (block, row) into a
//     "pair", written in order; phase 2 (k_rows) adds the pairs of each row
//     from all blocks in shared memory and finishes the row.
// Ranking by degree packs the entries into few runs: R-MAT scale 22 has 0.17
// pairs per entry (0.30 with blocks in vertex order).
//
// A graph with too many (block, row tile) cells for the list of steps (about
// 3 * 10^8 vertices and more) is laid out as one block of any size whose values are
// read from global memory (32-bit ranks instead of 16-bit indices).
// ---------------------------------------------------------------------------
constexpr int kThreads = 256;  // threads of the preparation and helper kernels

// Span flags of the batched solve's chunks (spmm.cu).
constexpr int32_t kHasHead = 1;    // the chunk's first row began in an earlier chunk
constexpr int32_t kHasTail = 2;    // the chunk's last row continues into a later chunk
constexpr int32_t kInterior = 4;   // the chunk lies inside one row (head and tail are that row)

// Sources per block: FP64 values of one block (176 KB, the correction sweep) and
// a tile of row sums per warp (48 KB) fill the shared memory of an SM.
constexpr int32_t kBlockSrc = 22528;
constexpr int kBlockBits = 15;     // bits of an index inside a block (kBlockSrc itself is the zero slot)
// Warp tiles of kTileItems entries, lane l owning entries 8l..8l+7.  A block's
// entries are padded to whole tiles with zero-slot entries.  A warp walks chunks of
// 2^chunk_shift tiles (counted from the block's first one); a run never leaves its
// chunk (a longer one becomes several pairs), so chunks are independent.
constexpr int kLaneItems = 8;
constexpr int kTileItems = 32 * kLaneItems;
static_assert(kTileItems == kCutTileEntries, "the cutting counts the layout's tiles");
// Per tile and lane one 16-bit word: the lane's run-end marks (low byte) and the
// number of marks in the lanes below it (high byte); 64 bytes per tile.
constexpr int kTileWords = 16;
// Row tiles of phase 2: runs of whole 32-row groups of about equal cost, at most
// kMaxTileRows rows, summed in one CTA's shared memory.
constexpr int kRowGroup = 32;
constexpr int32_t kMinTileRows = 256;    // wanted at least (fewer where rows are heavy)
constexpr int32_t kMaxTileRows = 12288;  // 96 KB of FP32 sweep sums (two CTAs per SM), 192 KB of FP64 ones
constexpr int kRowTilesPerSm = 2;        // CTAs of phase 2 that an SM holds
constexpr int kStepPairs = 128;          // pairs of one block that a warp adds at a time

// Per-graph device view used by the sweep kernels.
struct GraphDev {
    const uint16_t* idx;        // per padded entry: index of its source in the block (kBlockSrc: none)
    const int32_t* idx32;       // one-block layout without staging: rank of the source (-1: none); else NULL
    const float* w;             // weights of the padded entries, NULL = unit weights
    const uint32_t* tile_bits;  // per tile: kTileWords words (run-end marks, per-lane mark offsets)
    const int32_t* tile_pair;   // per tile: its first pair (ntiles + 1)
    const uint16_t* pair_row;   // per pair: its row in its row tile
    const int32_t* row_step;    // first step of each row tile (one more than there are row tiles)
    const int2* steps;          // (first pair, pairs): up to kStepPairs pairs of one block and row tile
    const int32_t* row_tile;    // first row of each row tile (one more than there are row tiles)
    void* pairs;                // per pair: its sum (FP32, or FP64 in the correction sweep)
    const double* outw;      // n, FP64 out-weight sums
    const int32_t* rank;     // n, rank of each source, -1 for a vertex without out-edges
    const double* scale;     // n, alpha/outw, 0 for a dangling vertex
    const float* tele;       // n, personalisation (NULL = uniform)
    float* x[2];             // ranks, double-buffered
    float* z[2];             // by source rank: x * alpha/outw, the value each out-edge carries
    double* out;             // n, FP64 result
    double* z64;             // by source rank: FP64 carried values for the correction sweep
    int32_t n;
    int32_t nsrc;            // ranked sources
    int32_t nblocks;
    int32_t chunk_shift;
};

struct GraphState {
    double alpha;
    double c1;         // (1 - alpha) / n
    double tol_n;      // tol * n
    double dmass;      // alpha * (dangling mass) / n for the next sweep
    double dmass_prev; // the value used by the last completed sweep
    double residual;   // L1 of the last sweep
    double residual64; // L1 of the FP64 correction sweep against x_{k-1}
    double xsum;       // sum of the last sweep's ranks (FP64 sweep: of the result)
    double dsum;       // dangling mass of the last sweep's ranks
    int32_t iter;
    int32_t max_iter;
    int32_t done;
    int32_t converged;
    int32_t personalised;  // teleport from GraphDev::tele instead of 1/n
};

struct Ctl {
    uint32_t queue;    // work-queue head
    uint32_t exited;   // CTAs that left the queue loop
    int32_t active;    // graphs still iterating
    int32_t launches;  // sweep launches so far
    int32_t cap;       // hard cap on sweep launches
    int32_t error;
};

constexpr int kAccWords = 8;  // words per accumulator slot (6 used; 64-byte slots)

struct SweepParams {
    const GatherUnit* units;
    const int32_t* cta_unit;       // per phase 1 CTA: its first unit (grid + 1)
    const int2* row_tiles;         // (graph, row tile), in row order
    int32_t nrow_tiles;
    int32_t max_rows;              // of a row tile in the plan: the size of a CTA's row sums
    const GraphDev* graphs;
    GraphState* states;
    // FP64 sums are accumulated as two's-complement fixed point (2 words: units
    // of 2^-32 and of 2^-64) with integer atomics, so their order does not
    // change the result.
    unsigned long long* acc;       // kAccWords per slot: err, dangling, rank sums
    int32_t acc_sub;               // accumulator slots per graph
    Ctl* ctl;
    cudaGraphConditionalHandle cond;
    int32_t use_cond;
    int32_t ngraphs;
};

// ---- device buffers --------------------------------------------------------
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    int dev = -1;         // device of the allocation
    bool pooled = false;  // from device_pool() (else cudaMalloc)
    int alloc(size_t b);
    void release();
    // Stream-ordered forms for buffers used by one stream only: grow_on keeps
    // a large enough buffer and otherwise frees and allocates in the order of
    // stream s; neither waits for the device.
    int grow_on(size_t b, cudaStream_t s);
    void release_on(cudaStream_t s);
    template <typename T>
    T* as() const { return static_cast<T*>(p); }
};

// ---- the work plan over one or more prepared graphs -------------------------
struct Plan {
    int32_t ngraphs = 0;
    int32_t grid = 0;        // CTAs of phase 1
    int32_t row_grid = 0;    // CTAs of phase 2
    int32_t nrow_tiles = 0;
    int32_t max_rows = 0;    // of a row tile
    int32_t max_n = 0;
    DevBuf d_units, d_cta_unit, d_row_tiles, d_graphs, d_states, d_ndang, d_ctl, d_acc;
    int32_t nacc = 0;                 // accumulator slots
    // the sweeps as a CUDA graph, without and with the watch for small row sums (sweep.cu)
    struct Loop {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        bool failed = false;
    } loops[2];
    ~Plan();
    void release_loops();
    void release();
    void release_on(cudaStream_t s);  // buffers used by stream s only: freed in its order
};

struct SpmmWork;  // batched personalised PageRank workspace (spmm.cu)

// ---------------------------------------------------------------------------
// The binned single-graph sweep (bins.cu; layout built in prep.cu).
//
// Vertices are renumbered: first the H sources of largest out-degree (the hub
// block, whose carried values the sweep stages in shared memory, so a source
// id below H is a shared-memory read), then every other vertex; inside each
// block vertices go by descending in-degree.  The inbound CSR in that order
// keeps, per row, the entries in ascending original-source order.  Rows of
// one length class are then contiguous, and the work queue holds:
//   kBinPiece  a piece of a long row (>= bin_piece entries), one warp; a row cut
//              into several pieces is finished by the last piece to arrive
//              (pieces add exact fixed-point sums)
//   kBinGroup  rows [r0, r1) of one length class, G lanes per row with G a
//              power of two sized so that each lane gathers 4..8 entries
//   kBinEmpty  rows [r0, r1) without inbound entries (teleport and dangling
//              terms only)
// ---------------------------------------------------------------------------
constexpr int32_t kBinPiece = 0;
constexpr int32_t kBinGroup = 1;
constexpr int32_t kBinEmpty = 2;

struct BinItem {
    int32_t kind;
    int32_t r0, r1;  // rows [r0, r1); kBinPiece: r0 is the row
    int32_t e0, e1;  // kBinPiece: entries [e0, e1)
    int32_t span;    // kBinPiece: span slot of a row cut into several pieces, -1 for one piece
    int32_t parts;   // kBinPiece: pieces of the row; kBinGroup: lanes per row (G)
    int32_t pad;
};

struct BinLayout {
    int32_t n = 0;
    int32_t hubs = 0;            // hub block [0, hubs)
    int64_t nnz = 0;
    DevBuf perm;                 // n: new id of each vertex
    DevBuf inv;                  // n: vertex of each new id
    DevBuf row;                  // n + 1 (+ pad): offsets of the renumbered inbound CSR
    DevBuf col;                  // nnz (+ pad): renumbered sources
    DevBuf w;                    // nnz (+ pad): FP32 weights (weighted graphs)
    DevBuf outw;                 // n: FP64 out-weight sums, renumbered
    std::vector<int32_t> h_row_bounds;  // row offsets at the class boundaries (host copy, item building)
    // work queue
    DevBuf items;
    int32_t nitems = 0;
    int32_t nspans = 0;
    int32_t piece = 2048;        // entries per piece of a long row (tuning)
    int32_t group_entries = 4096;  // target entries of a kBinGroup item (tuning)
    // per-solve state (renumbered)
    DevBuf scale, tele, x, z, z64, out64, states, ctl, acc, span_acc, span_cnt;
    int32_t acc_slots = 0;
    int32_t grid = 0;
    cudaGraph_t cg = nullptr;
    cudaGraphExec_t cg_exec = nullptr;
    cudaGraphConditionalHandle cond = 0;
    bool cg_failed = false;
    int64_t device_bytes() const {
        int64_t b = 0;
        for (const DevBuf* d : {&perm, &inv, &row, &col, &w, &outw, &items, &scale, &tele, &x, &z, &z64, &out64, &states,
                                &ctl, &acc, &span_acc, &span_cnt})
            b += (int64_t)d->bytes;
        return b;
    }
    ~BinLayout();
};

// ---- the one-kernel solve of a small graph (small.cu) ------------------------
struct SmallState {
    // residual, dangling mass and rank sum, 2 fixed-point words each; sweep i adds
    // to set i % 3 while set (i + 1) % 3 is clear
    unsigned long long acc[3][6];
    double residual;
    int32_t iter;
    int32_t converged;
    int32_t ndang;
    uint32_t arrived;           // barrier arrivals of the running kernel
    int32_t error;
    int32_t pad;
    unsigned long long t_begin; // global timer (ns) when the solve's first kernel started
    unsigned long long t_end;   // global timer (ns) when its last CTA ended
};

// The inbound CSR (natural source ids) and out-weight sums.
struct SmallGraph {
    int32_t n;
    int64_t nnz;
    const int32_t* in_row;
    const int32_t* in_col;
    const float* in_w;       // NULL = unit weights
    const double* outw;
    const float* tele;       // teleport vector, NULL = uniform
};

struct SmallWork {
    SmallState* st;
    float* x[2];             // n each
    float* z[2];             // n each
    double* z64;             // n: the correction sweep's carried values (may lie over z)
};

// ---- prepared graph handle ---------------------------------------------------
}  // namespace egpr

struct egpr_graph {
    std::mutex mu;
    int device = -1;
    int32_t n = 0;
    int64_t m_input = 0;
    int64_t nnz = 0;
    int32_t weighted = 0;
    int32_t n_dangling = 0;        // out-weight <= 0 (reference mask)
    int32_t n_dangling_solve = 0;  // out-weight <= 1e-15 (EasyGraph CPU rule)
    double prep_seconds = 0.0;
    int32_t host_inputs_registered = 0;  // host input arrays page-locked for the upload
    int32_t host_inputs_locked = 0;      // host input arrays that were page-locked already
    int32_t host_inputs_staged = 0;      // host input arrays copied through the staging pool
    // prepared graph
    egpr::DevBuf in_row, in_col, in_w, outw, dangling01, rank;
    // the sweep's layout (see build_sweep_layout)
    egpr::DevBuf idx, sw_w, tile_bits, tile_pair, pair_row, row_step, steps, row_tile, pairs;
    int32_t nsrc = 0;              // ranked sources
    int32_t nblocks = 0;
    int32_t chunk_shift = 0;       // log2 of the tiles per chunk
    int32_t global_block = 0;      // one block, values read from global memory (idx holds 32-bit ranks)
    int32_t max_tile_rows = 0;     // rows of the largest row tile, rounded up
    std::vector<int32_t> h_block_tile;  // first tile of each block (nblocks + 1)
    std::vector<int32_t> h_block_pair;  // first pair of each block (nblocks + 1)
    int32_t nrow_tiles = 0;
    // layout parameters (egpr_tuning); defaults from the environment
    int32_t tune_cpw = 8;           // sweep: sets the row tile size (row tiles per resident warp)
    int32_t tune_rc = 4;            // sweep: cost of a pair, in entries, when phase 1 is cut into CTA shares
    int32_t tune_spmm_chunk = 0;    // batched solve: entries per work unit
    int32_t tuning_recorded = 0;    // the layout came from the persisted tuner choices
    // solve workspace
    egpr::DevBuf scale, tele, x0, x1, z0, out, z64;
    egpr::DevBuf seed_ids;         // seed set of a single-vector PPR solve
    int32_t one_kernel = 0;        // single-vector solves run as one kernel (small.cu)
    int32_t counted = 0;           // a one-kernel solve of this graph is counted as in flight
    int32_t last_one_kernel = 0;   // the last one did (also for an alpha that the sweep does not take)
    egpr::DevBuf small_state;      // its state
    egpr::DevBuf vertex_z;         // its carried values where z0 and z64 are by source rank
    egpr::Plan plan;               // single-graph plan
    egpr::SpmmWork* spmm = nullptr; // batched personalised PageRank workspace
    egpr::BinLayout* bins = nullptr; // binned single-graph sweep (null: the other paths serve single solves)
    int32_t sessions = 0;            // live batched-solve sessions (egpr_session_*) on this graph
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr; // active stream (own or user-given)
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // state of an enqueued solve
    bool pending = false;
    int32_t pending_launches = 0;
    double pending_t0 = 0.0;
    int64_t device_bytes() const;
};

namespace egpr {

// The library's memory pool of the current device: device buffers and
// preparation scratch come from it, and it keeps up to EGPR_POOL_KEEP_MB
// (default: a quarter of the device) MiB of freed memory for reuse (null if
// pools are unavailable).
cudaMemPool_t device_pool();

// Status helpers.
int set_cuda_error(cudaError_t e, const char* what);
int arg_error(const char* why);  // EGPR_INVALID_ARGUMENT with a message
bool graph_loop_enabled();       // sweeps loop in a CUDA-graph while node (EGPR_GRAPH_LOOP != 0)
int check_device(const egpr_graph* g);
double wall_seconds();

// Preparation (prep.cu).
int prepare_graph(egpr_graph* g, const int32_t* V, const int32_t* E, const double* W);
int rebuild_sweep_layout(egpr_graph* g, cudaStream_t s);  // for the graph's current layout parameters
// Destination of every inbound entry, in entry order (row offsets expanded).
void expand_rows(const int32_t* row, int32_t n, int32_t* dst, cudaStream_t s);
int default_chunks_per_warp();  // EGPR_CHUNKS_PER_WARP, else 8
int default_row_cost();         // EGPR_ROW_COST, else 4
int32_t default_spmm_chunk();   // EGPR_SPMM_CHUNK, else 0
int32_t spmm_chunk_for(int64_t entries);  // the batched solve's tile for a graph of that size
int export_in_col(const egpr_graph* g, int32_t* host, cudaStream_t s);
// D2H of a result after the work enqueued on s: a plain async copy into
// page-locked memory (or under 1 MiB); into pageable memory through the
// page-locked staging pool, returning once the bytes are in dst.
int download_d2h(void* dst, const void* src, size_t bytes, cudaStream_t s, const char* what);

// Binned single-graph sweep (bins.cu).
bool bins_wanted(int32_t n, int64_t nnz);  // build the binned layout for this graph (EGPR_BINS, size)
int32_t bin_hub_cap();                      // hub block size limit (shared memory of one CTA)
int bins_build_items(egpr_graph* g, cudaStream_t s);
int bins_alloc_solve(egpr_graph* g, cudaStream_t s);
int bins_upload_tele(egpr_graph* g, cudaStream_t s);  // renumbers g->tele into the layout's order
int bins_enqueue(egpr_graph* g, double alpha, int32_t max_iter, double tol, bool personalised, uint32_t flags,
                 cudaStream_t s, int32_t* host_launches);
int bins_read_state(egpr_graph* g, cudaStream_t s, int32_t* iterations, int32_t* converged, double* residual,
                    int32_t* launches, int32_t* error);

// Plans and sweeps (sweep.cu).
int sweep_grid();
int sweep_resident_warps();
int work_grid(int64_t entries, int full);  // CTAs of a launch over that many entries
int64_t z_stride(int32_t nsrc);    // values per parity of z (whole 16-byte units past the last block)
int plan_build(Plan& plan, egpr_graph* const* graphs, int32_t count, cudaStream_t stream);
GraphDev graph_dev_view(const egpr_graph* g);
int launch_init(Plan& plan, double alpha, int32_t max_iter, double tol, bool personalised,
                cudaStream_t stream);
// Whether rows of a solve may get nothing but their sum: then phase 2 watches for small sums.
bool rows_need_watch(const Plan& plan, double alpha, bool personalised);
int launch_loop(Plan& plan, int32_t max_iter, bool watch, cudaStream_t stream, int32_t* launches);
int launch_finish(Plan& plan, bool correction, bool watch, cudaStream_t stream, int32_t* launches);

// The one-kernel solve (small.cu).
bool small_wanted(int32_t n, int64_t nnz);  // prepared graphs it serves
// others: one-kernel solves in flight on the device beside this one.
int small_solve(const SmallGraph& graph, const SmallWork& work, double alpha, double tol, int32_t max_iter,
                bool with_correction, double* ranks, int32_t others, cudaStream_t s);
// Number of one-kernel solves in flight on a device; the callers count theirs.
std::atomic<int32_t>& small_in_flight(int device);

// SpMM personalised PageRank (spmm.cu).  A batched sweep gathers a whole
// 32-column panel per entry, about seven single-vector sweeps' worth, so
// batches of fewer columns run as single-vector solves.
constexpr int32_t kSpmmMinColumns = 6;
void spmm_work_release(egpr_graph* g);
int ppr_batch_solve(egpr_graph* g, double alpha, int32_t max_iter, double tol, int32_t k,
                    const double* teleport_dense, const int32_t* seed_ptr, const int32_t* seeds,
                    uint32_t flags, double* out, egpr_stats* stats);

// Scan / sort helpers (prep.cu), exposed for the SpMM set-up.
int exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t len, cudaStream_t s);

}  // namespace egpr
