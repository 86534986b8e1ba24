// Internal helpers and device layouts shared by the libgpr translation units.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "gpr.h"

namespace gpr {

// Thread-local message of the last failure (gpr_last_error).
void set_error(const char *fmt, ...);

// Device allocation that records ENOMEM / ECUDA in the error slot.
int dmalloc(void **p, size_t bytes, const char *what);
template <typename T>
int dalloc(T **p, size_t count, const char *what) {
  return dmalloc(reinterpret_cast<void **>(p), (count ? count : 1) * sizeof(T), what);
}
void dfree(void *p);

// While an instance lives, dfree on this thread only records the pointers;
// the destructor frees them.  A freed block is handed out again behind a device
// synchronisation, so code that overlaps a copy on one stream with work on another
// holds one until both streams are done.
class DeferFrees {
 public:
  DeferFrees();
  ~DeferFrees();
  DeferFrees(const DeferFrees &) = delete;
  DeferFrees &operator=(const DeferFrees &) = delete;

 private:
  std::vector<void *> list_;
  std::vector<void *> *prev_;
};

// True if `p` is device (or managed) memory of the current context.
bool is_device_ptr(const void *p);

// Copies `bytes` from a host-or-device pointer into a fresh device buffer,
// or returns the pointer itself (owned = false) when it is already on the
// device.
int to_device(const void *any, size_t bytes, void **dev, bool *owned,
              cudaStream_t st, const char *what);

// ---------------------------------------------------------------------------
// Pull-graph layout after relabelling vertices by descending in-degree.
//
//   new row i  <->  old vertex perm[i]
//   rows [0, n_long)      in-degree > chunk_min: CSR whose row starts are
//                         16-byte aligned, each row cut into chunks of
//                         `chunk` edges (one warp per chunk)
//   rows [n_long, n_nz)   1 <= in-degree <= chunk_min: SELL-32 slices in
//                         width classes.  A class gives every row w lanes
//                         (w = 32, 16, 8, 4, 2, 1, widest first), w being the
//                         smallest power of two with ceil(deg / w) <= lane_max;
//                         a slice holds 32/w consecutive rows, column-major:
//                         element (j, lane) = edge j*w + (lane % w) of row
//                         lane / w.  With w = 1 a lane sums its row in the
//                         original CSR order.
//   rows [n_nz, m)        in-degree 0
//
// Every padding entry of either edge array holds the sentinel index m, whose
// contribution slot is kept at 0.
// ---------------------------------------------------------------------------
constexpr int kMaxCls = 6;

struct PrClasses {
  int n_cls = 0;
  int lw[kMaxCls] = {0};          // log2(lanes per row) of each class
  int row[kMaxCls + 1] = {0};     // first row of each class; row[n_cls] = n_nz
  int slice[kMaxCls + 1] = {0};   // first slice of each class; slice[n_cls] = n_slices
};

struct PrLayout {
  int m = 0;
  long long nnz = 0;
  int n_long = 0, n_nz = 0;
  int lane_max = 0, chunk_min = 0, chunk = 0;
  int n_chunks = 0, n_slices = 0, n_zblk = 0;
  int max_row_chunks = 0;         // chunks of the longest row
  PrClasses cls;
  int *perm = nullptr;            // [m] new -> old
  int *outdeg = nullptr;          // [m] out-degree in new order
  long long *long_ptr = nullptr;  // [n_long+1] padded offsets into long_col
  int *long_col = nullptr;        // relabelled sources of the long rows
  int *row_cbeg = nullptr;        // [n_long+1] first chunk of each long row
  int *chunk_row = nullptr;       // [n_chunks] row of each chunk
  int4 *chunk_desc = nullptr;     // [n_chunks] {row, first edge / 4, edges, first chunk of the
                                  // row or -1 when it has one}: one load per chunk
  long long *slice_ptr = nullptr; // [n_slices+1] offsets into sell_col
  int *sell_col = nullptr;        // relabelled sources, SELL-32 column-major
  int *csr_ptr = nullptr;         // [m+1] relabelled CSR (batched solvers only)
  int *csr_col = nullptr;         // [nnz]
  long long long_elems = 0, sell_elems = 0;
  long long device_bytes = 0;
};

// Class of slice s (classes are few; the scan is warp-uniform).
__host__ __device__ inline int slice_class(const PrClasses &c, int s) {
  int k = 0;
  while (k + 1 < c.n_cls && s >= c.slice[k + 1]) ++k;
  return k;
}

// Work packets: cuts units 0..n_units-1 (device costs `cost`, which the scan
// leaves unchanged) into runs of consecutive units of about equal total cost,
// about `want` of them; a unit costlier than the target is a packet alone.
// *pk_out (device, npk + 1 entries) receives the first unit of each packet and
// n_units last.  Synchronizes `st`.
int make_packets(long long *cost, int n_units, long long want, int **pk_out, int *npk_out,
                 cudaStream_t st);

// Relabelled layout of a pull graph.  When col_ready is given, d_col may
// still be arriving (a copy recorded on another stream): the build does all
// that needs only the row offsets and out-degrees first, then waits for the
// event and checks the column range before reading columns.
int build_pr_layout(int m, long long nnz, const int *d_rowptr, const int *d_col,
                    const int *d_outdeg, int lane_max, int chunk_min, int chunk,
                    bool keep_csr, PrLayout *L, cudaStream_t st, cudaEvent_t col_ready = nullptr);
void free_pr_layout(PrLayout *L);

// Destination-blocked, source-ordered layout of the rows [n_long, n_nz) of a
// PrLayout (gpr_blocked.cu describes the storage).
constexpr int kRunWords = 512;        // most entry words of one run (a warp's unit)
constexpr int kTileRuns = 1 << 16;    // most runs in one tile
constexpr int kBlockedRows = 12288;   // rows per block (accumulators in shared memory)
constexpr int kBlockedMaxRows = 12288;
constexpr int kTileWordsDefault = 1 << 20;
// GPR_FORM_AUTO picks the blocked form from this many edges up
constexpr long long kBlockedAutoMinEdges = 3LL << 24;

struct BlockedLayout {
  int R = 0, tile_slots = 0;
  int run_words = 0;  // most entry words per run: 128 x the kernel's index loads per lane
  int row0 = 0;      // first blocked row; rows [0, row0) are summed in chunks
  int n_chunks = 0;  // chunks of rows [0, row0): a prefix of the exact-order chunks
  int n_blocks = 0, n_tiles = 0;
  long long n_runs = 0, slots = 0, edges = 0;
  unsigned *entry = nullptr;             // [slots]
  uint2 *runs = nullptr;                 // [n_runs] {first word, segment << 16 | words}
  int4 *tiles = nullptr;                 // [n_tiles] {block, run0, run1, residual slot}
  int4 *blocks = nullptr;                // [n_blocks] {row0, nrows, tiles, row range}
  std::vector<int> range_tiles;          // [ranges + 1] residual slots of each row range
  unsigned long long *gacc = nullptr;    // [gacc_rows] sums of multi-tile blocks, rows row0 on
  long long gacc_rows = 0;
  int *bcnt = nullptr;                   // [n_blocks] tiles done in the current sweep
  long long device_bytes = 0;
};

// Fixed-point exponent S of the blocked form for a solve whose sweeps hold a total
// |score| of at most b0 (a sweep maps total mass M to at most (1-d) + d*M, so the
// larger of 1 and the initial mass bounds them all): a row's sum is at most that, so
// |sum| * 2^S < 2^63 needs S <= 62 - log2(b0), blocked_cap.  Within that, S puts a
// typical contribution (about b0 / nnz) near 2^28, so most fit the low 32-bit word of
// the accumulator; S >= 31 unless b0 > 2^31.
inline int blocked_cap(double b0) { return 62 - (int)ceil(log2(b0)); }

inline int blocked_shift(long long nnz, double b0) {
  const int pref = (int)floor(log2(std::max(1.0, (double)nnz) / b0)) + 28;
  return std::min(blocked_cap(b0), std::max(31, pref));
}

// The S from which on the rounding to 2^-S is lost in a score's own FP32 rounding:
// the roundings of a row of k contributions add up to about sqrt(k / 12) * 2^-S, and
// no score of a sweep from scores >= 0 is below the base (1-d) / m.  With the mean
// in-degree for k, that error is a quarter of 2^-24 of the base; rows of more
// in-edges hold more than the base.  No S is enough for d = 1.
inline double blocked_bits(int m, long long nnz, double d) {
  return 24.0 + log2((double)m / (1.0 - d)) + 0.5 * log2(std::max(1.0, (double)nnz / m));
}

constexpr int kSumBlocks = 256;  // CTAs of k_sum_abs

// The shared-memory carveout is a preference of a kernel, not of a launch: whoever sets
// it holds this until the launch (or the occupancy query) that it is for is made, so
// that handles with other block sizes on other threads do not come between.
std::mutex &carveout_mutex();

// Rows of the blocked form that stay chunked: the first *row0 rows of the
// exact-order layout's chunked rows [0, L.n_long), either those with more than
// long_min in-edges or, when long_min is 0, those with more than `least` that hold
// more than 1/8 of the in-edges of the R rows that start at them; and their
// *n_chunks chunks.
// Synchronizes st.
int blocked_split(const PrLayout &L, const int *d_rowptr, int long_min, int least, int R,
                  int *row0, int *n_chunks, cudaStream_t st);
int build_blocked_layout(int m, long long nnz, const int *d_rowptr, const int *d_col,
                         const PrLayout &L, int row0, int n_chunks, int R, int tile_slots,
                         int run_words, int workers, BlockedLayout *B, cudaStream_t st);
// The same for several row ranges of the relabelled order (perm: new -> old),
// ascending and disjoint (one per graph of a batch): blocks never span two
// ranges; blocks[b].w is the block's range, tiles[t].w the tile's residual
// slot, numbered range by range (B->range_tiles).
int build_blocked_ranges(int m, long long nnz, const int *d_rowptr, const int *d_col,
                         const int *d_perm, const std::vector<int> &rb,
                         const std::vector<int> &re, int R, int tile_slots, int run_words,
                         int workers, BlockedLayout *B, cudaStream_t st);
// CTAs per SM of the blocked kernel for blocks of R rows: two 512-thread CTAs
// when both fit beside an L1 of about half the SM's 256 KB, else one of 1024.
inline int blocked_ctas_per_sm(int R) { return R <= 8192 ? 2 : 1; }
void free_blocked_layout(BlockedLayout *B);

// Validates a device CSR (rowptr[0] = 0, monotone, rowptr[m] = nnz, every
// column in [0, ncols) when d_col is given) and, when d_outdeg is given,
// out-degrees >= 0.  validate_cols checks the columns alone.
int validate_csr(int m, long long nnz, int ncols, const int *d_rowptr,
                 const int *d_col, const int *d_outdeg, cudaStream_t st);
int validate_cols(long long nnz, int ncols, const int *d_col, cudaStream_t st);

// ---------------------------------------------------------------------------
// SpMV layout.  Rows with more than sell_max entries are long rows handled in
// chunks (listed in long_rows); every other row sits in a SELL-32 slice, one
// lane per row, with its own length.
//   even lengths   rows in natural order (x and y locality of a stencil):
//                  lane l of slice s is row 32 s + l, sell_len[row] its
//                  length (255: long row, the lane is idle)
//   ragged         (natural slices would be padded by more than 1/8, or a few long
//                  chunks would end late: kSpmvWarps) rows
//                  sorted by descending length inside windows of kSpmvWindow
//                  rows: slot_row[slot] is the row (-1: none), sell_len[slot]
//                  its length.  When enough entries fall on few columns, the
//                  `hot` most frequent columns are listed in hot_col and an
//                  entry of column hot_col[h] stores ~h instead of the column.
// ---------------------------------------------------------------------------
struct SpmvLayout {
  int m = 0;
  long long nnz = 0;
  int sell_max = 0, chunk = 0;
  int n_long = 0, n_chunks = 0, n_slices = 0;
  int *long_rows = nullptr;        // [n_long] row ids, ascending
  long long *long_ptr = nullptr;   // [n_long+1] padded offsets
  int *long_col = nullptr;
  float *long_val = nullptr;
  int *row_cbeg = nullptr;         // [n_long+1]
  int *chunk_row = nullptr;        // [n_chunks] index into long_rows
  long long *slice_ptr = nullptr;  // [n_slices+1]
  int *sell_col = nullptr;
  float *sell_val = nullptr;
  unsigned char *sell_len = nullptr;  // [32 n_slices] (even: rows, ragged: slots)
  bool ragged = false;
  int *slot_row = nullptr;         // [32 n_slices], ragged only
  int *slice_at = nullptr;         // [n_slices+1] slice_ptr / 32, ragged only
  int4 *chunk_desc = nullptr;      // [n_chunks], ragged only: {row, first entry / 4, entries,
                                   // index into long_rows or -1 when the row has one chunk}
  int hot = 0;                     // columns staged in shared memory
  int *hot_col = nullptr;          // [hot]
  long long long_elems = 0, sell_elems = 0;
  long long device_bytes = 0;
};

constexpr int kSpmvWindow = 1024;  // rows sorted together in a ragged layout
// Matrices with long rows (over 1/8 of the entries) that are not uneven otherwise take
// the ragged layout where the chain of loads of one chunk is what k_spmv ends on: the
// mean chunk is at least a warp's share of all entries (148 SMs x 32 warps) and long
// enough to take several rounds of k_spmv's 128 entries.  Else k_spmv is faster, whose
// many light CTAs stream at the memory's rate.  k_spmv_rag / k_spmv, us, rows of k even
// entries at random columns: 2M entries, k = 130 20.5 / 18.4, 300 18.5 / 14.3, 700 16.4 /
// 16.4, 1000 16.4 / 18.4, 5000 24.6 / 41.0; 8M, 700 30.7 / 28.7, 1000 28.1 / 24.6, 2000 24.6 /
// 30.8; 16M, 65 180 / 113, 1000 43 / 41, 5000 61 / 47; 40M, 81 349 / 241.  27-point stencil
// on 64^3 with 2,000 rows of 1,000: 32.8 / 26.6, with 64 of 30,000: 36.9 / 49.2.
constexpr int kSpmvWarps = 4736;
constexpr int kSpmvLongChunk = 640;
constexpr int kSpmvHotMax = 16384;
// hot_columns: look for columns to stage in shared memory (a histogram and a sort
// of the columns; worth it for a matrix that is multiplied more than once).
int build_spmv_layout(int m, long long nnz, const int *d_Ap, const int *d_Aj,
                      const float *d_Ax, int sell_max, int chunk, bool hot_columns,
                      SpmvLayout *L, cudaStream_t st);
void free_spmv_layout(SpmvLayout *L);

}  // namespace gpr

#define GPR_CUDA(call)                                                        \
  do {                                                                        \
    cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) {                                                  \
      gpr::set_error("%s:%d: %s: %s", __FILE__, __LINE__, #call,             \
                     cudaGetErrorString(e_));                                 \
      return GPR_ECUDA;                                                       \
    }                                                                         \
  } while (0)

namespace gpr {
// Status of one CUDA call, for code that must release buffers before it
// returns (GPR_CUDA returns at once): GPR_OK, or GPR_ECUDA with the error set.
inline int cuda_status(cudaError_t e, const char *file, int line, const char *what) {
  if (e == cudaSuccess) return GPR_OK;
  set_error("%s:%d: %s: %s", file, line, what, cudaGetErrorString(e));
  return GPR_ECUDA;
}
}  // namespace gpr
#define GPR_CUDA_RC(call) gpr::cuda_status((call), __FILE__, __LINE__, #call)

#define GPR_TRY(call)                                                         \
  do {                                                                        \
    int s_ = (call);                                                          \
    if (s_ != GPR_OK) return s_;                                              \
  } while (0)

// Device-resident pull graph behind the opaque gpr_graph handle.
struct gpr_graph {
  int device = 0;
  gpr::PrLayout L;
  float *s = nullptr;        // [m] scores, new order
  float *c0 = nullptr;       // [m+1] contributions (sweep parity 0 input)
  float *c1 = nullptr;       // [m+1]
  float *partial = nullptr;  // [n_chunks] partial sums of long-row chunks
  int *cnt = nullptr;        // [n_long] arrival counters of multi-chunk rows
  double *cta_err = nullptr; // [2 * max grid] per-CTA residual partials
  double *err_hist = nullptr;// [err_cap] residual of every sweep
  unsigned *bar = nullptr;   // [4] grid barrier: arrivals, generation
  int *status = nullptr;     // [8] error flags, sweeps done, done flag, launches, last
                             // residual (double)
  float *scores_tmp = nullptr; // [m] device copy of host scores
  double *res_tmp = nullptr;   // [m+1+n_long] FP64 residual scratch
  int err_cap = 0;
  int last_sweeps = 0;
  int hot = 0;                 // FP32 contributions staged in shared memory per sweep
  int hot_bytes = 0;           // shared-memory budget of the hot prefix
  int grid_hot[12] = {0};      // cooperative grid of each persistent sweep kernel
  void *h0 = nullptr, *h1 = nullptr;  // BF16 contributions of the mixed form (on first use)
  int *wq = nullptr;           // [2] chunk-queue heads of the blocked form
  bool hot_ok = false;         // every hot-kernel variant is co-resident at grid_hot
  int grid_step = 0, max_grid = 0;
  bool coop = false;
  cudaStream_t st = nullptr;
  bool own_stream = false;
  cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr, e3 = nullptr;
  // Chunk table of the batched solver (rows above b_dmax in-edges cut into
  // b_chunk-edge chunks), built on first use for a given (b_dmax, b_chunk).
  int *b_cbeg = nullptr, *b_crow = nullptr;
  int b_nlong = -1, b_nchunks = 0, b_dmax = 0, b_chunk = 0;
  // Chunk descriptors (int4 per chunk) and the packet table (first unit of
  // each of b_npk packets), rebuilt with the chunk table or for another
  // packet count b_pk_want.
  void *b_cdesc = nullptr;
  int *b_pk = nullptr;
  int b_npk = -1;
  long long b_pk_want = 0;
  // Packet tables of the narrower layouts a batched solve packs its
  // still-updating vectors into, by log2 of the rows per row group.
  int *b_pkr[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  int b_npkr[6] = {-1, -1, -1, -1, -1, -1};
  long long b_pkwr[6] = {0, 0, 0, 0, 0, 0};
  // Push solver without blocks: edges sorted by source and the per-vertex
  // accumulators, built on first use.
  int *push_src = nullptr, *push_dst = nullptr;
  float *push_sum = nullptr;
  // Graph mode: the instantiated sweep-loop graph and the kernel and
  // arguments it was built for.
  cudaGraph_t loop_graph = nullptr;
  cudaGraphExec_t loop_exec = nullptr;
  int loop_ki = -1;
  // Blocked form (GPR_LAYOUT_BLOCKED): its layout, the persistent kernel's
  // grid and co-residency, the tile-queue heads and the largest |score|.
  gpr::BlockedLayout B;
  bool has_blocked = false, blocked_ok = false;
  bool has_push = false;       // B was built by the push solver (pull solves do not use it)
  bool push_checked = false;   // the push solver has compared edges and out-degrees
  bool push_plain = false;     // the push solver does not use B: more edges than an
                               // out-degree says, or B could not be built
  int grid_blocked = 0, blocked_ctas = 1;  // blocked-form CTAs: total, per SM
  int blocked_carve = 0;       // shared-memory share of the SM for them, percent
  int *tq = nullptr;
  unsigned *fx_max = nullptr;
  double *fx_part = nullptr;   // per-CTA sums of |score| (k_sum_abs)
  alignas(8) unsigned char loop_args[512] = {0};
};

namespace gpr {
// The push solver's solve in the blocked form (gpr_pagerank.cu).  kPushFallback: the
// form does not apply (a non-finite score, too much mass for its precision, no
// co-resident grid); nothing was done.
constexpr int kPushFallback = 101;
int push_blocked(gpr_graph *g, float *any_scores, const gpr_pr_opts &opts, gpr_pr_stats *stats);

constexpr int kZeroRowsPerUnit = 128;  // rows per zero-in-degree work unit
constexpr int kSellMaxDefault = 64;    // SpMV: row length bound of the SELL bin;
                                       // PR: max edges per lane in a SELL slice
constexpr int kChunkMinDefault = 4096; // PR: rows with more in-edges are chunked
constexpr int kChunkDefault = 4096;    // edges per long-row chunk (multiple of 128)
constexpr int kBlock = 256;            // threads per CTA of the per-sweep kernels
constexpr int kHotDefault = 32768;     // contributions staged in shared memory (128 KB)
constexpr int kHotMin = 4096;
constexpr int kHotMax = 56832;         // 222 KB: the most one CTA may take

// Defaults of the chunk size (and of the in-degree above which rows are chunked)
// and of the staged prefix for a graph of nnz edges.  A chunk is about one warp's
// share of the edges (148 SMs x 32 warps), so that no warp works on its chunk while
// the others are done; below 2^19 edges a sweep is a few dependent loads, and the
// chunks' combination costs more than it saves.  Sweep loop, RMAT, chunks of 512 /
// 1024 / 2048 / 4096 edges: 10,007 vertices (0.11M edges) 101 / - / - / 91 us, 65,536
// (0.95M) 236 / 238 / - / 293, 250,007 (3.8M) 678 / 658 / - / 777, 1,000,003 (15M)
// 2078 / 1751 / 1743 / 1806, 3,000,017 (31M) 4293 / 3821 / 3781 / 3771.  Staging costs
// every SM the prefix once a sweep: 65,536 vertices with 4096 / 16384 / 32768 staged
// 208 / 212 / 238 us, 250,007 770 / 729 / 764; 10,007 with 4096 / all staged 168 / 160 us
// per call.  Other graphs, 20 sweeps, 4096 and 32768 against these defaults: Chung-Lu
// (exponent 2.1) of 65,536 vertices 275 / 179 us, 250,007 350 / 289, 1,000,003 753 / 765,
// 2,500,009 1796 / 1801; Erdos-Renyi of 40,000 158 / 162, 65,536 187 / 183, 250,007 402 / 396,
// 1,000,003 1344 / 1340.
inline int default_chunk(long long nnz) {
  if (nnz < (1 << 19)) return kChunkDefault;
  int c = 512;
  while (c < kChunkDefault && 2LL * c * 4736 <= nnz) c *= 2;
  return c;
}
inline int default_hot(long long nnz) {
  if (nnz < (1 << 19)) return kHotDefault;
  const long long h = nnz / 200 / 4 * 4;
  return (int)(h < kHotMin ? kHotMin : h > kHotDefault ? kHotDefault : h);
}

__host__ __device__ inline long long ceil_div(long long a, long long b) {
  return (a + b - 1) / b;
}

// Sweeps the reference's loop counts on a graph with no vertices
// (src/pr/omp_base.cc:23-43): every sweep's residual is 0, so the loop stops
// after the first sweep when 0 < tol and runs to max_iter otherwise.
inline int empty_graph_sweeps(double tol, int max_iter) {
  return max_iter <= 0 ? 0 : (0.0 < tol ? 1 : max_iter);
}
}  // namespace gpr
