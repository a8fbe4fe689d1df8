// knnsj_internal.h -- host-side declarations shared by the library's
// translation units (kernel launchers, pipeline, host I/O).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>
#include <vector>

#include "../../include/knnsj.h"
#include "knnsj_device.cuh"

namespace knnsj {

// ---- error plumbing ------------------------------------------------------
struct CudaError {
  cudaError_t err;
  const char* where;
};

#define KNNSJ_CUDA(call)                                                   \
  do {                                                                     \
    cudaError_t e_ = (call);                                               \
    if (e_ != cudaSuccess) throw ::knnsj::CudaError{e_, #call};            \
  } while (0)

struct StatusError {
  knnsj_status st;
  const char* what;
};

// Kernel launches of this host thread since the last reset (reported in
// knnsj_stats; batched joins run sets on several host threads).
extern thread_local unsigned long long g_launches;
// Set while a fixed-scratch join runs on this thread: any cudaMalloc-backed
// buffer, pinned host buffer or stream creation then fails with
// KNNSJ_ERR_EXCEEDS_FIXED_SCRATCH instead of allocating.
extern thread_local bool g_forbid_alloc;
#define KNNSJ_CHECK_LAUNCH()                 \
  do {                                       \
    KNNSJ_CUDA(cudaGetLastError());          \
    ++::knnsj::g_launches;                   \
  } while (0)

// Lets `kern` be launched with up to `limit` bytes of dynamic shared memory.
// The limit belongs to the kernel, not to the launch, and batched joins launch
// the same kernel from several host threads with different sizes: `limit` is
// the most any launch of the kernel asks for, so that no thread lowers it
// between another's setting and its launch (which the runtime then refuses).
template <typename F>
inline void allow_dynamic_smem(F* kern, size_t limit) {
  KNNSJ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
}

// ---- device buffers of one join (cached across calls, grow-only) --------
// A fixed device region carved out by bump allocation (no cudaMalloc).
struct Arena {
  unsigned char* base = nullptr;
  size_t cap = 0;
  size_t used = 0;
  void* take(size_t bytes);  // 256-byte aligned; throws when the region is full
};

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  Arena* arena = nullptr;  // non-null: carve from the arena instead of cudaMalloc
  void* get(size_t need);  // grows (contents not kept)
  void release();
};

// Grid index on the device, in cell order.
template <typename T>
struct DeviceGrid {
  GridGeom<T> geom;
  const T* ps = nullptr;                  // SoA coords in cell order: d x n
  const float* psf = nullptr;             // the same rounded to float (double data only)
  const uint32_t* pid = nullptr;          // original id of each sorted position
  const unsigned long long* ckeys = nullptr;  // sorted non-empty cell ids [C]
  const uint32_t* coff = nullptr;         // first sorted position of each cell [C+1]
  const uint32_t* dstart = nullptr;       // dense: first position of cell L [total+1]
  unsigned long long C = 0;
  int dense = 0;
};

// ---- kernel launchers (k_*.cu) -------------------------------------------
template <typename T>
// perm (host): input dimension of each column; soaf (optional): the columns
// rounded to float as well.
void launch_transpose_reorder(const T* aos, T* soa, float* soaf, uint64_t n, uint32_t d, const uint32_t* perm,
                              cudaStream_t s, uint32_t* d_nonfinite);
// Every `step`-th row (rows 0, step, ...; count of them), densely packed.
template <typename T>
void launch_gather_rows(const T* aos, uint64_t count, uint64_t step, uint32_t d, T* out, cudaStream_t s);
template <typename T>
void launch_minmax(const T* soa, uint64_t n, uint32_t di, T* d_minmax /*2*di*/, T* scratch /*1024*2*di*/,
                   cudaStream_t s);

// Constants of the distance histogram (k_eps.cu) for a range of buckets.
struct HistConst {
  double avg, bw;
  float inv_bw, errc, abs_q, flo, fhi, s_hi;
};
constexpr uint32_t HIST_FIRST = 256;  // buckets [0, HIST_FIRST) are counted first, the rest if need be
constexpr uint32_t HIST_BUCKETS = 10000;
struct EpsScratch {
  double* partial = nullptr;     // [eps_avg_threads * eps_avg_chunks]
  double* sample_sum = nullptr;  // [eps_avg_threads]
  double* avg_out = nullptr;     // [2]: mean distance, pair count
  uint32_t* hist = nullptr;      // [HIST_BUCKETS]
  HistConst* hc = nullptr;       // [2]: constants of the two bucket ranges
};
uint64_t eps_avg_threads(uint64_t n);
uint32_t eps_avg_chunks(uint64_t n);
uint32_t eps_sample_offset(uint64_t n);
template <typename T>
// (minmax: the columns' extremes, for the histogram's constants)
void launch_eps_avg(const T* soa, const T* minmax, uint64_t n, uint32_t d, const EpsScratch& sc, cudaStream_t s);
template <typename T>
// soaf: the columns rounded to float (float data: the columns themselves);
// range 0 or 1: which of the two bucket ranges is counted.
void launch_eps_hist(const T* soa, const float* soaf, uint64_t n, uint32_t d, const EpsScratch& sc, int range,
                     cudaStream_t s);
// Sum of squared result distances (the reference's verification figure,
// GPU.cu:3690-3693) in a fixed order; result in *d_out.
template <typename T>
void launch_checksum(const T* dists, uint64_t count, double* d_partial, double* d_out, cudaStream_t s);
// Sum of count doubles (the per-row verification sums) in a fixed order.
void launch_sum_f64(const double* v, uint64_t count, double* d_partial, double* d_out, cudaStream_t s);

struct GridScratch {
  unsigned long long* keys[2] = {nullptr, nullptr};
  uint32_t* vals[2] = {nullptr, nullptr};
  uint32_t* hist = nullptr;   // radix tile histograms
  uint32_t* scan_tmp = nullptr;
  uint32_t* flags = nullptr;
  size_t hist_elems = 0;
  size_t scan_tmp_elems = 0;
};
size_t radix_hist_elems(uint64_t n);
size_t scan_tmp_elems(size_t n);
void scan_exclusive_u32(const uint32_t* in, uint32_t* out, size_t n, uint32_t* tmp, cudaStream_t s);

template <typename T>
void launch_cell_ids(const T* soa, uint64_t n, const GridGeom<T>& g, unsigned long long* keys,
                     uint32_t* vals, cudaStream_t s);
// Stable LSD radix sort of (key, value) by the low `bits` bits of key.
// Returns the index (0/1) of the buffers holding the result.
// limit (optional, device): the largest key.  Passes above its highest digit
// are skipped on the device: the result is then in the buffers of the last
// pass that ran (index radix_passes(*limit) & 1), not in the returned ones.
int radix_sort_pairs(GridScratch& sc, uint64_t n, int bits, cudaStream_t s,
                     const unsigned long long* limit = nullptr);
__host__ __device__ inline int radix_passes(unsigned long long limit) {
  int p = 0;
  for (; limit; limit >>= 8) p++;
  return p;
}
// Non-empty cell table from sorted keys; writes C to *d_C.
void launch_compact_cells(const unsigned long long* skeys, uint64_t n, uint32_t* flags,
                          uint32_t* pos, uint32_t* scan_tmp, unsigned long long* ckeys,
                          uint32_t* coff, unsigned long long* d_C, cudaStream_t s);
void launch_dense_table(const unsigned long long* ckeys, const uint32_t* coff, const unsigned long long* d_C,
                        unsigned long long total_cells, uint32_t* dstart, cudaStream_t s);
// Number of cells that hold a point into *d_C, by a bitmap of the grid's cells
// (total_cells bits, rounded up to words).
template <typename T>
void launch_count_cells(const T* soa, uint64_t n, const GridGeom<T>& g, uint32_t* bitmap, unsigned long long* d_C,
                        cudaStream_t s);
// Morton (Z-order) codes of the cells of points given in cell-ordered
// columns ps (keys) and their positions (vals), `bits` bits per dimension.
template <typename T>
void launch_morton_keys(const T* ps, uint64_t n, const GridGeom<T>& g, int bits, unsigned long long* keys,
                        uint32_t* vals, cudaStream_t s);
// Grid by counting sort (points in any order within a cell): tbl (total+1
// entries) becomes the dense start table, ps/pid the cell-ordered columns and
// ids of the points given as columns src with ids src_ids (null: 0, 1, ...).
// scan_tmp: scan_tmp_elems(total).
template <typename T>
void launch_counting_grid(const T* src, const uint32_t* src_ids, uint64_t n, uint32_t d, const GridGeom<T>& g,
                          uint32_t* tbl, uint32_t* scan_tmp, T* ps, uint32_t* pid, cudaStream_t s);
// Number of cells with a point in a dense start table of `total` cells into *d_C.
void launch_count_table(const uint32_t* dstart, unsigned long long total, unsigned long long* d_C, cudaStream_t s);
template <typename T>
// psf (optional): the same columns rounded to float (double data: the
// search's float prefilter)
void launch_gather_sorted(const T* soa, uint64_t n, uint32_t d, const uint32_t* sorted_ids, T* ps, float* psf,
                          cudaStream_t s);

// ---- range search with fused top-K --------------------------------------
// State of the retry loop in device memory, for passes that run inside a
// CUDA graph (a conditional while node): the search kernel reads the pass's
// query count, lists and radius from here, and a one-thread step kernel
// advances it and decides whether another pass runs.
struct LoopCtl {
  uint32_t nq;         // queries of the next pass
  uint32_t iter;       // passes done
  uint32_t cur;        // list[cur] holds the next pass's queries
  uint32_t stop_iter;  // the graph stops before this pass
  uint32_t* list[2];
  double r;            // uniform radius (a value of the data type)
  double step;         // radius growth per pass
  double rmax;         // largest radius the next pass searches
  double rmax_seen;    // largest radius of any pass
  double rgrid;        // radius the grid must suit (plain: r; per-query: median failing radius)
  double r_limit;      // a grid rebuild is due when rgrid > r_limit and rgrid > width
  double width;
  unsigned long long queries_run;
  unsigned long long accepted;
  int per_query;       // per-query radii (learned starting radius)
  int go;              // the next pass runs (set by each pass's step)
  double ring_div;     // radii above width * ring_div / 2 force a rebuild (0: none)
  double redge[64];    // upper radius of each bin of the failing-radius histogram
};

// Grown radii of the queries that failed a pass (per-query radius mode):
// their largest value and a histogram in quarter octaves of eps0, bin
// floor(4 log2(r / eps0)) + 16 clamped to [0, 63].
struct FailRadii {
  unsigned long long rmax_bits;
  uint32_t hist[64];
};
constexpr int FAIL_RADIUS_BINS = 64;

// Launch shape of the search kernel; 0 = the default.
struct SearchShape {
  int warps_per_block = 0;  // 2..8
  int qchunk = 0;           // queries a warp takes per work fetch
  int buffer = 0;           // selection buffer capacity (power of two >= K+32)
};
template <typename T>
struct SearchLaunch {
  DeviceGrid<T> grid;
  const T* xs = nullptr;            // SoA coords in input order (failed queries)
  uint64_t n = 0;
  uint32_t d = 0;
  uint32_t K = 0;
  const uint32_t* qlist = nullptr;  // original ids; nullptr = all, in cell order
  uint32_t nq = 0;
  T radius = 0;                     // uniform radius (qradius == nullptr)
  T* qradius = nullptr;             // per-query radius by original id
  T step = 0;                       // radius growth written back on failure
  int32_t* out_ids = nullptr;
  T* out_d = nullptr;
  double* rowsum = nullptr;                 // per-row verification sums, by id (nullptr: none)
  uint32_t* fail_list = nullptr;
  uint32_t* fail_count = nullptr;
  unsigned long long* cand_count = nullptr;
  uint32_t* work_counter = nullptr;
  FailRadii* fail_radii = nullptr;          // grown radii of the failures (per-query radii)
  double coord_bound = 0.0;                 // largest |coordinate|: enables the float prefilter when finite
  SearchShape shape;                        // launch shape (autotuned for batched joins)
  const LoopCtl* ctl = nullptr;             // non-null: nq, lists and radius come from here (graph passes)
  const uint32_t* nq_dev = nullptr;         // non-null: the pass's query count is read here (nq is a bound)
  // tile search only: queries from these columns and ids, in tile order (when
  // the candidates come from another grid)
  const T* qps = nullptr;
  const uint32_t* qpid = nullptr;
};
template <typename T>
void launch_search(const SearchLaunch<T>& a, int sm_count, cudaStream_t s);
// Tile search (k_tile.cu): the first pass of float data with two or three
// dimensions, all indexed, K <= 65 and a dense cell table.  Queries it hands
// over (ring far wider than its tile's, exact ties at the K-th distance) are
// appended to defer_list / *defer_count for search_kernel at the same radius.
bool tile_search_applies(uint32_t d, uint32_t di, uint32_t K, int dense, size_t elem);
template <typename T>
void launch_tile_search(const SearchLaunch<T>& a, uint32_t* defer_list, uint32_t* defer_count, int sm_count,
                        cudaStream_t s);
// Clears bytes (a multiple of 4) with a kernel: unlike a runtime memset it
// never waits behind copies in flight on another stream.
void launch_zero_words(void* p, size_t bytes, cudaStream_t s);
void launch_copy_to_mapped(void* dst, const void* src, size_t bytes, int sm_count, cudaStream_t s);
int search_buffer_capacity(uint32_t K);
// Exact rows of the queries a.qlist[0..a.nq) by a scan over all points.
template <typename T>
void launch_brute(const SearchLaunch<T>& a, cudaStream_t s);

// Rows delivered to host buffers while the join runs (host-pointer calls
// whose output buffers are pinned): the first pass runs in chunks of query
// ids, each chunk's block of rows is copied out on a second stream as soon as
// its search is done, and the rows that later passes finish are written into
// the host buffers by a kernel at the end, after every chunk copy.
constexpr int MAX_ROW_CHUNKS = 32;
constexpr size_t MAIL_BYTES = 16384;  // mailbox: reads in the first half, writes in the second
// Staging blocks of result tables on their way into pageable host buffers, one
// per copying thread (up to 16 MB pinned per workspace).
constexpr int STAGE_BLOCKS = 8;
constexpr size_t STAGE_BYTES = 2u << 20;
// Largest dimension sample that is read through page-locked memory, which the
// workspace keeps (a 100th of the rows: 480 MB of them at 10^9 x 6 doubles).  At
// 100 M x 2 doubles, 16 MB, a join takes 383.7 ms either way.
constexpr size_t SAMPLE_PINNED_BYTES = 16u << 20;
struct RowStream {
  void* ids_host = nullptr;  // the host buffers
  void* d_host = nullptr;
  void* ids_dev = nullptr;   // their device-accessible addresses
  void* d_dev = nullptr;
  int chunks = 0;            // blocks of query ids in the first pass (>= 2)
  bool checksum = false;     // also compute the result's verification sum
  bool active = false;       // set by run_join when it streamed (rows complete on return)
  double total_distance = 0.0;
};

// ---- box tree (k_tree.cu, tree_search.cuh) ---------------------------------
// The points in an order that keeps neighbours together, 32 to a leaf, and
// the bounding boxes of the leaves and of every 32 nodes above them.
constexpr int TREE_MAX_LEVELS = 6;   // 32^6 leaves
constexpr uint32_t TREE_DIMS = 16;   // dimensions the boxes cover (the first ones: largest variance)
template <typename T>
struct BoxTree {
  // Everything a warp reads at a time lies together, 32 lanes wide: a leaf's
  // points are d rows of 32 coordinates, a node's children 2 * dims rows of 32
  // bounds (one address and immediate offsets instead of one per row).
  const T* ps = nullptr;         // [leaf][d][32]; the last leaf is filled up with infinities
  const float* psf = nullptr;    // double data: the same rounded to float (the float screen)
  const uint32_t* id = nullptr;  // original id of each tree position (filled up with 0xffffffff)
  const float* box = nullptr;    // [node / 32][2 * dims][32]: lower and upper bound of each dimension
  uint32_t dims = 0;             // min(d, TREE_DIMS)
  uint32_t nodes = 0;
  int levels = 0;                // level 0: the leaves; the last level has at most 32 nodes
  uint32_t count[TREE_MAX_LEVELS] = {};
  uint32_t offset[TREE_MAX_LEVELS] = {};
};
struct TreeScratch {
  GridScratch sort;          // keys, vals, hist, scan_tmp
  float* split = nullptr;    // tree_split_elems()
};
constexpr uint32_t TREE_KEY_DIMS = 8;    // dimensions of the space-filling curve
constexpr uint32_t TREE_BINS = 256;      // quantile bins per dimension
constexpr size_t tree_split_elems() { return (size_t)TREE_KEY_DIMS * (TREE_BINS + 1); }
// Largest k+1 of a tree search (its selection buffers hold 256 keys).
constexpr uint32_t tree_max_k(size_t elem) { return elem == 4 ? 224 : 192; }
inline uint64_t tree_stride(uint64_t n) { return (n + 31) & ~31ull; }
void tree_shape(uint64_t n, uint32_t d, uint32_t* count, uint32_t* offset, int* levels, uint32_t* nodes);
// Builds the tree of the n points given as input-order columns xs (stride n)
// into t's buffers (ps, psf, id, box; shape set).
template <typename T>
void launch_tree_build(const T* xs, const T* minmax, uint64_t n, uint32_t d, TreeScratch& sc, const BoxTree<T>& t,
                       cudaStream_t s);
template <typename T>
struct TreeLaunch {
  BoxTree<T> tree;
  uint64_t n = 0;
  uint32_t d = 0, K = 0, indexed = 1;
  const uint32_t* qmask = nullptr;   // bit b of word L: tree position 32 L + b is a query (nullptr: all)
  const uint32_t* nq_dev = nullptr;  // with qmask: how many there are
  T radius = 0;
  T* qradius = nullptr;              // per-query radii by original id
  int unbounded = 0;
  int32_t* out_ids = nullptr;
  T* out_d = nullptr;
  double* rowsum = nullptr;
  uint32_t* fail_mask = nullptr;     // bits of the failed queries (cleared before the pass)
  uint32_t* fail_count = nullptr;
  T* grow = nullptr;                 // grown radii of the failures, by original id
  unsigned long long* rmax_bits = nullptr;  // largest radius searched or grown
  unsigned long long* cand_count = nullptr;
};
template <typename T>
void launch_tree_search(const TreeLaunch<T>& a, int sm_count, cudaStream_t s);

// ---- per-device workspace --------------------------------------------------
struct Workspace {
  DevBuf model;                          // radius model (learned starting radius)
  unsigned model_version = 0;
  DevBuf in, ids, dists;                 // staging for host-pointer calls
  DevBuf xs, ps, psf, pid;               // input-order columns, cell-order columns (+ float copy), ids
  DevBuf keys0, keys1, vals0, vals1, hist, scan_tmp, flags, pos;  // grid build
  DevBuf ckeys, coff, dstart;            // cell tables
  DevBuf list0, list1, small, eps_partial, eps_sample, perm, minmax_part, qradius;
  DevBuf chunk_list, patch_rows;         // streamed rows: queries by id block, rows finished late
  DevBuf defer_list;                     // queries the tile search hands to search_kernel
  DevBuf rowsum;                         // per-row verification sums (host-pointer calls)
  DevBuf fps, fpid, fdstart;             // tile search: the finer candidate grid (columns, ids, start table)
  DevBuf tree_box, tree_split;           // box tree: node boxes, quantiles (points and ids in ps, psf, pid)
  DevBuf curve_ps;                       // tile search: columns along the space-filling curve
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[8] = {};
  cudaStream_t copy_stream = nullptr;    // streamed rows: device-to-host copies
  cudaEvent_t chunk_ev[MAX_ROW_CHUNKS + 1] = {};
  // The join's small reads of device memory go through the mailbox (mapped
  // pinned memory that a kernel writes): one kernel and one synchronisation
  // for several pieces, where each copy into pageable memory is staged and
  // waited for by itself.  While rows stream out, the copy engines are busy
  // for tens of ms: small writes then take the mailbox too, device copies run
  // on the SMs (`mail` set), and none of them queues behind the row copies.
  void* mail_host = nullptr;
  void* mail_dev = nullptr;
  bool mail = false;
  int sm_count = 0;
  void* stage = nullptr;                 // staging blocks (pinned) and their copies' events
  int stage_blocks = 0;
  cudaEvent_t stage_ev[STAGE_BLOCKS] = {};
  void* h_pinned = nullptr;
  size_t h_pinned_bytes = 0;
  void ensure_stream();
  void ensure_copy_stream();
  bool ensure_mail();          // false: no pinned memory to be had
  bool ensure_stage(int blocks);  // false: no pinned memory to be had
  void* pinned(size_t need);   // nullptr: no pinned memory to be had
  void pinned_release();
  void release_all();
  void attach_arena(Arena* a);  // every buffer carves from `a` from now on
};
Workspace& workspace(int device);

struct JoinConfig;
// Full join of n x d row-major data already on the device.  h_aos (optional)
// is the same data on the host, used for the dimension-order sample.
// rowsum (optional, n doubles): each result row's verification sum, and
// st->total_distance their sum.  d_ids / d_dists may be device-mapped host
// memory: the kernels then write the rows straight into the host buffers.
template <typename T>
void run_join(Workspace& w, const JoinConfig& cfg, const T* d_aos, const T* h_aos, uint64_t n, uint32_t d,
              uint32_t k, int32_t* d_ids, T* d_dists, knnsj_stats* st, cudaStream_t s,
              RowStream* rows = nullptr, double* rowsum = nullptr);
// Whether such a join is searched through the box tree, as far as that is known
// without the data: double coordinates too large for the float screen take the
// ring search all the same.
bool join_takes_tree(const JoinConfig& cfg, uint64_t n, uint32_t d, uint32_t K, size_t elem, bool streams);
template <typename T>
void finish_row_stream(Workspace& w, const RowStream& rows, const int32_t* d_ids, const T* d_dists, uint32_t K,
                       cudaStream_t s);
template <typename T>
void run_features(Workspace& w, const JoinConfig& cfg, const T* d_aos, const T* h_aos, uint64_t n, uint32_t d,
                  uint32_t k, float* d_out, double* eps0_out, cudaStream_t s);

// ---- learned starting radius (k_radius.cu, k_mlp.cu) -----------------------
double learned_max_cells(uint32_t di);
template <typename T>
void launch_radius_assign(const DeviceGrid<T>& g, uint64_t n, uint32_t d, uint32_t k, float beta,
                          const float* d_model, double eps0, float offset, double max_cells, T* qradius,
                          uint32_t* d_err, int sm_count, cudaStream_t s);
template <typename T>
void launch_radius_features(const DeviceGrid<T>& g, uint64_t n, uint32_t d, uint32_t k, float beta, float* out,
                            cudaStream_t s);
// d_err is set to 1 if a tensor-core wait timed out (the outputs then hold
// the fallback: eps0 radii, NaN predictions).
void launch_mlp_predict(const float* d_model, const float* d_feat, uint64_t n, float* d_out, uint32_t* d_err,
                        int sm_count, cudaStream_t s);
// Active model: a copy and its version (changes on every set).
unsigned radius_model_snapshot(std::vector<float>* out);
void radius_model_set(const float* model);  // nullptr restores the built-in model
void mlp_grad_device(const float* d_model, const float* d_X, const float* d_Y, const uint32_t* d_idx, uint64_t n,
                     float quantile, float inv_batch, float* d_part, double* d_part_loss, float* d_grad,
                     cudaStream_t s);
uint32_t mlp_grad_blocks(uint64_t n);  // elements of d_part_loss for n samples
size_t mlp_grad_partials(uint64_t n);  // floats of d_part
void train_model(const float* hX, const float* hY, uint64_t n, int epochs, uint32_t batch, float lr,
                 float quantile, uint64_t seed, float* model_out, float* loss_out, cudaStream_t s);

// Outlier scores of a result table on the device (k_outlier.cu): per point
// the mean table distance and its rank (decreasing), the in-degree and its
// rank (increasing); equal scores ranked by point id.
template <typename T>
void outlier_scores_device(Workspace& w, const int32_t* ids, const T* dists, uint64_t n, uint32_t K, double* mean,
                           int32_t* dist_rank, unsigned long long* indeg, uint32_t* degree_rank, cudaStream_t s);

// Verification figure of a result table on the device (synchronises s).
template <typename T>
double device_checksum(Workspace& w, const T* d_vals, uint64_t count, cudaStream_t s);

}  // namespace knnsj
