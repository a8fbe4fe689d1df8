// join.cu -- the self-join pipeline on one GPU.
//
// Host side of the reference's main()/KNNJoinPy (main.cu:109-510, 514-907),
// re-planned for one resident dataset:
//   1. dimension order (ReorderByDimension, main.cu:2521-2615) on the host,
//      from every 100th point, in the reference's float/double arithmetic;
//   2. one transpose into column arrays in that order (device);
//   3. eps0 from BETA (sampleNeighborsBruteForce, GPU.cu:3088-3566);
//   4. grid dimensions (generateNDGridDimensions, main.cu:2425-2488) and the
//      grid index at width eps0 (populateNDGridIndexAndLookupArrayGPU,
//      GPU.cu:3715-4067), built once and kept in HBM;
//   5. the retry loop (main.cu:312-430): search all queries at eps0, then the
//      failed ones at eps0 + m*eps0/2 over the widened cell ring of the same
//      grid.  The reference repeats a pass at an unchanged radius when at
//      most 25% failed (main.cu:330); that pass cannot succeed, so here the
//      radius grows every pass.  When the ring would need many more cells
//      than 3^NUMINDEXEDDIM, the grid is rebuilt at the current radius, as
//      the reference does on every growth (main.cu:353).
// Every device buffer lives in a per-device workspace reused across calls.

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <vector>

#include "knnsj_internal.h"
#include "knnsj_host.h"
#include "radius_model.cuh"
#include "ring_policy.h"

namespace knnsj {

thread_local unsigned long long g_launches = 0;
thread_local bool g_forbid_alloc = false;

void* Arena::take(size_t bytes) {
  const size_t at = (used + 255) & ~(size_t)255;
  if (at + bytes > cap)
    throw StatusError{KNNSJ_ERR_EXCEEDS_FIXED_SCRATCH, "problem exceeds the fixed scratch array"};
  used = at + bytes;
  return base + at;
}

void Workspace::attach_arena(Arena* a) {
  DevBuf* bufs[] = {&model, &in, &ids, &dists, &xs, &ps, &psf, &pid, &keys0, &keys1, &vals0, &vals1, &hist,
                    &scan_tmp, &flags, &pos, &ckeys, &coff, &dstart, &list0, &list1, &small,
                    &eps_partial, &eps_sample, &perm, &minmax_part, &qradius, &chunk_list, &patch_rows, &defer_list,
                    &fps, &fpid, &fdstart, &rowsum, &tree_box, &tree_split, &curve_ps};
  for (DevBuf* b : bufs) {
    b->arena = a;
    b->p = nullptr;
    b->bytes = 0;
  }
  model_version = 0;
}

void* DevBuf::get(size_t need) {
  if (need == 0) need = 16;
  if (arena) {
    if (need > bytes) {
      unsigned char* b = (unsigned char*)p;
      if (b && b + bytes == arena->base + arena->used && (size_t)(b - arena->base) + need <= arena->cap) {
        arena->used = (size_t)(b - arena->base) + need;  // the last block carved grows in place
      } else {
        p = arena->take(need);
      }
      bytes = need;
    }
    return p;
  }
  if (need > bytes) {
    if (g_forbid_alloc) throw StatusError{KNNSJ_ERR_EXCEEDS_FIXED_SCRATCH, "buffer outside the fixed scratch array"};
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    cudaError_t e = cudaMalloc(&p, need);
    if (e != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
      throw StatusError{KNNSJ_ERR_OUT_OF_MEMORY, "cudaMalloc"};
    }
    bytes = need;
  }
  return p;
}

void DevBuf::release() {
  if (p && !arena) cudaFree(p);
  p = nullptr;
  bytes = 0;
}

Workspace& workspace(int device) {
  static std::vector<Workspace*> all;
  static std::mutex m;
  std::lock_guard<std::mutex> g(m);
  if ((int)all.size() <= device) all.resize(device + 1, nullptr);
  if (!all[device]) all[device] = new Workspace();
  return *all[device];
}

void Workspace::release_all() {
  model_version = 0;
  DevBuf* bufs[] = {&model, &in, &ids, &dists, &xs, &ps, &psf, &pid, &keys0, &keys1, &vals0, &vals1, &hist,
                    &scan_tmp, &flags, &pos, &ckeys, &coff, &dstart, &list0, &list1, &small,
                    &eps_partial, &eps_sample, &perm, &minmax_part, &qradius, &chunk_list, &patch_rows, &defer_list,
                    &fps, &fpid, &fdstart, &rowsum, &tree_box, &tree_split, &curve_ps};
  for (DevBuf* b : bufs) b->release();
  if (stream) cudaStreamDestroy(stream);
  stream = nullptr;
  if (copy_stream) cudaStreamDestroy(copy_stream);
  copy_stream = nullptr;
  for (auto& e : ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  for (auto& e : chunk_ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  if (mail_host) cudaFreeHost(mail_host);
  mail_host = mail_dev = nullptr;
  mail = false;
  if (stage) cudaFreeHost(stage);
  stage = nullptr;
  stage_blocks = 0;
  for (auto& e : stage_ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  pinned_release();
}

void Workspace::pinned_release() {
  if (h_pinned) cudaFreeHost(h_pinned);
  h_pinned = nullptr;
  h_pinned_bytes = 0;
}

// Page-locked, mapped host memory, or false where there is none to be had.
// KNNSJ_TEST_PINNED_KB=n (tests only): blocks above n KB are refused, with a line
// on stderr.
static bool alloc_pinned(void** p, size_t bytes) {
  const char* e = std::getenv("KNNSJ_TEST_PINNED_KB");
  const bool refuse = e && bytes > (size_t)std::atoll(e) * 1024;
  if (!refuse && cudaHostAlloc(p, bytes, cudaHostAllocMapped) == cudaSuccess) return true;
  if (refuse) fprintf(stderr, "knnsj: refused %zu bytes of page-locked memory\n", bytes);
  cudaGetLastError();
  *p = nullptr;
  return false;
}

void* Workspace::pinned(size_t need) {
  if (need > h_pinned_bytes) {
    if (g_forbid_alloc) throw StatusError{KNNSJ_ERR_EXCEEDS_FIXED_SCRATCH, "pinned buffer in a fixed-scratch join"};
    pinned_release();
    if (!alloc_pinned(&h_pinned, need)) return nullptr;
    h_pinned_bytes = need;
  }
  return h_pinned;
}

void Workspace::ensure_stream() {
  if (g_forbid_alloc && !stream) throw StatusError{KNNSJ_ERR_EXCEEDS_FIXED_SCRATCH, "stream in a fixed-scratch join"};
  if (!stream) KNNSJ_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  for (auto& e : ev)
    if (!e) KNNSJ_CUDA(cudaEventCreate(&e));
}

void Workspace::ensure_copy_stream() {
  if (g_forbid_alloc) throw StatusError{KNNSJ_ERR_EXCEEDS_FIXED_SCRATCH, "copy stream in a fixed-scratch join"};
  if (!copy_stream) KNNSJ_CUDA(cudaStreamCreateWithFlags(&copy_stream, cudaStreamNonBlocking));
  for (auto& e : chunk_ev)
    if (!e) KNNSJ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  if (!ensure_mail()) throw CudaError{cudaErrorMemoryAllocation, "mailbox of streamed rows"};
}

bool Workspace::ensure_mail() {
  if (mail_host) return true;
  // (joins with fixed scratch, or without page-locked memory, copy into pageable memory)
  if (g_forbid_alloc || !alloc_pinned(&mail_host, MAIL_BYTES)) return false;
  KNNSJ_CUDA(cudaHostGetDevicePointer(&mail_dev, mail_host, 0));
  return true;
}

bool Workspace::ensure_stage(int blocks) {
  if (g_forbid_alloc) return false;
  if (blocks > stage_blocks) {
    if (stage) cudaFreeHost(stage);
    stage = nullptr;
    stage_blocks = 0;
    if (!alloc_pinned(&stage, (size_t)blocks * STAGE_BYTES)) return false;
    stage_blocks = blocks;
  }
  for (int i = 0; i < blocks; i++)
    if (!stage_ev[i]) KNNSJ_CUDA(cudaEventCreateWithFlags(&stage_ev[i], cudaEventDisableTiming));
  return true;
}

namespace {

__global__ void copy_words_kernel(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src, uint64_t words) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

__global__ void zero_words_kernel(uint32_t* __restrict__ p, uint64_t words) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = 0u;
}

void launch_copy_words(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  const uint64_t words = bytes / 4;
  const uint64_t blocks = std::min<uint64_t>((words + 255) / 256, 1024);
  if (blocks == 0) return;
  copy_words_kernel<<<(unsigned)blocks, 256, 0, s>>>((uint32_t*)dst, (const uint32_t*)src, words);
  KNNSJ_CHECK_LAUNCH();
}

__global__ void copy_vec16_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src, uint64_t n16) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

}  // namespace

// Copies a device table into mapped pinned host memory with an SM kernel:
// 16-byte loads and stores in address order, so the host receives whole
// cache lines (13 GB of rows in 67 ms on GB300, the rate of a copy-engine
// copy).  Unaligned buffers fall back to 4-byte words, then to a copy.
void launch_copy_to_mapped(void* dst, const void* src, size_t bytes, int sm_count, cudaStream_t s) {
  const uintptr_t a = (uintptr_t)dst | (uintptr_t)src;
  if ((a & 15) == 0) {
    const uint64_t n16 = bytes / 16;
    if (n16) {
      const uint64_t blocks = std::min<uint64_t>((n16 + 511) / 512, (uint64_t)std::max(sm_count, 1) * 2);
      copy_vec16_kernel<<<(unsigned)blocks, 512, 0, s>>>((uint4*)dst, (const uint4*)src, n16);
      KNNSJ_CHECK_LAUNCH();
    }
    const size_t done = n16 * 16;
    if (bytes > done && (bytes - done) % 4 == 0)
      launch_copy_words((char*)dst + done, (const char*)src + done, bytes - done, s);
    else if (bytes > done)
      KNNSJ_CUDA(cudaMemcpyAsync((char*)dst + done, (const char*)src + done, bytes - done, cudaMemcpyDefault, s));
  } else if ((a & 3) == 0 && bytes % 4 == 0) {
    launch_copy_words(dst, src, bytes, s);
  } else {
    KNNSJ_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, s));
  }
}

void launch_zero_words(void* p, size_t bytes, cudaStream_t s) {
  const uint64_t words = bytes / 4;
  const uint64_t blocks = std::min<uint64_t>((words + 255) / 256, 1024);
  if (blocks == 0) return;
  zero_words_kernel<<<(unsigned)blocks, 256, 0, s>>>((uint32_t*)p, words);
  KNNSJ_CHECK_LAUNCH();
}

// Device-to-device copy (bytes a multiple of 4).
static void dev_copy(Workspace& w, void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (w.mail)
    launch_copy_words(dst, src, bytes, s);
  else
    KNNSJ_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s));
}

// One piece of a device-to-host read (a multiple of 4 bytes).
struct Piece {
  void* dst;
  const void* src;
  size_t bytes;
};
namespace {
constexpr int MAX_PIECES = 4;
struct PieceList {
  const uint32_t* src[MAX_PIECES];
  uint32_t words[MAX_PIECES];
};
// Gathers the pieces one after the other at dst (mapped host memory).
__global__ void __launch_bounds__(1024) collect_kernel(uint32_t* __restrict__ dst, const PieceList l) {
  uint32_t at = 0;
  for (int p = 0; p < MAX_PIECES; p++) {
    for (uint32_t i = threadIdx.x; i < l.words[p]; i += blockDim.x) dst[at + i] = l.src[p][i];
    at += l.words[p];
  }
}
}  // namespace

// Device-to-host reads of a few small pieces with one synchronisation of s.
static void read_pieces(Workspace& w, std::initializer_list<Piece> pieces, cudaStream_t s) {
  size_t bytes = 0;
  for (const Piece& p : pieces) bytes += p.bytes;
  if (w.ensure_mail() && bytes <= MAIL_BYTES / 2 && pieces.size() <= MAX_PIECES) {
    PieceList l{};
    int i = 0;
    for (const Piece& p : pieces) {
      l.src[i] = (const uint32_t*)p.src;
      l.words[i++] = (uint32_t)(p.bytes / 4);
    }
    collect_kernel<<<1, bytes > 1024 ? 1024 : 128, 0, s>>>((uint32_t*)w.mail_dev, l);
    KNNSJ_CHECK_LAUNCH();
    KNNSJ_CUDA(cudaStreamSynchronize(s));
    const unsigned char* at = (const unsigned char*)w.mail_host;
    for (const Piece& p : pieces) {
      std::memcpy(p.dst, at, p.bytes);
      at += p.bytes;
    }
    return;
  }
  if (w.mail) throw StatusError{KNNSJ_ERR_UNSUPPORTED, "mailbox read too large"};
  for (const Piece& p : pieces) KNNSJ_CUDA(cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToHost, s));
  KNNSJ_CUDA(cudaStreamSynchronize(s));
}

static void read_small(Workspace& w, void* dst, const void* src, size_t bytes, cudaStream_t s) {
  read_pieces(w, {Piece{dst, src, bytes}}, s);
}

// Host-to-device write of a few bytes (a multiple of 4); the source may be
// reused on return.
static void write_small(Workspace& w, void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (w.mail) {
    if (bytes > MAIL_BYTES / 2) throw StatusError{KNNSJ_ERR_UNSUPPORTED, "mailbox write too large"};
    unsigned char* in_host = (unsigned char*)w.mail_host + MAIL_BYTES / 2;
    std::memcpy(in_host, src, bytes);
    launch_copy_words(dst, (unsigned char*)w.mail_dev + MAIL_BYTES / 2, bytes, s);
    KNNSJ_CUDA(cudaStreamSynchronize(s));  // the mailbox is free again
    return;
  }
  KNNSJ_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
  KNNSJ_CUDA(cudaStreamSynchronize(s));
}

namespace {

// What the host reads of a join (cleared when the join starts).
struct SmallHead {
  uint32_t nonfinite;
  uint32_t fail_count;
  uint32_t work_counter;
  uint32_t defer_count;                 // queries the tile search handed to search_kernel (current launch)
  unsigned long long C0;                // non-empty cells of the eps0 grid
  unsigned long long cand;
  double avg[2];
  unsigned long long defer_total;       // all queries handed over by the tile search in this join
  unsigned long long tree_rmax;         // tree search: largest radius searched (bits)
  uint32_t tree_fail[2];                // tree search: failures of its first two passes
  uint32_t mlp_err;                     // the tensor-core radius MLP timed out
  uint32_t pad;
  double csum;
};
struct SmallDev : SmallHead {  // layout of Workspace::small
  uint32_t hist[HIST_BUCKETS];
  unsigned long long C;                 // non-empty cells of a rebuilt grid
  HistConst hc[2];
  double cpart[1024];
  FailRadii fr;
  LoopCtl ctl;
  uint32_t chunk_fill[MAX_ROW_CHUNKS];  // streamed rows: queries placed per id block
  uint32_t patch_count;                 // streamed rows: first-pass failures
};

template <typename T>
T host_fallback_eps(const std::vector<T>& mn, const std::vector<T>& mx, uint64_t n, uint32_t K) {
  double ext = 0.0;
  for (size_t j = 0; j < mn.size(); j++) ext = std::max(ext, (double)mx[j] - (double)mn[j]);
  if (!(ext > 0)) return (T)1;
  const double per_dim = std::max(1.0, std::floor(std::pow((double)n / K, 1.0 / mn.size())));
  return (T)(ext / per_dim);
}

}  // namespace

// generateNDGridDimensions (main.cu:2425-2488), in DTYPE.
template <typename T>
static GridGeom<T> grid_geometry(uint32_t di, const std::vector<T>& mn, const std::vector<T>& mx, T width) {
  GridGeom<T> g{};
  g.di = di;
  g.width = width;
  unsigned long long mult = 1;
  bool overflow = false;
  for (uint32_t j = 0; j < di; j++) {
    const T lo = mn[j] - width;
    const T hi = mx[j] + width;
    const T cells = std::ceil((hi - lo) / width);
    if (!(cells < 4294967295.0)) throw StatusError{KNNSJ_ERR_UNSUPPORTED, "grid too fine"};
    g.minv[j] = lo;
    g.ncell[j] = (uint32_t)cells;
    if (g.ncell[j] == 0) g.ncell[j] = 1;
    g.mult[j] = mult;
    if (mult > ~0ull / g.ncell[j]) overflow = true;
    mult *= g.ncell[j];
  }
  if (overflow) throw StatusError{KNNSJ_ERR_UNSUPPORTED, "more than 2^64 grid cells"};
  g.total_cells = mult;
  return g;
}

// Whether a grid of that many cells gets a dense cell table.
static bool dense_table(const JoinConfig& cfg, uint64_t n, unsigned long long total) {
  const unsigned long long limit =
      cfg.dense_cells_cap ? cfg.dense_cells_cap : std::max<unsigned long long>(4ull * n, 1ull << 24);
  if (total >= (1ull << 31) || cfg.dense_mode == 0) return false;
  // (forced dense tables still respect an explicit cap: a fixed scratch array sets one)
  return total <= limit || (cfg.dense_mode == 2 && !cfg.dense_cells_cap);
}

// The grid index of width `width`; d_C receives its number of non-empty cells.
template <typename T>
static void build_grid(Workspace& w, const JoinConfig& cfg, uint64_t n, uint32_t d, uint32_t di,
                       const std::vector<T>& mn, const std::vector<T>& mx, T width, unsigned long long* d_C,
                       DeviceGrid<T>* out, cudaStream_t s) {
  const GridGeom<T> g = grid_geometry<T>(di, mn, mx, width);
  int bits = 0;
  while (bits < 64 && ((g.total_cells - 1) >> bits) != 0) bits++;

  GridScratch sc;
  sc.keys[0] = (unsigned long long*)w.keys0.get(n * 8);
  sc.keys[1] = (unsigned long long*)w.keys1.get(n * 8);
  sc.vals[0] = (uint32_t*)w.vals0.get(n * 4);
  sc.vals[1] = (uint32_t*)w.vals1.get(n * 4);
  sc.hist_elems = radix_hist_elems(n);
  sc.hist = (uint32_t*)w.hist.get(sc.hist_elems * 4);
  sc.scan_tmp_elems = scan_tmp_elems(std::max<size_t>(sc.hist_elems, n + 1));
  sc.scan_tmp = (uint32_t*)w.scan_tmp.get(sc.scan_tmp_elems * 4);
  const T* xs = (const T*)w.xs.p;
  launch_cell_ids<T>(xs, n, g, sc.keys[0], sc.vals[0], s);
  const int cur = radix_sort_pairs(sc, n, bits, s);
  const unsigned long long* skeys = sc.keys[cur];
  const uint32_t* sids = sc.vals[cur];
  uint32_t* flags = (uint32_t*)w.flags.get(n * 4);
  uint32_t* pos = (uint32_t*)w.pos.get(n * 4);
  unsigned long long* ckeys = (unsigned long long*)w.ckeys.get(n * 8);
  uint32_t* coff = (uint32_t*)w.coff.get((n + 1) * 4);
  launch_compact_cells(skeys, n, flags, pos, sc.scan_tmp, ckeys, coff, d_C, s);
  // (the box tree keeps its points in the same buffers, in whole leaves)
  T* ps = (T*)w.ps.get(tree_stride(n) * d * sizeof(T));
  float* psf = sizeof(T) == 8 ? (float*)w.psf.get(tree_stride(n) * d * sizeof(float)) : nullptr;
  uint32_t* pid = (uint32_t*)w.pid.get(tree_stride(n) * 4);
  dev_copy(w, pid, sids, n * 4, s);
  launch_gather_sorted<T>(xs, n, d, sids, ps, psf, s);
  out->geom = g;
  out->ps = ps;
  out->psf = psf;
  out->pid = pid;
  out->ckeys = ckeys;
  out->coff = coff;
  out->C = 0;
  out->dense = dense_table(cfg, n, g.total_cells);
  out->dstart = nullptr;
  if (out->dense) {
    uint32_t* dstart = (uint32_t*)w.dstart.get((g.total_cells + 1) * 4);
    launch_dense_table(ckeys, coff, d_C, g.total_cells, dstart, s);
    out->dstart = dstart;
  } else {  // the searches of the cell list take its length
    read_small(w, &out->C, d_C, sizeof(out->C), s);
  }
}

// The radius a rebuilt grid is sized for when queries carry their own radii:
// the median grown radius of the failed queries (bin upper edge, at most the
// largest), so that most of them search small rings; the few with far larger
// radii search wider rings of the same grid.
__host__ __device__ inline double median_fail_radius(const uint32_t* hist, uint32_t nfail, const double* redge,
                                                     double rmax) {
  const uint32_t target = (nfail + 1) / 2;
  uint32_t cum = 0;
  for (int b = 0; b < FAIL_RADIUS_BINS; b++) {
    cum += hist[b];
    if (cum >= target) return redge[b] < rmax ? redge[b] : rmax;
  }
  return rmax;
}

namespace {

// One pass's bookkeeping inside the retry graph, mirroring the host loop of
// run_join: count the pass, swap the lists, grow the radius, and let the next
// pass run unless every query is done, a rebuild is due or the pass budget
// of this graph launch is spent (the loop always ends: iter grows by one per
// pass and stop_iter is finite).
template <typename T>
__global__ void loop_step_kernel(LoopCtl* c, const uint32_t* __restrict__ fail_count,
                                 const FailRadii* __restrict__ fr, cudaGraphConditionalHandle handle,
                                 int in_graph) {
  const uint32_t nfail = *fail_count;
  c->queries_run += c->nq;
  c->accepted += c->nq - nfail;
  c->iter++;
  c->cur ^= 1u;
  c->nq = nfail;
  if (nfail > 0) {
    if (c->per_query) {
      const unsigned long long b = fr->rmax_bits;
      c->rmax = sizeof(T) == 4 ? (double)__uint_as_float((uint32_t)b) : __longlong_as_double((long long)b);
      c->rgrid = median_fail_radius(fr->hist, nfail, c->redge, c->rmax);
    } else {
      c->r = (double)(T)__dadd_rn(c->r, c->step);  // main.cu:336
      c->rmax = c->r;
      c->rgrid = c->r;
    }
    c->rmax_seen = fmax(c->rmax_seen, c->rmax);
  }
  const bool regrid = regrid_due(c->rgrid, c->rmax, c->r_limit, c->width, c->ring_div);
  c->go = (nfail > 0 && c->iter < c->stop_iter && !regrid) ? 1 : 0;
  if (in_graph) cudaGraphSetConditional(handle, c->go ? 1u : 0u);
}

// First node of the retry graph: the loop runs while the loop state says so.
__global__ void loop_cond_kernel(const LoopCtl* c, cudaGraphConditionalHandle handle) {
  cudaGraphSetConditional(handle, c->go ? 1u : 0u);
}

// Streamed rows: the queries of each block of crow consecutive ids, in the
// cell order they have in pid, visited in `order` when given (nearby queries
// stay together), block c at
// lists[c * crow ...].  Lanes of a warp with the same block take consecutive
// slots from one atomic.
__global__ void chunk_lists_kernel(const uint32_t* __restrict__ pid, const uint32_t* __restrict__ order, uint32_t n,
                                   uint32_t crow, uint32_t* __restrict__ fill, uint32_t* __restrict__ lists) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool live = i < n;
  const uint32_t id = live ? pid[order ? order[i] : i] : 0u;
  const uint32_t c = live ? id / crow : 0xffffffffu;
  const unsigned peers = __match_any_sync(0xffffffffu, c);
  const int leader = __ffs(peers) - 1;
  uint32_t base = 0;
  if (live && lane == leader) base = atomicAdd(&fill[c], (uint32_t)__popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (live) lists[(uint64_t)c * crow + base + __popc(peers & ((1u << lane) - 1u))] = id;
}

// Streamed rows: the first pass's failures (count on the device), kept for
// the patch after the lists are reused by later passes.
__global__ void save_fail_list_kernel(const uint32_t* __restrict__ src, const uint32_t* __restrict__ count,
                                      uint32_t* __restrict__ dst, uint32_t* __restrict__ saved) {
  const uint32_t nf = *count;
  if (blockIdx.x == 0 && threadIdx.x == 0) *saved = nf;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) dst[i] = src[i];
}

// Streamed rows: rows finished after the first pass, copied from the device
// table into the host buffers (one warp per row).
template <typename T>
__global__ void patch_rows_kernel(const uint32_t* __restrict__ rows, const uint32_t* __restrict__ count,
                                  const int32_t* __restrict__ ids, const T* __restrict__ dists, uint32_t K,
                                  int32_t* h_ids, T* h_d) {
  const uint32_t nrows = *count;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t wid = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; wid < nrows; wid += nwarps) {
    const uint64_t base = (uint64_t)rows[wid] * K;
    for (uint32_t j = lane; j < K; j += 32) {
      h_ids[base + j] = ids[base + j];
      h_d[base + j] = dists[base + j];
    }
  }
}

// Adds the tile search's hand-over count to the join's total and clears it
// for the next launch.
__global__ void defer_roll_kernel(uint32_t* __restrict__ count, unsigned long long* __restrict__ total) {
  *total += *count;
  *count = 0u;
}

}  // namespace

// Sorts the points (columns ps) along a space-filling curve over their cells
// (Hilbert in two dimensions, Morton otherwise) on a grid 16 times finer than
// eps0, so that the few queries of a tile lie close together, not anywhere in
// one eps0 cell: the union box of their rings then stays near the size of one
// ring.  Returns the positions in curve order.
template <typename T>
static const uint32_t* curve_order(Workspace& w, const GridGeom<T>& g, const T* ps, uint64_t n, T eps0,
                                   cudaStream_t s) {
  constexpr int ORDER_FINE = 16;
  GridGeom<T> gm = g;
  gm.width = (T)((double)eps0 / ORDER_FINE);
  int bits = 1;
  for (uint32_t j = 0; j < g.di; j++)
    while (bits < 21 && (1ull << bits) < (unsigned long long)g.ncell[j] * ORDER_FINE) bits++;
  GridScratch sc;
  sc.hist_elems = radix_hist_elems(n);
  sc.keys[0] = (unsigned long long*)w.keys0.get(n * 8);
  sc.keys[1] = (unsigned long long*)w.keys1.get(n * 8);
  sc.vals[0] = (uint32_t*)w.vals0.get(n * 4);
  sc.vals[1] = (uint32_t*)w.vals1.get(n * 4);
  sc.hist = (uint32_t*)w.hist.get(sc.hist_elems * 4);
  launch_morton_keys<T>(ps, n, gm, bits, sc.keys[0], sc.vals[0], s);
  return sc.vals[radix_sort_pairs(sc, n, bits * (int)g.di, s)];
}

// The eps0 grid of a join searched by query tiles: the points are sorted once,
// along the tiles' curve, and counted into the cells from there (any order
// within a cell; neighbours on the curve share cells, so the counting sort's
// atomics and writes stay together).  Sorting by cell id first, and again along
// the curve, took 4.0 ms of the 25M-point sky join, this 2.7 (37.6 -> 36.6 ms).
template <typename T>
static void build_curve_grid(Workspace& w, const GridGeom<T>& g, const T* xs, uint64_t n, uint32_t d, T eps0,
                             unsigned long long* d_C, DeviceGrid<T>* out, const T** curve_ps,
                             const uint32_t** curve_ids, cudaStream_t s) {
  const uint32_t* ids = curve_order<T>(w, g, xs, n, eps0, s);
  T* cps = (T*)w.curve_ps.get(n * d * sizeof(T));
  launch_gather_sorted<T>(xs, n, d, ids, cps, nullptr, s);
  T* ps = (T*)w.ps.get(tree_stride(n) * d * sizeof(T));
  uint32_t* pid = (uint32_t*)w.pid.get(tree_stride(n) * 4);
  uint32_t* tbl = (uint32_t*)w.dstart.get((g.total_cells + 1) * 4);
  uint32_t* tmp = (uint32_t*)w.scan_tmp.get(
      std::max(scan_tmp_elems(std::max<size_t>(radix_hist_elems(n), n + 1)), scan_tmp_elems(g.total_cells)) * 4);
  launch_counting_grid<T>(cps, ids, n, d, g, tbl, tmp, ps, pid, s);
  launch_count_table(tbl, g.total_cells, d_C, s);
  out->geom = g;
  out->ps = ps;
  out->psf = nullptr;
  out->pid = pid;
  out->ckeys = nullptr;
  out->coff = nullptr;
  out->C = 0;
  out->dense = 1;
  out->dstart = tbl;
  *curve_ps = cps;
  *curve_ids = ids;
}

// Set-up of the tile search for the first pass: the order in which tiles
// take the queries (Hilbert or Morton order of their cells on a grid 16
// times finer than eps0, so that consecutive queries are close in every
// dimension) and
// the grid the candidates come from (a finer grid of width eps0 / f when its
// dense table fits).
template <typename T>
struct TileSetup {
  bool on = false;
  DeviceGrid<T> cand;                 // candidate grid
  const T* qps = nullptr;             // query columns and ids: in curve order (query tiles) or in the eps0
  const uint32_t* qpid = nullptr;     // grid's cell order
  int fine = 1;                       // eps0 / candidate cell width
  bool per_query = false;             // search_kernel (one warp per query) on the candidate grid
};

template <typename T>
static void prepare_tile(Workspace& w, bool tiles, int fine_max, const DeviceGrid<T>& g, const T* curve_ps,
                         const uint32_t* curve_ids, uint64_t n, uint32_t d, T eps0, const std::vector<T>& mx,
                         TileSetup<T>* t, cudaStream_t s) {
  const uint32_t di = g.geom.di;
  GridScratch sc;
  sc.hist_elems = radix_hist_elems(n);
  sc.scan_tmp_elems = scan_tmp_elems(std::max<size_t>(sc.hist_elems, n + 1));
  t->per_query = !tiles;
  // 1. the order of the queries
  t->qps = g.ps;
  t->qpid = g.pid;
  if (tiles) {
    t->qps = curve_ps;
    t->qpid = curve_ids;
  }
  // 2. candidate grid: width eps0 / f, the largest f <= fine_max whose
  // dense table stays within max(8 n, 2^24) cells
  t->cand = g;
  t->fine = 1;
  const unsigned long long limit = std::max<unsigned long long>(8ull * n, 1ull << 24);
  for (int f = fine_max; f >= 2; f--) {
    GridGeom<T> gf = g.geom;
    gf.width = (T)((double)eps0 / (double)f);
    if (!(gf.width > 0)) continue;
    unsigned long long mult = 1;
    bool fits = true;
    for (uint32_t j = 0; j < di && fits; j++) {
      const T hi = mx[j] + eps0;
      const T cells = std::ceil((hi - gf.minv[j]) / gf.width);
      if (!(cells < 4294967295.0)) {
        fits = false;
        break;
      }
      gf.ncell[j] = std::max<uint32_t>((uint32_t)cells, 1u);
      gf.mult[j] = mult;
      if (mult > limit / gf.ncell[j]) fits = false;
      mult *= gf.ncell[j];
    }
    if (!fits || mult > limit) continue;
    gf.total_cells = mult;
    uint32_t* tbl = (uint32_t*)w.fdstart.get((mult + 1) * 4);
    uint32_t* tmp = (uint32_t*)w.scan_tmp.get(std::max(sc.scan_tmp_elems, scan_tmp_elems(mult)) * 4);
    T* fps = (T*)w.fps.get(n * d * sizeof(T));
    uint32_t* fpid = (uint32_t*)w.fpid.get(n * 4);
    // (points visited in curve or eps0-cell order: neighbours fall in the same cells)
    launch_counting_grid<T>(t->qps, t->qpid, n, d, gf, tbl, tmp, fps, fpid, s);
    t->cand.geom = gf;
    t->cand.ps = fps;
    t->cand.psf = nullptr;
    t->cand.pid = fpid;
    t->cand.ckeys = nullptr;
    t->cand.coff = nullptr;
    t->cand.C = 0;
    t->cand.dense = 1;
    t->cand.dstart = tbl;
    t->fine = f;
    break;
  }
  t->on = true;
}

// One search pass over the queries of a.qlist (or all points in cell order):
// the tile search where it is set up, then search_kernel over the queries it
// handed over, at the same radius on the eps0 grid; otherwise search_kernel
// alone.
template <typename T>
static void first_pass_search(Workspace& w, const SearchLaunch<T>& a, const TileSetup<T>& tile, SmallDev* sm,
                              cudaStream_t s) {
  if (tile.on && tile.per_query) {  // search_kernel over the finer candidate grid, queries in its cell order
    SearchLaunch<T> t = a;
    t.grid = tile.cand;
    launch_search<T>(t, w.sm_count, s);
    return;
  }
  if (tile.on) {
    uint32_t* defer = (uint32_t*)w.defer_list.get(a.n * 4);
    SearchLaunch<T> t = a;
    t.grid = tile.cand;
    t.qps = tile.qps;
    t.qpid = tile.qpid;
    launch_tile_search<T>(t, defer, &sm->defer_count, w.sm_count, s);
    SearchLaunch<T> b = a;
    b.qlist = defer;
    b.nq_dev = &sm->defer_count;
    launch_search<T>(b, w.sm_count, s);
    defer_roll_kernel<<<1, 1, 0, s>>>(&sm->defer_count, &sm->defer_total);
    KNNSJ_CHECK_LAUNCH();
    return;
  }
  launch_search<T>(a, w.sm_count, s);
}

// Whether the first pass runs by query tiles (given a dense cell table and no
// streamed rows): per-query starting radii, or when asked for.
template <typename T>
static bool query_tiles(const JoinConfig& cfg, uint32_t d, uint32_t di, uint32_t K) {
  return tile_search_applies(d, di, K, 1, sizeof(T)) &&
         (cfg.tile_search == 3 || (cfg.tile_search == 1 && cfg.radius_mode == KNNSJ_RADIUS_LEARNED));
}

// Steps 1-4 of the pipeline: dimension order, column transpose, eps0 and
// the grid index at eps0.
template <typename T>
struct Prepared {
  DeviceGrid<T> grid;
  T* xs = nullptr;
  const T* minmax = nullptr;  // device: extremes of every column
  const T* curve_ps = nullptr;          // tile search: columns and ids along the tiles' curve
  const uint32_t* curve_ids = nullptr;
  T eps0 = 0;
  int bucket = -1;
  double avg = 0.0;
  double max_abs = 0.0;  // largest |coordinate| over all dimensions
  std::vector<T> mn, mx;
};

// Joins searched through the box tree.  Not those whose rows stream out in
// blocks of ids during the first pass, nor those with a cap on the passes of
// the radius schedule, which counts the schedule's own passes, nor double data
// that the float screen cannot hold (or is told not to: the ring search then
// takes every distance in double), nor where a grid search is asked for
// (tile_search 2 and 3).
//
// Whole joins measured on both sides, 2 000 to 3 000 000 points, k = 8, 64 and
// 120, float and double, BETA 0.025 (ring over tree time):
//   four and more dimensions: the ring of cells visits several times the
//     points and most first passes fail; 1.4x (4-D) to 27x (12-D);
//   three dimensions: 0.98-3.1x, the tile kernel's learned joins of up to a
//     million points included;
//   one dimension, a uniform radius: 1.4-80x, 2 000 to 25 M points, k = 1 to 180
//     (against the ring search's first form);
//   two dimensions, a uniform radius: 0.97-2.5x from 30 000 points on (most
//     first passes fail; the tree needs no schedule of passes), 1.0-1.3x at
//     2 000 (0.8x at k = 120, where few passes fail);
//   two dimensions, learned radii: rings of a few cells, few failures.  The
//     tile kernel (float, k + 1 <= 65) 0.5-0.9x at 3 M; one warp per query
//     0.9-1.2x below a million points, 1.04-1.36x at 3 M.
//   k + 1 above 224 (float) or 192 (double): the selection buffer of 256 keys
//     is reduced too often, and larger ones are sorted whole; 100 000-300 000
//     points, k = 200: 1.06-5.7x float, 0.88-4.6x double, k = 223 double
//     0.7-2.1x, k = 1000 0.65-1.0x, k = 4000 0.5-0.7x.
constexpr uint64_t TREE_LEARNED_2D_MIN = 1000000;

// Large three-dimensional learned joins whose occupied cells hold about k + 1
// points each (an evenly filled space or surface, with a dense cell table) stay
// with the query tiles: their rings are a few cells wide and nearly every query
// succeeds at once.  Uneven density makes wide rings beside dense cells and
// outliers.  Whole joins, k = 1 to 64, tree time over tile time:
//   0.8 (k + 1) points per occupied cell or more (uniform, a sphere's surface):
//     0.8-1.1x at 300 000 points, 0.99-1.4x at 1 M, 1.06-1.5x at 5 M, 1.2-1.7x at
//     20 M;
//   fewer, 1 to 20 M: normal data (0.3-0.8 of k + 1) 0.4-1.5x with no order in n
//     or k (the tiles wait for a few outliers), mixtures 0.1-1.1x.
constexpr uint64_t TILE_3D_MIN = 1000000;
constexpr double TILE_3D_FILL = 0.8;
template <typename T>
static bool tree_applies(const JoinConfig& cfg, uint64_t n, uint32_t d, uint32_t di, uint32_t K, double max_abs,
                         bool will_stream) {
  if (!cfg.tree_search || will_stream || cfg.max_iterations > 0) return false;
  if (sizeof(T) == 8 && (!cfg.float_prefilter || !(4.0 * std::sqrt((double)d) * max_abs < 1e18))) return false;
  if (K > tree_max_k(sizeof(T))) return false;
  if (cfg.tree_search == 2) return true;
  if (cfg.tile_search >= 2) return false;
  if (d >= 3 || cfg.radius_mode != KNNSJ_RADIUS_LEARNED) return true;
  return n >= TREE_LEARNED_2D_MIN && !(cfg.tile_search && tile_search_applies(d, di, K, 1, sizeof(T)));
}

bool join_takes_tree(const JoinConfig& cfg, uint64_t n, uint32_t d, uint32_t K, size_t elem, bool streams) {
  return elem == 4 ? tree_applies<float>(cfg, n, d, cfg.num_indexed_dims, K, 0.0, streams)
                   : tree_applies<double>(cfg, n, d, cfg.num_indexed_dims, K, 0.0, streams);
}

template <typename T>
static void prepare(Workspace& w, const JoinConfig& cfg, const T* d_aos, const T* h_aos, uint64_t n, uint32_t d,
                    uint32_t k, knnsj_stats* st, cudaStream_t s, Prepared<T>* P, bool will_stream = false,
                    bool* use_tree = nullptr) {
  const uint32_t K = k + 1;
  const uint32_t di = cfg.num_indexed_dims;

  // 1. dimension order
  std::vector<uint32_t> perm(d);
  for (uint32_t j = 0; j < d; j++) perm[j] = j;
  if (!cfg.no_reorder) {
    const uint64_t ns = (n + 99) / 100;
    std::vector<T> sample;
    const T* sp = nullptr;
    if (h_aos) {
      sample.resize(ns * d);
      for (uint64_t i = 0; i < ns; i++)
        std::memcpy(&sample[i * d], h_aos + i * 100 * d, d * sizeof(T));
      sp = sample.data();
    } else if (!g_forbid_alloc) {
      // gathered by a kernel straight into mapped memory (a strided copy of
      // rows of a few bytes is slow on the copy engines); large samples, and any
      // where there is no page-locked memory, through the buffer of the columns,
      // which are not there yet
      const size_t bytes = ns * d * sizeof(T);
      T* host = bytes <= SAMPLE_PINNED_BYTES ? (T*)w.pinned(bytes) : nullptr;
      void* dev = w.xs.get(n * d * sizeof(T));
      if (host) KNNSJ_CUDA(cudaHostGetDevicePointer(&dev, host, 0));
      launch_gather_rows<T>(d_aos, ns, 100, d, (T*)dev, s);
      if (!host) {
        sample.resize(ns * d);
        KNNSJ_CUDA(cudaMemcpyAsync(sample.data(), dev, bytes, cudaMemcpyDeviceToHost, s));
      }
      KNNSJ_CUDA(cudaStreamSynchronize(s));
      sp = host ? host : sample.data();
    } else {
      sample.resize(ns * d);
      KNNSJ_CUDA(cudaMemcpy2DAsync(sample.data(), d * sizeof(T), d_aos, 100 * d * sizeof(T),
                                   d * sizeof(T), ns, cudaMemcpyDeviceToHost, s));
      KNNSJ_CUDA(cudaStreamSynchronize(s));
      sp = sample.data();
    }
    reorder_from_sample<T>(sp, ns, n, d, perm.data(), nullptr);
  }
  if (st)
    for (uint32_t j = 0; j < d && j < 64; j++) st->perm[j] = perm[j];

  // 2. transpose into column arrays
  SmallDev* sm = (SmallDev*)w.small.get(sizeof(SmallDev));
  KNNSJ_CUDA(cudaMemsetAsync(sm, 0, offsetof(SmallDev, C), s));  // the head and the histogram
  T* xs = (T*)w.xs.get(n * d * sizeof(T));
  // (double data: a float copy too, for the histogram's brackets; the buffer
  // later holds the cell-ordered float columns)
  float* xsf = sizeof(T) == 8 ? (float*)w.psf.get(tree_stride(n) * d * sizeof(float)) : nullptr;
  launch_transpose_reorder<T>(d_aos, xs, xsf, n, d, perm.data(), s, &sm->nonfinite);
  if (!xsf) xsf = reinterpret_cast<float*>(xs);
  T* mm_part = (T*)w.minmax_part.get(1024 * 2 * d * sizeof(T) + 2 * d * sizeof(T));
  T* d_minmax = mm_part + 1024 * 2 * d;
  launch_minmax<T>(xs, n, d, d_minmax, mm_part, s);

  // 3. eps0 (GPU.cu:3088-3566): the mean distance and the first range of the
  // histogram, then one look at the results (the rest of the histogram only if
  // the crossing lies beyond)
  EpsScratch es;
  const uint64_t nthr = eps_avg_threads(n);
  es.partial = (double*)w.eps_partial.get(std::max<uint64_t>(nthr * eps_avg_chunks(n), 1) * 8);
  es.sample_sum = (double*)w.eps_sample.get(std::max<uint64_t>(nthr, 1) * 8);
  es.avg_out = sm->avg;
  es.hist = sm->hist;
  es.hc = sm->hc;
  launch_eps_avg<T>(xs, d_minmax, n, d, es, s);
  launch_eps_hist<T>(xs, xsf, n, d, es, 0, s);
  SmallHead head;
  std::vector<T> hmm(2 * d);
  std::vector<uint32_t> hh(HIST_BUCKETS, 0);
  read_pieces(w, {Piece{&head, static_cast<SmallHead*>(sm), sizeof(head)},
                  Piece{hh.data(), sm->hist, HIST_FIRST * 4},
                  Piece{hmm.data(), d_minmax, 2 * d * sizeof(T)}}, s);
  if (head.nonfinite) throw StatusError{KNNSJ_ERR_NONFINITE_INPUT, "NaN or infinite coordinate"};
  double max_abs = 0.0;
  for (uint32_t j = 0; j < 2 * d; j++) max_abs = std::max(max_abs, std::fabs((double)hmm[j]));
  P->max_abs = max_abs;
  EpsChoice ec = choose_eps(hh.data(), HIST_FIRST, head.avg[0], n, k, cfg.beta);
  if (!ec.complete) {
    launch_eps_hist<T>(xs, xsf, n, d, es, 1, s);
    KNNSJ_CUDA(cudaMemcpyAsync(hh.data(), sm->hist, HIST_BUCKETS * 4, cudaMemcpyDeviceToHost, s));
    KNNSJ_CUDA(cudaStreamSynchronize(s));
    ec = choose_eps(hh.data(), HIST_BUCKETS, head.avg[0], n, k, cfg.beta);
  }
  T eps0 = (T)ec.eps;
  P->mn.assign(di, 0);
  P->mx.assign(di, 0);
  for (uint32_t j = 0; j < di; j++) {
    P->mn[j] = hmm[2 * j];
    P->mx[j] = hmm[2 * j + 1];
  }
  int bucket = ec.bucket;
  if (!(eps0 > 0) || !std::isfinite((double)eps0)) {
    // The reference divides by a zero epsilon here (N <= 1000 gives a zero
    // sampled mean); any positive width keeps the join exact.
    eps0 = host_fallback_eps<T>(P->mn, P->mx, n, K);
    bucket = -1;
  }
  P->eps0 = eps0;
  P->bucket = bucket;
  P->avg = head.avg[0];
  P->xs = xs;
  P->minmax = d_minmax;
  if (st) {
    st->eps0 = (double)eps0;
    st->eps_bucket = bucket;
    st->avg_distance = head.avg[0];
  }

  // 4. grid at eps0.  A box-tree search with a uniform radius does not read it:
  // its cells are only counted, where a bitmap of them fits (up to 32 MB, or
  // what the fixed scratch array grants a dense table).
  if (use_tree) *use_tree = tree_applies<T>(cfg, n, d, di, k + 1, max_abs, will_stream);
  if (use_tree && *use_tree && cfg.tree_search == 1 && d == 3 && n >= TILE_3D_MIN &&
      cfg.radius_mode == KNNSJ_RADIUS_LEARNED && query_tiles<T>(cfg, d, di, k + 1)) {
    const GridGeom<T> g = grid_geometry<T>(di, P->mn, P->mx, eps0);
    if (dense_table(cfg, n, g.total_cells)) {
      launch_count_cells<T>(xs, n, g, (uint32_t*)w.dstart.get((size_t)((g.total_cells + 31) / 32) * 4), &sm->C0, s);
      unsigned long long occupied = 0;
      read_small(w, &occupied, &sm->C0, sizeof(occupied), s);
      launch_zero_words(&sm->C0, sizeof(sm->C0), s);  // (counted again by the grid)
      *use_tree = (double)n < TILE_3D_FILL * (double)(k + 1) * (double)occupied;
    }
  }
  if (use_tree && *use_tree && cfg.radius_mode != KNNSJ_RADIUS_LEARNED) {
    const GridGeom<T> g = grid_geometry<T>(di, P->mn, P->mx, eps0);
    P->grid.geom = g;
    const unsigned long long cap = cfg.dense_cells_cap ? 32ull * cfg.dense_cells_cap : 1ull << 28;
    if (g.total_cells <= cap) {
      launch_count_cells<T>(xs, n, g, (uint32_t*)w.dstart.get((size_t)((g.total_cells + 31) / 32) * 4), &sm->C0, s);
      return;
    }
  }
  if (use_tree && !*use_tree && !will_stream && query_tiles<T>(cfg, d, di, k + 1)) {
    const GridGeom<T> g = grid_geometry<T>(di, P->mn, P->mx, eps0);
    if (dense_table(cfg, n, g.total_cells)) {
      build_curve_grid<T>(w, g, xs, n, d, eps0, &sm->C0, &P->grid, &P->curve_ps, &P->curve_ids, s);
      return;
    }
  }
  build_grid<T>(w, cfg, n, d, di, P->mn, P->mx, eps0, &sm->C0, &P->grid, s);
}

// The radius model used by the learned starting radius, uploaded to the
// device when it changed since the last call.
static const float* device_model(Workspace& w, cudaStream_t s) {
  std::vector<float> m;
  const unsigned v = radius_model_snapshot(&m);
  float* dm = (float*)w.model.get(MODEL_FLOATS * 4);
  if (w.model_version != v) {
    KNNSJ_CUDA(cudaMemcpyAsync(dm, m.data(), MODEL_FLOATS * 4, cudaMemcpyHostToDevice, s));
    KNNSJ_CUDA(cudaStreamSynchronize(s));
    w.model_version = v;
  }
  return dm;
}

template <typename T>
static double decode_radius(unsigned long long bits) {
  if (sizeof(T) == 4) {
    const uint32_t b = (uint32_t)bits;
    float f;
    std::memcpy(&f, &b, 4);
    return (double)f;
  }
  double x;
  std::memcpy(&x, &bits, 8);
  return x;
}

// Runs retry passes on the device: a CUDA graph whose conditional while node
// repeats [clear the pass counters, search, loop_step_kernel] until the step
// kernel stops it.  c holds the loop state on entry and is updated on return.
// Returns false, having run nothing, when conditional graph nodes are not
// available.
template <typename T>
static bool run_graph_passes(Workspace& w, SearchLaunch<T> a, LoopCtl& c, LoopCtl* dctl, SmallDev* sm,
                             int sm_count, cudaStream_t s, cudaEvent_t e0, cudaEvent_t e1, double* kernel_ms,
                             bool upload = true, uint32_t iter_before = 0,
                             const std::function<void()>& after_launch = {}) {
  // launches are counted as they ran: the body's once per pass, the
  // condition node once
  if (upload) iter_before = c.iter;
  unsigned long long body = 0;
  cudaGraph_t g = nullptr;
  KNNSJ_CUDA(cudaGraphCreate(&g, 0));
  cudaGraphConditionalHandle h;
  if (cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault) != cudaSuccess) {
    cudaGetLastError();
    cudaGraphDestroy(g);
    return false;
  }
  // the loop state decides whether the first pass runs at all
  cudaGraphNode_t cond_node;
  {
    const LoopCtl* cp = dctl;
    void* args[] = {(void*)&cp, (void*)&h};
    cudaKernelNodeParams kp{};
    kp.func = (void*)loop_cond_kernel;
    kp.gridDim = dim3(1);
    kp.blockDim = dim3(1);
    kp.kernelParams = args;
    if (cudaGraphAddKernelNode(&cond_node, g, nullptr, 0, &kp) != cudaSuccess) {
      cudaGetLastError();
      cudaGraphDestroy(g);
      return false;
    }
  }
  // (the parameter union has no default constructor: zeroed raw storage)
  alignas(cudaGraphNodeParams) unsigned char np_raw[sizeof(cudaGraphNodeParams)];
  std::memset(np_raw, 0, sizeof(np_raw));
  cudaGraphNodeParams* np = reinterpret_cast<cudaGraphNodeParams*>(np_raw);
  np->type = cudaGraphNodeTypeConditional;
  np->conditional.handle = h;
  np->conditional.type = cudaGraphCondTypeWhile;
  np->conditional.size = 1;
  cudaGraphNode_t node;
  if (cudaGraphAddNode(&node, g, &cond_node, nullptr, 1, np) != cudaSuccess) {
    cudaGetLastError();
    cudaGraphDestroy(g);
    return false;
  }
  cudaGraph_t body_graph = np->conditional.phGraph_out[0];
  cudaGraphExec_t ex = nullptr;
  try {
    if (upload) write_small(w, dctl, &c, sizeof(LoopCtl), s);
    const unsigned long long l0 = g_launches;
    KNNSJ_CUDA(cudaStreamBeginCaptureToGraph(s, body_graph, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    try {
      a.ctl = dctl;
      a.qlist = c.list[c.cur];  // placeholders: the kernel reads the live values from dctl
      a.fail_list = c.list[c.cur ^ 1];
      a.nq = c.nq;
      launch_zero_words(&sm->fail_count, 4, s);
      launch_zero_words(&sm->fr, sizeof(FailRadii), s);
      launch_search<T>(a, sm_count, s);
      loop_step_kernel<T><<<1, 1, 0, s>>>(dctl, &sm->fail_count, &sm->fr, h, 1);
      KNNSJ_CHECK_LAUNCH();
    } catch (...) {
      cudaGraph_t dummy = nullptr;
      cudaStreamEndCapture(s, &dummy);
      throw;
    }
    KNNSJ_CUDA(cudaStreamEndCapture(s, &body_graph));
    body = g_launches - l0;
    KNNSJ_CUDA(cudaGraphInstantiate(&ex, g, 0));
    KNNSJ_CUDA(cudaEventRecord(e0, s));
    KNNSJ_CUDA(cudaGraphLaunch(ex, s));
    KNNSJ_CUDA(cudaEventRecord(e1, s));
    if (after_launch) after_launch();  // device work that can precede the host's look at the state
    read_small(w, &c, dctl, sizeof(LoopCtl), s);
    const unsigned long long passes = c.iter - iter_before;
    g_launches = g_launches - body + body * passes + 1;
  } catch (...) {
    if (ex) cudaGraphExecDestroy(ex);
    cudaGraphDestroy(g);
    throw;
  }
  float ms = 0.f;
  KNNSJ_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  *kernel_ms += ms;
  cudaGraphExecDestroy(ex);
  cudaGraphDestroy(g);
  return true;
}

// Builds the tree over the grid's point buffers (the grid is not searched
// afterwards) and runs the passes: each reads its query count on the device,
// so nothing waits for the host in between (verbose 2: a line per pass, each
// waited for).
template <typename T>
static void run_tree(Workspace& w, const Prepared<T>& P, uint64_t n, uint32_t d, uint32_t di, uint32_t K, T* qrad,
                     int32_t* d_ids, T* d_dists, double* rowsum, uint32_t* list, SmallDev* sm, int verbose,
                     cudaStream_t s) {
  BoxTree<T> t;
  tree_shape(n, d, t.count, t.offset, &t.levels, &t.nodes);
  t.dims = std::min(d, TREE_DIMS);
  t.ps = (T*)w.ps.get(tree_stride(n) * d * sizeof(T));
  t.psf = sizeof(T) == 8 ? (float*)w.psf.get(tree_stride(n) * d * sizeof(float)) : nullptr;
  t.id = (uint32_t*)w.pid.get(tree_stride(n) * 4);
  t.box = (float*)w.tree_box.get((size_t)2 * t.dims * t.nodes * 4);
  TreeScratch sc;
  sc.sort.keys[0] = (unsigned long long*)w.keys0.get(n * 8);
  sc.sort.keys[1] = (unsigned long long*)w.keys1.get(n * 8);
  sc.sort.vals[0] = (uint32_t*)w.vals0.get(n * 4);
  sc.sort.vals[1] = (uint32_t*)w.vals1.get(n * 4);
  sc.sort.hist_elems = radix_hist_elems(n);
  sc.sort.hist = (uint32_t*)w.hist.get(sc.sort.hist_elems * 4);
  sc.sort.scan_tmp_elems = scan_tmp_elems(std::max<size_t>(sc.sort.hist_elems, n + 1));
  sc.sort.scan_tmp = (uint32_t*)w.scan_tmp.get(sc.sort.scan_tmp_elems * 4);
  sc.split = (float*)w.tree_split.get(tree_split_elems() * 4);
  launch_tree_build<T>(P.xs, P.minmax, n, d, sc, t, s);
  uint32_t* mask[2] = {list, list + t.count[0]};
  launch_zero_words(list, (size_t)2 * t.count[0] * 4, s);
  TreeLaunch<T> a;
  a.tree = t;
  a.n = n;
  a.d = d;
  a.K = K;
  a.indexed = di;
  a.radius = P.eps0;
  a.qradius = qrad;
  a.out_ids = d_ids;
  a.out_d = d_dists;
  a.rowsum = rowsum;
  a.fail_mask = mask[0];
  a.fail_count = &sm->tree_fail[0];
  a.grow = (T*)w.qradius.get(n * sizeof(T));
  a.rmax_bits = &sm->tree_rmax;
  a.cand_count = &sm->cand;
  const bool report = verbose >= 2;
  uint32_t nq = (uint32_t)n;
  auto pass = [&](int i) {
    const bool timed = report && w.ev[6] && w.ev[7];
    if (timed) KNNSJ_CUDA(cudaEventRecord(w.ev[6], s));
    launch_tree_search<T>(a, w.sm_count, s);
    if (timed) KNNSJ_CUDA(cudaEventRecord(w.ev[7], s));
    if (!report) return;
    SmallHead head;
    read_small(w, &head, static_cast<SmallHead*>(sm), sizeof(head), s);
    const uint32_t nfail = i < 2 ? head.tree_fail[i] : 0u;
    float ms = 0.f;
    if (timed) KNNSJ_CUDA(cudaEventElapsedTime(&ms, w.ev[6], w.ev[7]));
    if (nq > 0)
      fprintf(stderr, "knnsj: pass %d: %u queries, %u failed, box tree, %s (largest so far %g), %.3f ms, "
              "candidates so far %llu\n", i, nq, nfail, a.unbounded ? "no radius" : "radii", decode_radius<T>(head.tree_rmax),
              ms, head.cand);
    nq = nfail;
  };
  if (w.ev[4]) KNNSJ_CUDA(cudaEventRecord(w.ev[4], s));
  pass(0);
  a.qmask = mask[0];
  a.nq_dev = &sm->tree_fail[0];
  a.qradius = a.grow;
  a.fail_mask = mask[1];
  a.fail_count = &sm->tree_fail[1];
  pass(1);
  a.qmask = mask[1];
  a.nq_dev = &sm->tree_fail[1];
  a.qradius = nullptr;
  a.unbounded = 1;
  pass(2);
  if (w.ev[5]) KNNSJ_CUDA(cudaEventRecord(w.ev[5], s));
}

template <typename T>
void run_join(Workspace& w, const JoinConfig& cfg, const T* d_aos, const T* h_aos, uint64_t n, uint32_t d,
              uint32_t k, int32_t* d_ids, T* d_dists, knnsj_stats* st, cudaStream_t s, RowStream* rows,
              double* rowsum) {
  const uint32_t K = k + 1;
  const uint32_t di = cfg.num_indexed_dims;
  cudaEvent_t* ev = w.ev;
  // a workspace without events (fixed-scratch calls) records no timings
  auto rec = [&](int i) {
    if (ev[i]) KNNSJ_CUDA(cudaEventRecord(ev[i], s));
  };
  auto elapsed = [&](int a, int b) -> float {
    float ms = 0.f;
    if (ev[a] && ev[b]) KNNSJ_CUDA(cudaEventElapsedTime(&ms, ev[a], ev[b]));
    return ms;
  };
  g_launches = 0;
  rec(0);
  Prepared<T> P;
  const bool will_stream = rows && rows->chunks >= 2 && n >= (uint64_t)rows->chunks;
  bool use_tree = false;
  prepare<T>(w, cfg, d_aos, h_aos, n, d, k, st, s, &P, will_stream, &use_tree);
  SmallDev* sm = (SmallDev*)w.small.p;
  rec(1);

  // 5. starting radii: eps0 for every query (plain), or one per query
  T* qrad = nullptr;
  double rmax = (double)P.eps0;
  if (cfg.radius_mode == KNNSJ_RADIUS_LEARNED) {
    qrad = (T*)w.qradius.get(n * sizeof(T));
    // (a box-tree search does not care how many cells a radius spans)
    const double max_cells = use_tree ? 64.0 : learned_max_cells(di);
    launch_radius_assign<T>(P.grid, n, d, k, (float)cfg.beta, device_model(w, s), (double)P.eps0,
                            (float)cfg.radius_offset, max_cells, qrad, &sm->mlp_err, w.sm_count, s);
    rmax = (double)P.eps0 * max_cells;
  }
  // 5b. the first pass's tile search (2-D / 3-D float data, all indexed)
  TileSetup<T> tile;
  if (!use_tree && cfg.tile_search && tile_search_applies(d, di, K, P.grid.dense, sizeof(T))) {
    // per-query starting radii: query tiles over a grid of width eps0/4; a
    // uniform radius: one warp per query over a grid of width eps0/2
    // (measured best for each on the 25M-point sky-like set).  Streamed rows
    // search blocks of query ids, spread over the whole dataset: one warp
    // per query there.
    const bool tiles = !will_stream && query_tiles<T>(cfg, d, di, K);
    const int fine = cfg.tile_fine > 0 ? cfg.tile_fine : (tiles ? 4 : 2);
    prepare_tile<T>(w, tiles, fine, P.grid, P.curve_ps, P.curve_ids, n, d, P.eps0, P.mx, &tile, s);
  }

  // 6. retry loop (main.cu:312-430)
  uint32_t* list[2] = {(uint32_t*)w.list0.get(n * 4), (uint32_t*)w.list1.get(n * 4)};
  SearchLaunch<T> a;
  a.grid = P.grid;
  a.xs = P.xs;
  a.n = n;
  a.d = d;
  a.K = K;
  a.out_ids = d_ids;
  a.out_d = d_dists;
  a.rowsum = rowsum;
  a.fail_count = &sm->fail_count;
  a.cand_count = &sm->cand;
  a.work_counter = &sm->work_counter;
  a.fail_radii = &sm->fr;
  a.qradius = qrad;
  a.shape.warps_per_block = cfg.search_warps;
  a.shape.qchunk = cfg.search_qchunk;
  a.shape.buffer = cfg.search_buffer;
  a.coord_bound = cfg.float_prefilter ? P.max_abs : INFINITY;
  T r = P.eps0;
  const double step = (double)P.eps0 * 0.5;
  a.step = (T)step;
  uint32_t nq = (uint32_t)n;
  int iter = 0, regrids = 0, cur = 0;
  uint64_t queries_run = 0;
  double kernel_ms = 0.0, alg_bytes = 0.0, rmax_seen = rmax;
  double rgrid = rmax;  // the radius a rebuilt grid is sized for
  double redge[FAIL_RADIUS_BINS];
  for (int b = 0; b < FAIL_RADIUS_BINS; b++) redge[b] = (double)P.eps0 * std::exp2((b - 15) / 4.0);
  const int max_iter = cfg.max_iterations > 0 ? cfg.max_iterations : 100000;
  double r_limit = regrid_limit((double)a.grid.geom.width, di);
  const double ring_div = ring_div_of(di);
  // passes after the first run inside a CUDA graph (no host round trip per
  // pass) unless the stream cannot be captured (the legacy default stream)
  bool graph_ok = cfg.use_graph && s != nullptr && ev[4] != nullptr && cfg.verbose < 2;
  LoopCtl* dctl = &sm->ctl;

  // 6a. streamed rows: the first pass in blocks of query ids, each block's
  // rows copied into the host buffers while the next block searches.  The
  // copies keep the host link busy, so the pass bookkeeping stays on the
  // device (the step kernel, then the retry graph) with no host round trip
  // until the graph stops.
  // (the caller waits for the copies and patches the late rows in:
  // finish_row_stream)
  const bool streamed = will_stream;
  bool checksum_done = false;  // streamed rows: the checksum of the final table is launched
  if (streamed) {
    w.ensure_copy_stream();
    w.mail = true;
    rows->active = true;
    const int C = std::min(rows->chunks, MAX_ROW_CHUNKS);
    const uint32_t crow = (uint32_t)((n + C - 1) / C);
    uint32_t* clist = (uint32_t*)w.chunk_list.get(n * 4);
    const bool dev_loop = graph_ok;
    LoopCtl c{};
    c.nq = (uint32_t)n;
    c.iter = 0;
    c.cur = 0;
    c.stop_iter = (uint32_t)std::min<int64_t>((int64_t)max_iter, 256);
    c.list[0] = list[0];
    c.list[1] = list[1];
    c.r = (double)r;
    c.step = step;
    c.rmax = rmax;
    c.rgrid = rgrid;
    c.rmax_seen = rmax_seen;
    for (int b = 0; b < FAIL_RADIUS_BINS; b++) c.redge[b] = redge[b];
    c.r_limit = r_limit;
    c.width = (double)a.grid.geom.width;
    c.per_query = qrad ? 1 : 0;
    c.ring_div = ring_div;
    c.go = 0;
    if (dev_loop) write_small(w, dctl, &c, sizeof(LoopCtl), s);
    launch_zero_words(sm->chunk_fill, sizeof(sm->chunk_fill), s);
    chunk_lists_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a.grid.pid, nullptr, (uint32_t)n, crow,
                                                                   sm->chunk_fill, clist);
    KNNSJ_CHECK_LAUNCH();
    launch_zero_words(&sm->fail_count, 4, s);
    launch_zero_words(&sm->fr, sizeof(FailRadii), s);
    a.radius = r;
    a.fail_list = list[1];
    KNNSJ_CUDA(cudaEventRecord(ev[6], s));
    for (int ch = 0; ch < C; ch++) {
      const uint64_t r0 = (uint64_t)ch * crow;
      if (r0 >= n) break;
      const uint64_t nr = std::min<uint64_t>(crow, n - r0);
      a.qlist = clist + r0;
      a.nq = (uint32_t)nr;
      // (the queries of a block of ids are spread over the whole dataset:
      // the per-query search, over the finer grid when one is set up)
      SearchLaunch<T> c = a;
      if (tile.on) c.grid = tile.cand;
      launch_search<T>(c, w.sm_count, s);
      KNNSJ_CUDA(cudaEventRecord(w.chunk_ev[ch], s));
      KNNSJ_CUDA(cudaStreamWaitEvent(w.copy_stream, w.chunk_ev[ch], 0));
      KNNSJ_CUDA(cudaMemcpyAsync((int32_t*)rows->ids_host + r0 * K, d_ids + r0 * K, nr * K * 4,
                                 cudaMemcpyDeviceToHost, w.copy_stream));
      KNNSJ_CUDA(cudaMemcpyAsync((T*)rows->d_host + r0 * K, d_dists + r0 * K, nr * K * sizeof(T),
                                 cudaMemcpyDeviceToHost, w.copy_stream));
    }
    KNNSJ_CUDA(cudaEventRecord(ev[7], s));
    // the block lists are spent: they keep the failures for the patch
    save_fail_list_kernel<<<(unsigned)(w.sm_count * 4), 256, 0, s>>>(list[1], &sm->fail_count, clist,
                                                                    &sm->patch_count);
    KNNSJ_CHECK_LAUNCH();
    alg_bytes += (double)n * d * sizeof(T);  // the pass's candidate columns; the rest is counted below
    bool ran = false;
    if (dev_loop) {
      loop_step_kernel<T><<<1, 1, 0, s>>>(dctl, &sm->fail_count, &sm->fr, 0, 0);
      KNNSJ_CHECK_LAUNCH();
      // the result checksum goes right behind the graph: if the graph
      // finishes the join, it overlaps the row copies (the host's read of the
      // loop state waits behind them)
      auto early_checksum = [&]() {
        if (rows->checksum) {
          launch_checksum<T>(d_dists, n * K, sm->cpart, &sm->csum, s);
          checksum_done = true;
        }
      };
      ran = run_graph_passes<T>(w, a, c, dctl, sm, w.sm_count, s, ev[4], ev[5], &kernel_ms, false, 1,
                                early_checksum);
      if (ran) {
        const int passes = (int)c.iter - 1;
        alg_bytes += (double)passes * n * d * sizeof(T);
      } else {
        graph_ok = false;
        read_small(w, &c, dctl, sizeof(LoopCtl), s);
      }
    } else {  // host bookkeeping, as after any host-driven pass
      uint32_t nfail = 0;
      FailRadii fr{};
      read_small(w, &nfail, &sm->fail_count, 4, s);
      if (qrad) read_small(w, &fr, &sm->fr, sizeof(FailRadii), s);
      c.queries_run = n;
      c.accepted = n - nfail;
      c.nq = nfail;
      c.iter = 1;
      c.cur = 1;
      if (nfail > 0) {
        if (qrad) {
          c.rmax = decode_radius<T>(fr.rmax_bits);
          c.rgrid = median_fail_radius(fr.hist, nfail, redge, c.rmax);
        } else {
          c.r = (double)(T)((double)r + step);  // main.cu:336
          c.rmax = c.r;
          c.rgrid = c.rmax;
        }
        c.rmax_seen = std::max(c.rmax_seen, c.rmax);
      }
    }
    float first_ms = 0.f;
    KNNSJ_CUDA(cudaEventSynchronize(ev[7]));
    KNNSJ_CUDA(cudaEventElapsedTime(&first_ms, ev[6], ev[7]));
    kernel_ms += first_ms;
    alg_bytes += (double)c.queries_run * d * sizeof(T) + (double)c.accepted * K * (4.0 + sizeof(T));
    queries_run += c.queries_run;
    iter = (int)c.iter;
    cur = (int)c.cur;
    nq = c.nq;
    r = (T)c.r;
    rmax = c.rmax;
    rgrid = c.rgrid;
    rmax_seen = c.rmax_seen;
  }

  // 6b. the box tree: every query at its starting radius, the failures at a
  // radius grown from what they found, and the rest without a radius
  if (use_tree) {
    run_tree<T>(w, P, n, d, di, K, qrad, d_ids, d_dists, rowsum, list[0], sm, cfg.verbose, s);
    regrids = 1;  // the index was rebuilt once, as the tree
    nq = 0;       // (the passes are counted from the head below)
  }

  while (nq > 0) {
    checksum_done = false;  // more passes change the table
    if (iter >= max_iter) throw StatusError{KNNSJ_ERR_NO_CONVERGENCE, "iteration cap reached"};
    // learned starting radii are clamped so their rings stay small on the
    // eps0 grid: no rebuild for the first pass
    const bool first_learned = qrad && iter == 0;
    if (!first_learned && regrid_due(rgrid, rmax, r_limit, (double)a.grid.geom.width, ring_div)) {
      // sparse-query tail: when the largest radius has outgrown the grid
      // (its ring would pass the row cap) and only a handful of queries are
      // left (nq * n <= 2^32 distances), they are finished exactly by a scan
      // over all points instead of a grid coarse enough for that radius
      // (tail_brute 2, for tests: at any due rebuild)
      const bool outgrown = ring_too_wide(rmax, (double)a.grid.geom.width, ring_div) || cfg.tail_brute == 2;
      if (cfg.tail_brute && outgrown && nq <= 4096 && (uint64_t)nq * n <= (1ull << 32)) {
        a.qlist = list[cur];
        a.nq = nq;
        rec(4);
        launch_brute<T>(a, s);
        rec(5);
        KNNSJ_CUDA(cudaStreamSynchronize(s));
        kernel_ms += elapsed(4, 5);
        alg_bytes += (double)nq * n * d * sizeof(T) + (double)nq * K * (4.0 + sizeof(T));
        queries_run += nq;
        iter++;
        nq = 0;
        break;
      }
      // coarser grid for the radius in flight (like main.cu:333-356); the
      // widened width keeps that radius's ring at three cells per dimension
      const T wnew = (T)(rgrid * (1.0 + 1.0 / 32768.0));
      build_grid<T>(w, cfg, n, d, di, P.mn, P.mx, wnew, &sm->C, &a.grid, s);
      r_limit = regrid_limit((double)a.grid.geom.width, di);
      regrids++;
    }
    if (graph_ok && iter >= 1) {
      LoopCtl c{};
      c.nq = nq;
      c.iter = (uint32_t)iter;
      c.cur = (uint32_t)cur;
      c.stop_iter = (uint32_t)std::min<int64_t>((int64_t)max_iter, (int64_t)iter + 256);
      c.list[0] = list[0];
      c.list[1] = list[1];
      c.r = (double)r;
      c.step = step;
      c.rmax = rmax;
      c.rgrid = rgrid;
      c.rmax_seen = rmax_seen;
      for (int b = 0; b < FAIL_RADIUS_BINS; b++) c.redge[b] = redge[b];
      c.r_limit = r_limit;
      c.width = (double)a.grid.geom.width;
      c.per_query = qrad ? 1 : 0;
      c.ring_div = ring_div;
      c.go = 1;
      if (run_graph_passes<T>(w, a, c, dctl, sm, w.sm_count, s, ev[4], ev[5], &kernel_ms)) {
        const int passes = (int)c.iter - iter;
        alg_bytes += (double)passes * n * d * sizeof(T) + (double)c.queries_run * d * sizeof(T) +
                     (double)c.accepted * K * (4.0 + sizeof(T));
        queries_run += c.queries_run;
        iter = (int)c.iter;
        cur = (int)c.cur;
        nq = c.nq;
        r = (T)c.r;
        rmax = c.rmax;
        rgrid = c.rgrid;
        rmax_seen = c.rmax_seen;
        continue;
      }
      graph_ok = false;  // conditional graphs unavailable: host-driven passes
    }
    a.qlist = iter == 0 ? nullptr : list[cur];
    a.nq = nq;
    a.radius = r;
    a.fail_list = list[cur ^ 1];
    launch_zero_words(&sm->fail_count, 4, s);
    launch_zero_words(&sm->fr, sizeof(FailRadii), s);
    rec(4);
    if (iter == 0)
      first_pass_search<T>(w, a, tile, sm, s);
    else
      launch_search<T>(a, w.sm_count, s);
    rec(5);
    struct {
      uint32_t fail;
      uint32_t pad;
      FailRadii fr;
    } tail;
    read_small(w, &tail.fail, &sm->fail_count, 4, s);
    if (qrad) read_small(w, &tail.fr, &sm->fr, sizeof(FailRadii), s);
    const uint32_t nfail = tail.fail;
    const float pass_ms = elapsed(4, 5);
    kernel_ms += pass_ms;
    if (cfg.verbose >= 2) {  // one line per pass
      unsigned long long cand_now = 0;
      KNNSJ_CUDA(cudaMemcpy(&cand_now, &sm->cand, 8, cudaMemcpyDeviceToHost));
      fprintf(stderr, "knnsj: pass %d: %u queries, %u failed, radius %g (largest %g), grid width %g, %.3f ms, "
              "candidates so far %llu\n", iter, nq, nfail, (double)r, rmax, (double)a.grid.geom.width, pass_ms,
              cand_now);
    }
    // candidate columns read once, query rows read, accepted rows written
    alg_bytes += (double)n * d * sizeof(T) + (double)nq * d * sizeof(T) +
                 (double)(nq - nfail) * K * (4.0 + sizeof(T));
    queries_run += nq;
    nq = nfail;
    cur ^= 1;
    iter++;
    if (nq > 0) {
      if (qrad) {
        rmax = decode_radius<T>(tail.fr.rmax_bits);  // largest grown radius among the failures
        rgrid = median_fail_radius(tail.fr.hist, nfail, redge, rmax);
      } else {
        r = (T)((double)r + step);  // main.cu:336
        rmax = (double)r;
        rgrid = rmax;
      }
      rmax_seen = std::max(rmax_seen, rmax);
    }
  }
  rec(2);
  if (streamed) {
    // the result checksum runs while the last row copies are in flight; the
    // wait for them and the late rows follow, and the small reads below come
    // after the copies instead of queueing behind them
    if (rows->checksum && !checksum_done) launch_checksum<T>(d_dists, n * K, sm->cpart, &sm->csum, s);
    finish_row_stream<T>(w, *rows, d_ids, d_dists, K, s);
    rec(3);
    w.mail = false;
    if (rows->checksum) read_small(w, &rows->total_distance, &sm->csum, sizeof(double), s);
  }
  if (rowsum && st) launch_sum_f64(rowsum, n, sm->cpart, &sm->csum, s);
  SmallHead head;
  read_small(w, &head, static_cast<SmallHead*>(sm), sizeof(head), s);
  if (rowsum && st) st->total_distance = head.csum;
  const unsigned long long cand = head.cand;
  const uint32_t mlp_err = qrad ? head.mlp_err : 0u;
  if (use_tree) {
    iter = 1 + (head.tree_fail[0] > 0) + (head.tree_fail[1] > 0);
    queries_run = n + head.tree_fail[0] + head.tree_fail[1];
    kernel_ms += elapsed(4, 5);
    alg_bytes += (double)iter * n * d * sizeof(T) + (double)queries_run * d * sizeof(T) +
                 (double)n * K * (4.0 + sizeof(T));
    rmax_seen = decode_radius<T>(head.tree_rmax);
  }
  if (mlp_err && cfg.verbose)  // rows are still exact: the affected queries started at eps0
    fprintf(stderr, "knnsj: the tensor-core radius model timed out (%u); those queries started at eps0\n", mlp_err);
  if (st) {
    st->iterations = iter;
    st->regrids = regrids;
    st->eps_final = qrad || use_tree ? rmax_seen : (double)r;
    st->candidates = cand;
    st->queries_run = queries_run;
    st->kernel_launches = g_launches;
    st->ms_search_kernels = kernel_ms;
    st->search_alg_bytes = alg_bytes;
    st->search_alg_flops = 3.0 * d * (double)cand;
    st->radius_model_error = (double)mlp_err;
    st->tile_handovers = (double)head.defer_total;
    st->nonempty_cells = head.C0;
    const float a01 = elapsed(0, 1), a12 = elapsed(1, 2);
    st->ms_prep = a01;
    st->ms_search = a12;
    st->ms_total = a01 + a12;
    if (streamed) st->ms_transfer = elapsed(2, 3);  // the row copies that outlast the join
  }
}

// Features of the learned starting radius for every point (by input row),
// on the eps0 grid of a (plain) join of the same data and k.
template <typename T>
void run_features(Workspace& w, const JoinConfig& cfg, const T* d_aos, const T* h_aos, uint64_t n, uint32_t d,
                  uint32_t k, float* d_out, double* eps0_out, cudaStream_t s) {
  g_launches = 0;
  Prepared<T> P;
  prepare<T>(w, cfg, d_aos, h_aos, n, d, k, nullptr, s, &P);
  launch_radius_features<T>(P.grid, n, d, k, (float)cfg.beta, d_out, s);
  KNNSJ_CUDA(cudaStreamSynchronize(s));
  if (eps0_out) *eps0_out = (double)P.eps0;
}

template <typename T>
double device_checksum(Workspace& w, const T* d_vals, uint64_t count, cudaStream_t s) {
  SmallDev* sm = (SmallDev*)w.small.get(sizeof(SmallDev));
  launch_checksum<T>(d_vals, count, sm->cpart, &sm->csum, s);
  double v = 0.0;
  read_small(w, &v, &sm->csum, sizeof(v), s);
  return v;
}
template double device_checksum<float>(Workspace&, const float*, uint64_t, cudaStream_t);
template double device_checksum<double>(Workspace&, const double*, uint64_t, cudaStream_t);

// Streamed rows: waits (on s) for every block copy, then writes the rows
// that passes after the first finished into the host buffers.  The caller
// synchronises s.
template <typename T>
void finish_row_stream(Workspace& w, const RowStream& rows, const int32_t* d_ids, const T* d_dists, uint32_t K,
                       cudaStream_t s) {
  SmallDev* sm = (SmallDev*)w.small.p;
  KNNSJ_CUDA(cudaEventRecord(w.chunk_ev[MAX_ROW_CHUNKS], w.copy_stream));
  KNNSJ_CUDA(cudaStreamWaitEvent(s, w.chunk_ev[MAX_ROW_CHUNKS], 0));
  patch_rows_kernel<T><<<(unsigned)(w.sm_count * 8), 256, 0, s>>>((const uint32_t*)w.chunk_list.p, &sm->patch_count,
                                                                  d_ids, d_dists, K, (int32_t*)rows.ids_dev,
                                                                  (T*)rows.d_dev);
  KNNSJ_CHECK_LAUNCH();
}

template void finish_row_stream<float>(Workspace&, const RowStream&, const int32_t*, const float*, uint32_t,
                                       cudaStream_t);
template void finish_row_stream<double>(Workspace&, const RowStream&, const int32_t*, const double*, uint32_t,
                                        cudaStream_t);

template void run_join<float>(Workspace&, const JoinConfig&, const float*, const float*, uint64_t, uint32_t,
                              uint32_t, int32_t*, float*, knnsj_stats*, cudaStream_t, RowStream*, double*);
template void run_join<double>(Workspace&, const JoinConfig&, const double*, const double*, uint64_t,
                               uint32_t, uint32_t, int32_t*, double*, knnsj_stats*, cudaStream_t,
                               RowStream*, double*);
template void run_features<float>(Workspace&, const JoinConfig&, const float*, const float*, uint64_t, uint32_t,
                                  uint32_t, float*, double*, cudaStream_t);
template void run_features<double>(Workspace&, const JoinConfig&, const double*, const double*, uint64_t,
                                   uint32_t, uint32_t, float*, double*, cudaStream_t);

}  // namespace knnsj
