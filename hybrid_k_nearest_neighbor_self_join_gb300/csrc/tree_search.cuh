// tree_search.cuh -- search of the box tree (k_tree.cu): the k+1 nearest points
// of a tile of queries by one warp.  Compiled once per data type
// (k_tree_f32.cu, k_tree_f64.cu).
//
// A warp owns Q queries of one leaf.  From that leaf it goes up the tree: the
// 32 children of a node are tested 32 lanes at a time against every query of
// the tile, the boxes that can hold a point under a query's threshold are
// descended, and a leaf's 32 points are loaded once and evaluated for each
// query that needs them.  A query's
// threshold starts at its radius (or without bound) and falls as its buffer
// of keys is reduced to the K best.
//
// Exactness: a box is skipped for a query only when no point in it can have a
// computed squared distance at or below the threshold.  Float data: for a
// point inside the box every rounded difference p - q is at least the rounded
// gap between the box and q, and the chain of fused multiply-adds is monotone
// in each term, so the same chain over the gaps is a lower bound of the
// computed distance, bit for bit.  Double data: boxes (rounded outward) and
// points are compared in float against a widened threshold (screen_bound), and
// what passes gets its distance in double, 32 points at a time.
//
// What bounds it: issue slots and latency at 24 warps per SM (80 registers),
// not memory (L2 hits 98 %): 5 550 warp instructions per query of a 1 M-point
// 6-D double join at 0.52 per cycle and scheduler; 65 leaves per query at 10 M.
// Search kernels of whole joins, one warp per query on the grid's ring
// (k_search.cu) before, this now: 10 M x 6-D double k = 16 790 -> 129 ms, 5 M x
// 4-D float k = 128 103 -> 45 ms, 60 k x 12-D k = 15 125 -> 2.2 ms, 1 M x 3-D
// k = 32 9.6 -> 4.2-4.9 ms.  Queries per warp, measured before the points lay in
// rows per leaf: 2 at 24 warps per SM 147 and 49 ms, 4 at 16 warps 146 and 51
// ms, 8 spill (333 and 61 ms).  Blocks of 8 warps on consecutive tiles share
// the L1 better than blocks of 4 (4 queries per warp, 6-D: 146 against 154 ms).
#pragma once

#include <cmath>

#include "knnsj_internal.h"
#include "select.cuh"

namespace knnsj {

namespace {

constexpr int TREE_THREADS = 256;  // largest block
// blocks per SM: 80 registers, and 64 in three dimensions (1M points: 4.5 and
// 4.2 ms; two dimensions 11.2 and 11.1 ms at 3M but 0.21 and 0.22 at 100 000;
// six spill: 147 and 187 ms)
constexpr int tree_min_blocks(int d) { return d == 3 ? 4 : 3; }
constexpr int TREE_Q = 2;          // queries per warp
constexpr int TREE_QUEUE = 64;     // double data: candidates that passed the float screen, per query
constexpr size_t TREE_MAX_SMEM = 110 * 1024;  // dynamic shared memory of a block
constexpr int TREE_STACK = 6;      // levels above the leaves' parents
constexpr uint32_t TREE_CHUNK = 64;  // tiles of a block's run of consecutive queries

template <typename T>
struct TreeParams {
  BoxTree<T> t;
  uint64_t n;
  uint32_t d, K, B;
  const uint32_t* qmask;   // bit b of word L: tree position 32 L + b is a query (nullptr: all)
  const uint32_t* nq_dev;  // with qmask: how many there are
  T radius;
  T* qradius;              // per-query radii by original id (nullptr: radius for all)
  int unbounded;           // no radius: every query ends with its K nearest
  float inv_di;            // 1 / indexed dimensions (growth of a failed radius)
  int32_t* out_ids;
  T* out_d;
  double* rowsum;
  uint32_t* fail_mask;     // bits of the failed queries (cleared before the pass)
  uint32_t* fail_count;
  T* grow;                 // radii of the failed queries by original id
  unsigned long long* rmax_bits;  // largest radius searched or grown
  unsigned long long* cand_count;
};

// Double data is searched in float first.  A point at distance sqrt(t) or less
// from the query has a float distance (coordinates of both rounded to float,
// float chain) whose square is at most the result, and so has the gap to any
// box that holds it: rounding moves a coordinate x by at most 2^-24 |x|, the
// point lies within |q| + sqrt(t) of the origin, and the chain of d terms is
// off by (d + 8) 2^-23 of the result and, where terms are subnormal, by half of
// the smallest float (2^-149) per term.
__device__ __forceinline__ float screen_bound(float t_up, float qnorm, uint32_t d) {
  const float s = __fsqrt_ru(__fmul_ru(t_up, 1.0f + 1.0f / 1048576.0f));
  const float e = __fmaf_ru(__fmaf_ru(2.0f, qnorm, s), 1.01f / 16777216.0f, 1e-37f);
  const float w = __fadd_ru(s, e);
  return __fadd_ru(__fmul_ru(__fmul_ru(w, w), 1.0f + (float)(d + 8) * 1.2e-7f), __uint_as_float(d));  // (d 2^-149)
}

// A warp's state in shared memory, one entry per query of its tile.  The scan
// works on register copies; the rare steps (settle, the row's write) loop over
// the queries here, so that their code exists once: the first version unrolled
// them per query and spent 21 of 27 cycles per instruction waiting for
// instruction fetches.
template <typename T, int Q>
struct alignas(16) TreeState {  // (what follows it in shared memory is read 16 bytes at a time)
  typename Key<T>::type tau[Q];  // a key passes when it is below
  uint32_t len[Q];               // keys held
  uint32_t trig[Q];              // more keys than this are reduced
  uint32_t qn[Q];                // double data: queued candidates
};

// Appends the lanes' keys that pass to query i's buffer and reduces the buffer
// when it is due.
template <typename T, int Q>
__device__ __forceinline__ void tree_shrink(const TreeParams<T>& p, TreeState<T, Q>* ts, typename Key<T>::type* buf,
                                            uint32_t* hist, int i, int lane) {
  Sel<T> st;
  st.len = ts->len[i];
  st.tau = ts->tau[i];
  st.tight = false;
  // (without a bound the first reduction only finds the largest key)
  int rounds = to_float_up(Key<T>::acc(st.tau)) < 3.0e38f ? 1 : 2;
#pragma unroll 1
  for (; rounds > 0; rounds--) st = reduce<T>(buf, hist, st, p.K, p.B, lane);
  __syncwarp();
  if (lane == 0) {
    ts->len[i] = st.len;
    ts->tau[i] = st.tau;
    // the next reduction pays once half as many keys again have come in
    ts->trig[i] = min(p.B - 32, st.len + max(p.K >> 1, 24u));
  }
  __syncwarp();
}

// Queued candidates of double data whose queue holds `least` or more get
// their exact distances, 32 at a time; buffers past their trigger are reduced.
template <typename T, int D, int Q>
__device__ __noinline__ void tree_settle(const TreeParams<T>& p, TreeState<T, Q>* ts, typename Key<T>::type* bufs,
                                         uint32_t* hist, const uint32_t* queue, const T* qsm, uint32_t least) {
  using Kt = Key<T>;
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int i = 0; i < Q; i++) {
    typename Kt::type* buf = bufs + (size_t)i * p.B;
    if constexpr (sizeof(T) == 8) {
      uint32_t qn = ts->qn[i];
      if (qn >= least) {
        const uint32_t cnt = min(qn, 32u);
        qn -= cnt;
        bool pass = false;
        typename Kt::type key = Kt::maxv();
        if (lane < (int)cnt) {
          const uint32_t j = queue[i * TREE_QUEUE + qn + lane];
          const T* qc = qsm + (D > 0 ? i * D : i * (int)p.d);
          const T* x = p.t.ps + (uint64_t)(j >> 5) * 32 * (D > 0 ? (uint32_t)D : p.d) + (j & 31u);
          T acc = 0;
          if (D > 0) {
#pragma unroll
            for (int l = 0; l < (D > 0 ? D : 1); l++) {
              const T t = Num<T>::sub(x[l * 32], qc[l]);
              acc = Num<T>::fma(t, t, acc);
            }
          } else {
#pragma unroll 4
            for (uint32_t l = 0; l < p.d; l++) {
              const T t = Num<T>::sub(x[l * 32], qc[l]);
              acc = Num<T>::fma(t, t, acc);
            }
          }
          key = Kt::make(acc, p.t.id[j]);
          pass = Kt::less(key, ts->tau[i]);
        }
        const unsigned m = __ballot_sync(FULL, pass);
        const uint32_t len = ts->len[i];
        if (pass) buf[len + __popc(m & lanemask_lt())] = key;
        __syncwarp();
        if (lane == 0) {
          ts->len[i] = len + __popc(m);
          ts->qn[i] = qn;
        }
        __syncwarp();
      }
    }
    if (ts->len[i] > ts->trig[i]) tree_shrink<T, Q>(p, ts, buf, hist, i, lane);
  }
}

template <typename T, int D, int Q>
struct TreeTile {
  using Kt = Key<T>;
  using KT = typename Kt::type;
  static constexpr int QD = D > 0 ? D : 1;
  const TreeParams<T>& p;
  const int lane;
  TreeState<T, Q>* ts;
  KT* buf;           // [Q][B]
  uint32_t* hist;    // [256]
  float* stk;        // [TREE_STACK][32]
  uint32_t* queue;   // [Q][TREE_QUEUE] (double)
  T* qsm;            // [Q][d]: query coordinates (double data)
  float* qfm;        // [d][Q]: the same in float (runtime d)
  float q[Q][QD];    // query coordinates rounded to float (exact for float data)
  float tauf[Q];     // bound of the float distance of points and boxes that matter; -1: no query
  uint32_t tid[Q];   // float data: the threshold key's id
  uint32_t len[Q], trig[Q];
  float qnorm[Q];    // double data: at least |q|
  uint32_t qn[Q];    // double: queue length
  uint32_t scanned = 0;  // leaves scanned, per query

  __device__ __forceinline__ TreeTile(const TreeParams<T>& p_, int lane_) : p(p_), lane(lane_) {}

  // registers from the shared state (a query without a threshold stays off)
  __device__ __forceinline__ void load_state() {
#pragma unroll
    for (int i = 0; i < Q; i++) {
      len[i] = ts->len[i];
      trig[i] = ts->trig[i];
      const KT t = ts->tau[i];
      float b = to_float_up(Kt::acc(t));
      if constexpr (sizeof(T) == 4) {
        tid[i] = Kt::id(t);
      } else {
        qn[i] = ts->qn[i];
        b = screen_bound(b, qnorm[i], p.d);
      }
      if (tauf[i] >= 0.0f) tauf[i] = b;
    }
  }

  // `flush`: every queued candidate (at the end of a tile)
  __device__ __forceinline__ void settle(bool flush) {
    __syncwarp();
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < Q; i++) {
        ts->len[i] = len[i];
        if constexpr (sizeof(T) == 8) ts->qn[i] = qn[i];
      }
    }
    __syncwarp();
    tree_settle<T, D, Q>(p, ts, buf, hist, queue, qsm, flush ? 1u : 32u);
    __syncwarp();
    load_state();
  }

  // The points of leaf c of a node for the queries whose masks pm hold bit c.
  // True when the shared state has changed.
  __device__ __forceinline__ bool scan_leaf(uint32_t leaf, int c, const unsigned (&pm)[Q]) {
    // (the points that fill up the last leaf lie at infinity, with an id that
    // no threshold key exceeds)
    const float* src = (sizeof(T) == 4 ? reinterpret_cast<const float*>(p.t.ps) : p.t.psf) +
                       (uint64_t)leaf * 32 * (D > 0 ? (uint32_t)D : p.d) + lane;
    bool due = false;
    auto take = [&](int i, float a) {
      bool pass = a <= tauf[i];
      unsigned m = __ballot_sync(FULL, pass);
      scanned++;
      if (m) {
        if constexpr (sizeof(T) == 4) {
          const uint32_t id = p.t.id[leaf * 32 + lane];
          // (equal to the threshold distance: the smaller id passes)
          pass = pass && (a < tauf[i] || id < tid[i]);
          m = __ballot_sync(FULL, pass);
          if (pass) buf[(size_t)i * p.B + len[i] + __popc(m & lanemask_lt())] = Kt::make(a, id);
          len[i] += __popc(m);
          due |= len[i] > trig[i];
        } else {
          if (pass) queue[i * TREE_QUEUE + qn[i] + __popc(m & lanemask_lt())] = leaf * 32 + lane;
          qn[i] += __popc(m);
          due |= qn[i] >= 32;
        }
      }
    };
    if (D > 0) {
      float x[QD];
#pragma unroll
      for (int l = 0; l < QD; l++) x[l] = src[l * 32];
#pragma unroll
      for (int i = 0; i < Q; i++) {
        if (pm[i] >> c & 1u) {
          float a = 0.0f;
#pragma unroll
          for (int l = 0; l < QD; l++) {
            const float t = __fsub_rn(x[l], q[i][l]);
            a = __fmaf_rn(t, t, a);
          }
          take(i, a);
        }
      }
    } else {
      float acc[Q];
#pragma unroll
      for (int i = 0; i < Q; i++) acc[i] = 0.0f;
#pragma unroll 4
      for (uint32_t l = 0; l < p.d; l++) {
        const float x = src[l * 32];
#pragma unroll
        for (int i = 0; i < Q; i++) {
          const float t = __fsub_rn(x, qfm[l * Q + i]);
          acc[i] = __fmaf_rn(t, t, acc[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < Q; i++)
        if (pm[i] >> c & 1u) take(i, acc[i]);
    }
    if (due) settle(false);
    return due;
  }

  // Lower bounds of the (float) squared distance from each query to the points
  // in the box of child lane ^ flip of a node, at `level` (NaN: no such child).
  __device__ __forceinline__ void box_bounds(uint32_t level, uint32_t node, uint32_t flip, float (&lb)[Q]) {
    const uint32_t c = lane ^ flip;
    const bool there = node * 32 + c < p.t.count[level];
    const float* box = p.t.box + (uint64_t)((p.t.offset[level] >> 5) + node) * 64 * (D > 0 ? (uint32_t)D : p.t.dims) + c;
#pragma unroll
    for (int i = 0; i < Q; i++) lb[i] = 0.0f;
    auto dim = [&](uint32_t l, auto qof) {
      const float lo = box[l * 64];
      const float hi = box[l * 64 + 32];
#pragma unroll
      for (int i = 0; i < Q; i++) {
        const float v = qof(i);
        const float g = fmaxf(fmaxf(__fsub_rn(lo, v), __fsub_rn(v, hi)), 0.0f);
        lb[i] = __fmaf_rn(g, g, lb[i]);
      }
    };
    if (D > 0) {
#pragma unroll
      for (int l = 0; l < QD; l++) dim(l, [&](int i) { return q[i][l]; });
    } else {
#pragma unroll 2
      for (uint32_t l = 0; l < p.t.dims; l++) dim(l, [&](int i) { return qfm[l * Q + i]; });
    }
#pragma unroll
    for (int i = 0; i < Q; i++)
      if (!there) lb[i] = __int_as_float(0x7fc00000);
  }

  // The walk: the own leaf's parent first, then for every node above it the
  // other children, nearest first, down to the leaves.
  __device__ __forceinline__ void search(uint32_t own) {
    const float none = __int_as_float(0x7fc00000);
    const int root = p.t.levels;  // level of the (virtual) root, the parent of the last level
    int top = 1, level = 1;       // the children of `node`, at level - 1, come next
    uint32_t node = own >> 5;
    bool fresh = false;           // node lies on the path to the own leaf
    for (;;) {
      // (lane l tests child l ^ flip: under the own node the leaves come in
      // the order of the splits that part them from the own leaf)
      const uint32_t flip = level == 1 && top == 1 ? own & 31u : 0u;
      float lb[Q];
      box_bounds(level - 1, node, flip, lb);
      float cur = none;  // level > 1: smallest bound over the queries that can use this lane's child
      if (level == 1) {
        unsigned pm[Q], todo = FULL;
        bool changed = true;
        for (;;) {
          if (changed) {
#pragma unroll
            for (int i = 0; i < Q; i++) pm[i] = __ballot_sync(FULL, lb[i] <= tauf[i]);
          }
          unsigned open = pm[0];
#pragma unroll
          for (int i = 1; i < Q; i++) open |= pm[i];
          open &= todo;
          if (!open) break;
          const int c = __ffs(open) - 1;
          todo = ~1u << c;
          changed = scan_leaf(node * 32 + (c ^ flip), c, pm);
        }
      } else {
#pragma unroll
        for (int i = 0; i < Q; i++)
          if (lb[i] <= tauf[i]) cur = fminf(cur, lb[i]);
        // (the own leaf's branch is done)
        if (fresh && lane == (int)((own >> (5 * (level - 1))) & 31u)) cur = none;
      }
      // the next node: the nearest open child, or on with the parent
      fresh = false;
      for (;;) {
        if (level > 1) {
          float tmax = tauf[0];
#pragma unroll
          for (int i = 1; i < Q; i++) tmax = fmaxf(tmax, tauf[i]);
          const uint32_t key = cur <= tmax ? __float_as_uint(cur) : 0xffffffffu;
          const uint32_t b = __reduce_min_sync(FULL, key);
          if (b != 0xffffffffu) {
            const int c = __ffs(__ballot_sync(FULL, key == b)) - 1;
            if (lane == c) cur = none;
            stk[(level - 2) * 32 + lane] = cur;
            level--;
            node = node * 32 + c;
            break;
          }
        }
        if (level == top) {
          if (top == root) return;
          top++;
          level = top;
          node = top < root ? own >> (5 * top) : 0u;
          fresh = true;
          break;
        }
        level++;
        node >>= 5;
        cur = stk[(level - 2) * 32 + lane];
      }
    }
  }
};

// position of the set bit number k (from 0) of a word with more than k bits
__device__ __forceinline__ uint32_t nth_bit(unsigned w, uint32_t k) {
  for (; k > 0; k--) w &= w - 1;
  return __ffs(w) - 1;
}

template <typename T, int D, int Q>
__global__ void __launch_bounds__(TREE_THREADS, tree_min_blocks(D)) tree_kernel(const TreeParams<T> p) {
  using Kt = Key<T>;
  using KT = typename Kt::type;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  TreeTile<T, D, Q> t(p, lane);
  t.buf = reinterpret_cast<KT*>(smem) + (size_t)wib * Q * p.B;
  unsigned char* at = smem + (size_t)wpb * Q * p.B * sizeof(KT);
  t.ts = reinterpret_cast<TreeState<T, Q>*>(at) + wib;
  at += (size_t)wpb * sizeof(TreeState<T, Q>);
  t.hist = reinterpret_cast<uint32_t*>(at) + wib * 256;
  at += (size_t)wpb * 1024;
  t.stk = reinterpret_cast<float*>(at) + wib * TREE_STACK * 32;
  at += (size_t)wpb * TREE_STACK * 128;
  t.queue = nullptr;
  t.qsm = nullptr;
  t.qfm = nullptr;
  if (sizeof(T) == 8) {
    t.queue = reinterpret_cast<uint32_t*>(at) + wib * Q * TREE_QUEUE;
    at += (size_t)wpb * Q * TREE_QUEUE * 4;
    t.qsm = reinterpret_cast<T*>(at) + (size_t)wib * Q * p.d;
    at += (size_t)wpb * Q * p.d * sizeof(T);
  }
  if (D == 0) t.qfm = reinterpret_cast<float*>(at) + (size_t)wib * Q * p.d;
  __shared__ uint32_t s_ticket;
  if (threadIdx.x == 0) s_ticket = 0;
  __syncthreads();

  if (p.qmask && *p.nq_dev == 0) return;
  T rmax = 0;
  // Tile g of a leaf: its queries number g Q ... g Q + Q - 1.  A block takes
  // runs of consecutive tiles, so that its warps read the same part of the
  // tree at the same time; a small tree is spread over all blocks.
  constexpr uint32_t PER_LEAF = 32 / Q;
  const uint64_t tiles = (uint64_t)p.t.count[0] * PER_LEAF;
  const uint32_t run = (uint32_t)min((unsigned long long)TREE_CHUNK,
                                     max((unsigned long long)wpb, (unsigned long long)(tiles / (gridDim.x * 4))));
  for (;;) {
    uint32_t tk = 0;
    if (lane == 0) tk = atomicAdd(&s_ticket, 1u);
    tk = __shfl_sync(FULL, tk, 0);
    const uint64_t tile = ((uint64_t)(tk / run) * gridDim.x + blockIdx.x) * run + tk % run;
    if (tile >= tiles) {
      // (the block's later runs lie beyond as well, its current run's rest too)
      break;
    }
    const uint32_t own = (uint32_t)(tile / PER_LEAF), first = (uint32_t)(tile % PER_LEAF) * Q;
    const uint32_t in_leaf = (uint32_t)min(32ull, (unsigned long long)(p.n - (uint64_t)own * 32));
    const unsigned leaf_mask = p.qmask ? p.qmask[own] : (in_leaf < 32 ? (1u << in_leaf) - 1u : FULL);
    const uint32_t have = __popc(leaf_mask);
    if (first >= have) continue;
    // (one lane per query: the threshold of a double radius takes square roots)
    const uint32_t my_pos = own * 32 + nth_bit(leaf_mask, min(first + min(lane, Q - 1), have - 1));
    T thr = (T)INFINITY;
    if (!p.unbounded) {
      const T r0 = p.qradius ? p.qradius[p.t.id[my_pos]] : p.radius;
      thr = within_threshold(r0);
      rmax = r0 > rmax ? r0 : rmax;
    }
#pragma unroll
    for (int i = 0; i < Q; i++) {
      const uint32_t at_pos = __shfl_sync(FULL, my_pos, i);
      const uint64_t at0 = (uint64_t)own * 32 * (D > 0 ? (uint32_t)D : p.d) + (at_pos & 31u);
      if (D > 0) {
#pragma unroll
        for (int l = 0; l < (D > 0 ? D : 1); l++)
          t.q[i][l] = sizeof(T) == 8 ? p.t.psf[at0 + l * 32] : (float)p.t.ps[at0 + l * 32];
      }
      if (sizeof(T) == 8 || D == 0) {
        for (uint32_t l = lane; l < p.d; l += 32) {
          const T v = p.t.ps[at0 + l * 32];
          if (sizeof(T) == 8) t.qsm[i * p.d + l] = v;
          if (D == 0) t.qfm[l * Q + i] = (float)v;
        }
      }
      if (sizeof(T) == 8) {
        float s2 = 0.0f;
        if (D > 0) {
#pragma unroll
          for (int l = 0; l < (D > 0 ? D : 1); l++) s2 = __fmaf_ru(t.q[i][l], t.q[i][l], s2);
        } else {
          __syncwarp();
          for (uint32_t l = 0; l < p.d; l++) s2 = __fmaf_ru(t.qfm[l * Q + i], t.qfm[l * Q + i], s2);
        }
        t.qnorm[i] = __fmul_ru(__fsqrt_ru(s2), 1.000001f);
      }
    }
    if (lane < Q) {
      t.ts->tau[lane] = Kt::bound(thr);
      t.ts->len[lane] = 0;
      t.ts->qn[lane] = 0;
      t.ts->trig[lane] = p.unbounded ? min(p.B - 32, p.K - 1) : min(p.B - 32, p.K + max(p.K, 32u));
    }
#pragma unroll
    for (int i = 0; i < Q; i++) t.tauf[i] = first + i < have ? 0.0f : -1.0f;
    __syncwarp();
    t.load_state();
    t.search(own);
    t.settle(true);
#pragma unroll 1
    for (int i = 0; i < Q && first + i < have; i++) {
      KT* buf = t.buf + (size_t)i * p.B;
      const uint32_t len = t.ts->len[i];
      const KT tau = t.ts->tau[i];
      const uint32_t at_pos = own * 32 + nth_bit(leaf_mask, first + i);
      const uint32_t id = p.t.id[at_pos];
      if (len >= p.K) {
        const uint64_t row = (uint64_t)id * p.K;
        write_sorted_row<T>(buf, t.hist, len, tau, p.K, p.out_ids, p.out_d, row, lane, p.rowsum);
        if (p.unbounded) {
          const T a = Kt::acc(tau);
          rmax = a > rmax ? a : rmax;
        }
      } else if (lane == 0) {
        atomicAdd(p.fail_count, 1u);
        atomicOr(&p.fail_mask[own], 1u << (at_pos & 31u));
        // every point within the radius was found: their count gives the
        // local density, and the radius is scaled toward K points, with room
        // for the count's spread (without it and with 1.08 for 1.2 a fifth of
        // the queries failed again: 3M sky-like points 11.8 -> 11.0 ms, 1M x
        // 3-D 4.7 -> 4.5 ms)
        const float fl = (float)max(len, 1u);
        const float f = exp2f(log2f((float)p.K / fl * (1.0f + rsqrtf(fl))) * p.inv_di) * 1.2f;
        const T r0 = p.qradius ? p.qradius[id] : p.radius;
        const T g = (T)((double)r0 * (double)fmaxf(f, 1.2f));
        p.grow[id] = g;
        rmax = g > rmax ? g : rmax;
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int i = 1; i < Q; i++) {  // (the lanes that read the queries' radii)
    const T o = __shfl_sync(FULL, rmax, i);
    rmax = o > rmax ? o : rmax;
  }
  if (lane == 0) {
    if (t.scanned) atomicAdd(p.cand_count, 32ull * t.scanned);
    if (rmax > (T)0)
      atomicMax(p.rmax_bits, (unsigned long long)Num<T>::bits(p.unbounded ? Num<T>::sqrt(rmax) : rmax));
  }
}

// Dynamic shared memory of one warp: a selection buffer of B keys per query, the
// shared state, the reduction's bins, the walk's stack; double data also the
// queue and the queries, a runtime dimension count the queries in float.
template <typename T, int D, int Q>
constexpr size_t tree_warp_bytes(uint32_t B, uint32_t d) {
  return (size_t)Q * B * sizeof(typename Key<T>::type) + sizeof(TreeState<T, Q>) + 1024 + TREE_STACK * 128 +
         (sizeof(T) == 8 ? (size_t)Q * TREE_QUEUE * 4 + (size_t)Q * d * sizeof(T) : 0) +
         (D == 0 ? (size_t)Q * d * 4 : 0);
}
static_assert(tree_warp_bytes<double, 0, TREE_Q>(HIST_MAX_B, MAX_D) <= TREE_MAX_SMEM, "one warp fits a block");

template <typename T, int D, int Q>
void launch_tree_one(const TreeParams<T>& p, int sm_count, cudaStream_t s) {
  const size_t per_warp = tree_warp_bytes<T, D, Q>(p.B, p.d);
  int wpb = TREE_THREADS / 32;
  while (wpb > 1 && per_warp * wpb > TREE_MAX_SMEM) wpb--;
  const size_t smem = per_warp * wpb;
  auto kern = tree_kernel<T, D, Q>;
  allow_dynamic_smem(kern, TREE_MAX_SMEM);
  int per_sm = 0;
  KNNSJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, wpb * 32, smem));
  if (per_sm < 1) throw StatusError{KNNSJ_ERR_UNSUPPORTED, "tree search kernel does not fit"};
  const uint64_t tiles = (uint64_t)p.t.count[0] * (32 / Q);
  uint64_t blocks = (uint64_t)per_sm * sm_count;
  blocks = std::min<uint64_t>(blocks, std::max<uint64_t>((tiles + wpb - 1) / wpb, 1));
  kern<<<(unsigned)blocks, wpb * 32, smem, s>>>(p);
  KNNSJ_CHECK_LAUNCH();
}

template <typename T, int Q>
void launch_tree_d(const TreeParams<T>& p, int sm_count, cudaStream_t s) {
  switch (p.d) {
    case 2: launch_tree_one<T, 2, Q>(p, sm_count, s); break;
    case 3: launch_tree_one<T, 3, Q>(p, sm_count, s); break;
    case 4: launch_tree_one<T, 4, Q>(p, sm_count, s); break;
    case 5: launch_tree_one<T, 5, Q>(p, sm_count, s); break;
    case 6: launch_tree_one<T, 6, Q>(p, sm_count, s); break;
    case 7: launch_tree_one<T, 7, Q>(p, sm_count, s); break;
    case 8: launch_tree_one<T, 8, Q>(p, sm_count, s); break;
    default: launch_tree_one<T, 0, Q>(p, sm_count, s); break;
  }
}

}  // namespace

template <typename T>
void launch_tree_search(const TreeLaunch<T>& a, int sm_count, cudaStream_t s) {
  TreeParams<T> p{};
  p.t = a.tree;
  p.n = a.n;
  p.d = a.d;
  p.K = a.K;
  // selection buffer: room for K <= tree_max_k keys, what comes in between two
  // reductions and a full leaf
  p.B = a.K <= 48 ? 128u : HIST_MAX_B;
  p.qmask = a.qmask;
  p.nq_dev = a.nq_dev;
  p.radius = a.radius;
  p.qradius = a.qradius;
  p.unbounded = a.unbounded;
  p.inv_di = 1.0f / (float)a.indexed;
  p.out_ids = a.out_ids;
  p.out_d = a.out_d;
  p.rowsum = a.rowsum;
  p.fail_mask = a.fail_mask;
  p.fail_count = a.fail_count;
  p.grow = a.grow;
  p.rmax_bits = a.rmax_bits;
  p.cand_count = a.cand_count;
  launch_tree_d<T, TREE_Q>(p, sm_count, s);
}

}  // namespace knnsj
