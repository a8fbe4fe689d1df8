// k_tile.cu -- range search of low-dimensional float data by tiles of
// queries: one warp owns QPT queries (4 by default) that are neighbours along
// a space-filling curve of their cells (Hilbert in two dimensions, Morton in
// three), 32 / QPT lanes per query, and the tile's queries share one pass over the candidates of the union of their rings.
//
// Replaces, for the first search pass of float data with two or three
// dimensions (all indexed) and k+1 <= 65, the same reference steps as
// search_kernel (k_search.cu): kernelNDGridIndexGlobalkNN with evaluateCell
// and evalPoint (kernel.cu:61-225), the pair buffer and the two
// thrust::stable_sort_by_key (GPU.cu:1629-1634), and the K-row extraction of
// storeNeighborTableForkNNOnTheFly (GPU.cu:3610-3704).
//
// Per tile (one warp):
//   1. each query's cell ring, the union box of the tile's rings (a query
//      whose ring is much wider than the tile's mean is handed to
//      search_kernel instead, so one outlier does not widen everyone's
//      scan); each row of the box (consecutive cells along dimension 0) is
//      one contiguous run of the cell-ordered columns;
//   2. the box's candidates are staged in shared memory 64 at a time
//      (coalesced loads: coordinates and id in one 16-byte record, the next
//      chunk in flight while the current one is evaluated); lane (slot q,
//      phase p) evaluates candidates p, p + 32 / QPT, ... for query q;
//   3. the single pass over the candidates: every key (squared distance,
//      id) within the query's radius goes to the query's list in shared
//      memory, its slot from a ballot over the query's lanes (no atomics);
//      a query that finds more keys than the list holds (0.04 % of the sky
//      join) is handed to search_kernel, one that finds fewer than K fails
//      (the reference's acceptance rule, GPU.cu:3659-3669);
//   4. each accepted query's list is sorted by the whole warp as 32-bit words
//      (25 bits of squared distance over its list index), 4 per lane, in
//      registers; words of equal distance bits are put in order of their full
//      keys by passes over neighbours (few queries have any; one that needs
//      more than SORT_FIXES passes is handed to search_kernel);
//   5. the warp writes the row with coalesced stores (distances as sqrt in the
//      data type).
// Squared distances use the reference's fma chain in dimension order
// (kernel.cu:139-140) exactly as search_kernel does, so rows are identical.
// Keys are (squared distance bits, id) in one u64: ties are ordered by id.

#include <cmath>
#include <cstdlib>

#include "knnsj_internal.h"

namespace knnsj {

namespace {

constexpr int TILE_WARPS = 4;                    // warps per block
constexpr int TILE_THREADS = TILE_WARPS * 32;
constexpr int TILE_CH = 64;                      // staged candidates per chunk
constexpr int SORT_FIXES = 24;                   // passes over neighbours of equal distance bits
constexpr uint32_t TILE_MAX_ROWS = 4096;         // larger union boxes go to search_kernel

struct alignas(16) Cand {
  float x[3];
  uint32_t id;
};

// Capacity of a query's key list: more than twice k+1 (the learned radius
// finds 1.4 (k+1) keys on average; the few queries that find more are
// handed to search_kernel), the most that 8 blocks of 4 warps of 4 queries
// leave room for, the pitch in u64 words = 4 (mod 16) so that the lists of a
// warp's queries spread over the banks.
constexpr int tile_list_cap(int kmax) { return kmax >= 65 ? 164 : kmax >= 33 ? 84 : 52; }

// shared memory of one warp (bytes): QPT queries with rows of up to KMAX
// keys.  The staging chunk and the row's list indices share one region (used
// one after the other).
template <int QPT, int KMAX>
struct TileSmem {
  static constexpr int C = tile_list_cap(KMAX);                 // list capacity per query (u64 keys)
  static constexpr int R = C <= 64 ? 2 : 4;                     // words per lane of a sorted list
  static constexpr int LIST = 0;                                // [QPT][C] u64
  static constexpr int CAND = LIST + QPT * C * 8;               // staging chunk | list indices
  static constexpr int RUNS = CAND + TILE_CH * 16;              // 2 x 32 u32
  static constexpr int BYTES = RUNS + 2 * 32 * 4;
};

struct TileParams {
  GridGeom<float> g;                    // candidate grid
  const float* __restrict__ ps;         // candidate columns in cell order (d x n)
  const uint32_t* __restrict__ pid;     // original id of each cell-ordered position
  const uint32_t* __restrict__ dstart;  // first position of every linear cell id (dense table)
  uint64_t n;
  uint32_t K;
  const float* __restrict__ qps;        // query columns: cell order (qlist null) or input order
  const uint32_t* __restrict__ qpid;    // ids of qps positions (qlist null)
  const uint32_t* __restrict__ qlist;   // query ids, or null: the positions of qps
  uint32_t nq;
  float radius;                         // uniform radius (qradius null)
  float* qradius;                       // per-query radius by id
  double step;                          // least growth of a failed per-query radius
  int32_t* out_ids;
  float* out_d;
  double* rowsum;                       // per-row verification sums (null: none)
  uint32_t* fail_list;
  uint32_t* fail_count;
  uint32_t* defer_list;                 // queries handed to search_kernel at the same radius
  uint32_t* defer_count;
  unsigned long long* cand_count;
  uint32_t* work_counter;
  FailRadii* fail_radii;
};

// Ascending bitonic sort of 32 R words across a warp; word i is v[i % R] of
// lane i / R, so that the strides below R stay within a lane.
template <int R>
__device__ __forceinline__ void warp_sort_words(uint32_t (&v)[R], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= R) {
        const bool keep_min = ((lane * R & k) == 0) == ((lane & (j / R)) == 0);
#pragma unroll
        for (int r = 0; r < R; r++) {
          const uint32_t o = __shfl_xor_sync(FULL, v[r], j / R);
          v[r] = keep_min ? min(v[r], o) : max(v[r], o);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (r & j) continue;
          const bool up = k < R ? (r & k) == 0 : (lane * R & k) == 0;
          const uint32_t lo = min(v[r], v[r | j]), hi = max(v[r], v[r | j]);
          v[r] = up ? lo : hi;
          v[r | j] = up ? hi : lo;
        }
      }
    }
  }
}

// Warp-aggregated append of this lane's value to a global list.
__device__ __forceinline__ void warp_append(bool want, uint32_t v, uint32_t* list, uint32_t* count, int lane) {
  const unsigned m = __ballot_sync(FULL, want);
  if (!m) return;
  const int leader = __ffs(m) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(m));
  base = __shfl_sync(FULL, base, leader);
  if (want) list[base + __popc(m & lanemask_lt())] = v;
}

// QPT queries per warp (4, 8 or 16), LPQ = 32 / QPT lanes per query: lane
// (slot qs = lane % QPT, phase ph = lane / QPT) evaluates the staged
// candidates ph, ph + LPQ, ... for query qs.  The query's lanes share its
// list in shared memory; the lane of phase 0 does the query's serial steps.  With 4 queries per warp the
// kernel is held to 64 registers: 8 blocks of 4 warps fit an SM.
template <int D, int KMAX, int QPT>
__global__ void __launch_bounds__(TILE_THREADS, QPT == 4 ? 8 : 5) tile_kernel(const TileParams p) {
  using SM = TileSmem<QPT, KMAX>;
  constexpr int LPQ = 32 / QPT;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int qs = lane % QPT;
  const int ph = lane / QPT;
  const bool lead = ph == 0;
  unsigned char* ws = smem + (size_t)wib * SM::BYTES;
  Cand* cand = reinterpret_cast<Cand*>(ws + SM::CAND);
  unsigned long long* lists = reinterpret_cast<unsigned long long*>(ws + SM::LIST);  // [QPT][C]
  unsigned long long* mylist = lists + (size_t)qs * SM::C;  // this query's keys, later its row
  uint32_t* runS = reinterpret_cast<uint32_t*>(ws + SM::RUNS);
  uint32_t* runP = runS + 32;
  // this query's lanes, and those of them below this lane
  unsigned qmask = 0;
#pragma unroll
  for (int pp = 0; pp < LPQ; pp++) qmask |= 1u << (qs + QPT * pp);
  const unsigned qbelow = qmask & lanemask_lt();

  __shared__ float s_minf[3];
  __shared__ float s_invw;
  if (threadIdx.x < 3) s_minf[threadIdx.x] = threadIdx.x < (unsigned)D ? (float)p.g.minv[threadIdx.x] : 0.0f;
  if (threadIdx.x == 0) s_invw = 1.0f / (float)p.g.width;
  __syncthreads();

  const uint64_t n = p.n;
  const uint32_t K = p.K;
  const uint32_t ntiles = (p.nq + QPT - 1) / QPT;
  unsigned long long scanned = 0;

  for (;;) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(p.work_counter, 1u);
    t = __shfl_sync(FULL, t, 0);
    if (t >= ntiles) break;
    const uint32_t qi = t * (uint32_t)QPT + (uint32_t)qs;
    const bool valid = qi < p.nq;
    uint32_t qid = 0;
    float q[D];
    float r = 0.0f;
#pragma unroll
    for (int j = 0; j < D; j++) q[j] = 0.0f;
    if (valid) {
      qid = p.qlist ? p.qlist[qi] : p.qpid[qi];
      const uint64_t col = p.qlist ? (uint64_t)qid : (uint64_t)qi;
#pragma unroll
      for (int j = 0; j < D; j++) q[j] = p.qps[(uint64_t)j * n + col];
      r = p.qradius ? p.qradius[qid] : p.radius;
    }

    // 1. the query's ring (as search_kernel computes it) and the union box
    const float rf = r * (1.0f + 1.0f / 8192.0f);
    uint32_t lo[D], hi[D];
    uint32_t ext = 0;
#pragma unroll
    for (int j = 0; j < D; j++) {
      const float slack = (fabsf(q[j]) + rf) * (1.0f / 2097152.0f);
      lo[j] = ring_cell(q[j] - rf - slack, s_minf[j], s_invw, p.g.ncell[j], false);
      hi[j] = ring_cell(q[j] + rf + slack, s_minf[j], s_invw, p.g.ncell[j], true);
      ext = max(ext, hi[j] - lo[j] + 1);
    }
    // queries whose ring is far wider than the tile's mean go to search_kernel
    // (one outlier would widen every query's scan)
    bool defer = false;
    {
      const uint32_t nv = __popc(__ballot_sync(FULL, valid));  // (each query counted LPQ times)
      const uint32_t sum = __reduce_add_sync(FULL, valid ? ext : 0u);
      const uint32_t mean = (sum + nv - 1) / nv;
      defer = valid && ext > 2u * mean + 2u;
    }
    bool in = valid && !defer;  // queries searched by this tile
    uint32_t LO[D], HI[D];
#pragma unroll
    for (int j = 0; j < D; j++) {
      LO[j] = __reduce_min_sync(FULL, in ? lo[j] : 0xffffffffu);
      HI[j] = __reduce_max_sync(FULL, in ? hi[j] : 0u);
    }
    uint32_t ext1 = HI[1] - LO[1] + 1;
    uint32_t ext2 = D == 3 ? HI[D - 1] - LO[D - 1] + 1 : 1u;
    uint64_t nrows64 = __ballot_sync(FULL, in) ? (uint64_t)ext1 * ext2 : 0;
    if (nrows64 > TILE_MAX_ROWS) {  // (uniform) the whole tile goes to search_kernel
      defer = valid;
      in = false;
      nrows64 = 0;
    }
    uint32_t nrows = (uint32_t)nrows64;
    warp_append(defer && lead, qid, p.defer_list, p.defer_count, lane);

    const float thr = in ? within_threshold(r) : -1.0f;  // acc <= thr never holds off the tile

    // Visits every candidate of the union box; body(c, live) runs on every
    // lane, live when c is a candidate of this lane's phase.
    auto for_each_candidate = [&](auto&& body) -> uint32_t {
      uint32_t visited = 0;
      for (uint32_t g0 = 0; g0 < nrows; g0 += 32) {
        const uint32_t ridx = g0 + (uint32_t)lane;
        uint32_t rs = 0, len = 0;
        if (ridx < nrows) {
          unsigned long long rbase;
          if constexpr (D == 2) {
            rbase = (unsigned long long)(LO[1] + ridx) * p.g.mult[1];
          } else {
            const uint32_t a1 = ridx % ext1, a2 = ridx / ext1;
            rbase = (unsigned long long)(LO[1] + a1) * p.g.mult[1] + (unsigned long long)(LO[D - 1] + a2) * p.g.mult[D - 1];
          }
          rs = p.dstart[rbase + LO[0]];
          len = p.dstart[rbase + HI[0] + 1] - rs;
        }
        uint32_t incl = len;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t tt = __shfl_up_sync(FULL, incl, off);
          if (lane >= off) incl += tt;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        visited += total;
        __syncwarp();
        runS[lane] = rs;
        runP[lane] = incl - len;
        __syncwarp();
        // chunks are loaded one ahead: the loads of chunk c + 1 are in flight
        // while chunk c is evaluated
        int row = 0;
        Cand pre[TILE_CH / 32];
        auto fetch = [&](uint32_t c0) {
#pragma unroll
          for (int m = 0; m < TILE_CH / 32; m++) {
            const uint32_t v = c0 + (uint32_t)(m * 32 + lane);
            if (v < total) {
              while (row < 31 && runP[row + 1] <= v) row++;
              const uint32_t pos = runS[row] + (v - runP[row]);
#pragma unroll
              for (int j = 0; j < 3; j++) pre[m].x[j] = j < D ? p.ps[(uint64_t)j * n + pos] : 0.0f;
              pre[m].id = p.pid[pos];
            }
          }
        };
        if (total) fetch(0);
        for (uint32_t c0 = 0; c0 < total; c0 += TILE_CH) {
          const uint32_t cnt = min((uint32_t)TILE_CH, total - c0);
          __syncwarp();
#pragma unroll
          for (int m = 0; m < TILE_CH / 32; m++)
            if (c0 + (uint32_t)(m * 32 + lane) < total) cand[m * 32 + lane] = pre[m];
          __syncwarp();
          if (c0 + TILE_CH < total) fetch(c0 + TILE_CH);
          const uint32_t steps = (cnt + LPQ - 1) / LPQ;
          uint32_t st = 0;
          for (; st + 4 <= steps; st += 4) {
            Cand c4[4];
            bool l4[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const uint32_t j = (st + u) * LPQ + ph;
              l4[u] = j < cnt;
              c4[u] = cand[l4[u] ? j : 0];
            }
#pragma unroll
            for (int u = 0; u < 4; u++) body(c4[u], l4[u]);
          }
          for (; st < steps; st++) {
            const uint32_t j = st * LPQ + ph;
            const bool live = j < cnt;
            const Cand cc = cand[live ? j : 0];
            body(cc, live);
          }
        }
        __syncwarp();
      }
      return visited;
    };
    auto sqdist = [&](const Cand& c) -> float {
      float acc = 0.0f;
#pragma unroll
      for (int j = 0; j < D; j++) {
        const float tt = __fsub_rn(c.x[j], q[j]);
        acc = __fmaf_rn(tt, tt, acc);
      }
      return acc;
    };

    // 3. pass 1: every key within the radius is appended to the query's
    // list (slots from a ballot over the query's lanes: no atomics); the
    // count goes on past the capacity, so `found` is exact
    uint32_t found = 0;
    const uint32_t box_points = for_each_candidate([&](const Cand& c, bool live) {
      const float acc = sqdist(c);
      const bool want = live && acc <= thr;
      const unsigned bal = __ballot_sync(FULL, want);
      const uint32_t slot = found + (uint32_t)__popc(bal & qbelow);
      if (want && slot < (uint32_t)SM::C)
        mylist[slot] = ((unsigned long long)__float_as_uint(acc) << 32) | c.id;
      found += (uint32_t)__popc(bal & qmask);
    });
    // candidates evaluated: the union box's points for every query it serves
    scanned += (unsigned long long)box_points * (unsigned)__popc(__ballot_sync(FULL, in && lead));
    // a query with more keys than its list holds goes to search_kernel
    const bool big = in && found > (uint32_t)SM::C;
    warp_append(big && lead, qid, p.defer_list, p.defer_count, lane);
    const bool ok = in && found >= K && !big;
    __syncwarp();

    // 4., 5. the accepted queries one after the other, by the whole warp
    unsigned accepted = __ballot_sync(FULL, ok && lead);
    while (accepted) {
      const int rl = __ffs(accepted) - 1;  // (a lead lane: its index is the query slot)
      accepted &= accepted - 1;
      const uint32_t rid = __shfl_sync(FULL, qid, rl);
      const uint32_t nl = __shfl_sync(FULL, found, rl);
      const float top = __shfl_sync(FULL, thr, rl);
      const unsigned long long* list = lists + (size_t)rl * SM::C;
      uint32_t* words = reinterpret_cast<uint32_t*>(ws + SM::CAND);
      constexpr int R = SM::R;
      constexpr uint32_t NE = 32 * R, NONE = 0xffffffffu;
      // word of a list entry: floor(acc * 2^25 / top), monotone in acc, over
      // the entry's index
      const float s25 = top > 0.0f && top < 3.0e38f ? __fdividef(33554400.0f, top) : 0.0f;
      auto dist_bits = [&](uint32_t e) -> uint32_t {
        const float acc = __uint_as_float((uint32_t)(list[e] >> 32));
        return min(__float2uint_rz(acc * s25), 33554430u);
      };
      uint32_t v[R];
      if (SM::C <= NE || nl <= NE) {
#pragma unroll
        for (int r = 0; r < R; r++) {
          const uint32_t e = r * 32 + lane;
          v[r] = e < nl ? dist_bits(e) << 7 | e : NONE;
        }
      } else {
        // more keys than words (1 % of the sky join): those up to a distance
        // that should leave between K and NE of them, their list indices
        // closed up in shared memory
        const uint32_t cut = (uint32_t)(33554432.0f * (0.5f * (float)(K + NE)) / (float)nl);
        uint32_t kept = 0;
        uint8_t* ix = reinterpret_cast<uint8_t*>(words) + NE;
        for (uint32_t e0 = 0; e0 < nl; e0 += 32) {
          const uint32_t e = e0 + lane;
          const bool keep = e < nl && dist_bits(e) < cut;
          const unsigned m = __ballot_sync(FULL, keep);
          const uint32_t at = kept + __popc(m & lanemask_lt());
          if (keep && at < NE) ix[at] = (uint8_t)e;
          kept += __popc(m);
        }
        __syncwarp();
        if (kept < K || kept > NE) {
          if (lane == 0) p.defer_list[atomicAdd(p.defer_count, 1u)] = rid;
          continue;
        }
        // (the words carry positions of the closed-up list)
#pragma unroll
        for (int r = 0; r < R; r++) {
          const uint32_t e = r * 32 + lane;
          v[r] = e < kept ? dist_bits(ix[e]) << 7 | e : NONE;
        }
      }
      const bool closed = SM::C > NE && nl > NE;
      const uint8_t* ix = reinterpret_cast<const uint8_t*>(words) + NE;
      auto key_of = [&](uint32_t w) -> unsigned long long { return list[closed ? ix[w & 127u] : w & 127u]; };
      warp_sort_words<R>(v, lane);
      // neighbours of equal distance bits, in the order of their full keys
      auto tied = [&](uint32_t a, uint32_t b) { return (a >> 7) == (b >> 7) && b != NONE; };
      bool any = false;
#pragma unroll
      for (int r = 0; r + 1 < R; r++) any |= tied(v[r], v[r + 1]);
      {
        const uint32_t nx = __shfl_down_sync(FULL, v[0], 1);
        any |= lane < 31 && tied(v[R - 1], nx);
      }
      if (__any_sync(FULL, any)) {
        int left = SORT_FIXES;
        for (; left > 0; left--) {
          bool moved = false;
          auto order = [&](uint32_t& a, uint32_t& b) {
            if (tied(a, b) && key_of(b) < key_of(a)) {
              const uint32_t t2 = a;
              a = b;
              b = t2;
              moved = true;
            }
          };
#pragma unroll
          for (int r = 0; r + 1 < R; r += 2) order(v[r], v[r + 1]);
#pragma unroll
          for (int r = 1; r + 1 < R; r += 2) order(v[r], v[r + 1]);
          // (both lanes of a pair take the same decision)
          const uint32_t nx = __shfl_down_sync(FULL, v[0], 1), pv = __shfl_up_sync(FULL, v[R - 1], 1);
          const bool give = lane < 31 && tied(v[R - 1], nx) && key_of(nx) < key_of(v[R - 1]);
          const bool take = lane > 0 && tied(pv, v[0]) && key_of(v[0]) < key_of(pv);
          if (give) v[R - 1] = nx;
          if (take) v[0] = pv;
          if (!__any_sync(FULL, moved || give || take)) break;
        }
        if (left == 0) {  // too many equal distances
          if (lane == 0) p.defer_list[atomicAdd(p.defer_count, 1u)] = rid;
          continue;
        }
      }
      // list indices by row slot, four bytes to a word
      uint32_t pack = 0;
#pragma unroll
      for (int r = 0; r < R; r++) pack |= (v[r] & 127u) << (8 * r);
      uint8_t* slots = reinterpret_cast<uint8_t*>(words);
      if (R == 4)
        words[lane] = pack;
      else
        reinterpret_cast<uint16_t*>(words)[lane] = (uint16_t)pack;
      __syncwarp();
      const uint64_t base = (uint64_t)rid * K;
      float rsq = 0.0f;
      for (uint32_t s = (uint32_t)lane; s < K; s += 32) {
        const unsigned long long key = key_of(slots[s]);
        const float dist = __fsqrt_rn(__uint_as_float((uint32_t)(key >> 32)));
        p.out_ids[base + s] = (int32_t)(uint32_t)key;
        p.out_d[base + s] = dist;
        rsq = __fadd_rn(rsq, __fmul_rn(dist, dist));
      }
      if (p.rowsum) store_row_sum<float>(p.rowsum, rid, rsq, lane);
      __syncwarp();
    }
    // failures: fewer than K points within the radius
    const bool fail = in && found < K;
    warp_append(fail && lead, qid, p.fail_list, p.fail_count, lane);
    if (fail && lead && p.qradius) {
      // per-query radii grow by at least eps0/2, toward K points from the
      // count found within the radius: (K / found)^(1/dims), at most 4x
      double rn = (double)r + p.step;
      const float f = exp2f(log2f((float)K / (float)max(found, 1u)) / (float)D) * 1.05f;
      rn = fmax(rn, (double)r * (double)fminf(fmaxf(f, 1.0f), 4.0f));
      const float rt = (float)rn;
      p.qradius[qid] = rt;
      atomicMax(&p.fail_radii->rmax_bits, (unsigned long long)__float_as_uint(rt));
      const float oct = log2f(rt / (2.0f * (float)p.step));  // log2(r / eps0)
      const int bin = min(max((int)floorf(4.0f * oct) + 16, 0), FAIL_RADIUS_BINS - 1);
      atomicAdd(&p.fail_radii->hist[bin], 1u);
    }
    __syncwarp();
  }
  if (lane == 0 && scanned) atomicAdd(p.cand_count, scanned);
}

template <int D, int KMAX, int QPT>
void launch_tile_kernel(const TileParams& prm, int sm_count, cudaStream_t s) {
  using SM = TileSmem<QPT, KMAX>;
  const size_t smem = (size_t)SM::BYTES * TILE_WARPS;
  auto kern = tile_kernel<D, KMAX, QPT>;
  KNNSJ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  KNNSJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TILE_THREADS, smem));
  if (per_sm < 1) throw StatusError{KNNSJ_ERR_UNSUPPORTED, "tile kernel does not fit"};
  const uint64_t tiles = ((uint64_t)prm.nq + QPT - 1) / QPT;
  uint64_t blocks = (uint64_t)per_sm * sm_count;
  const uint64_t need = (tiles + TILE_WARPS - 1) / TILE_WARPS;
  if (need < blocks) blocks = need;
  if (blocks < 1) blocks = 1;
  kern<<<(unsigned)blocks, TILE_THREADS, smem, s>>>(prm);
  KNNSJ_CHECK_LAUNCH();
}

}  // namespace

bool tile_search_applies(uint32_t d, uint32_t di, uint32_t K, int dense, size_t elem) {
  return elem == 4 && (d == 2 || d == 3) && di == d && K <= 65 && dense;
}

template <typename T>
void launch_tile_search(const SearchLaunch<T>& a, uint32_t* defer_list, uint32_t* defer_count, int sm_count,
                        cudaStream_t s) {
  if constexpr (sizeof(T) != 4) {
    throw StatusError{KNNSJ_ERR_UNSUPPORTED, "tile search is float only"};
  } else {
    if (a.nq == 0) return;
    TileParams p{};
    p.g = a.grid.geom;
    p.ps = a.grid.ps;
    p.pid = a.grid.pid;
    p.dstart = a.grid.dstart;
    p.n = a.n;
    p.K = a.K;
    p.qlist = a.qlist;
    p.qps = a.qlist ? a.xs : (a.qps ? a.qps : a.grid.ps);
    p.qpid = a.qps ? a.qpid : a.grid.pid;
    p.nq = a.nq;
    p.radius = a.radius;
    p.qradius = a.qradius;
    p.step = (double)a.step;
    p.out_ids = a.out_ids;
    p.out_d = a.out_d;
    p.rowsum = a.rowsum;
    p.fail_list = a.fail_list;
    p.fail_count = a.fail_count;
    p.defer_list = defer_list;
    p.defer_count = defer_count;
    p.cand_count = a.cand_count;
    p.work_counter = a.work_counter;
    p.fail_radii = a.fail_radii;
    launch_zero_words(a.work_counter, sizeof(uint32_t), s);
    const bool d3 = a.d == 3;
    // queries per tile: 8 share a box best (fewest candidates per query),
    // but their lists need twice the shared memory of 4; with 4 (64
    // registers, 8 blocks of 4 warps per SM) the kernel keeps 32 warps per
    // SM against 20, and the tile kernel is bound by latency: 4 is faster
    int qpt = 4;
    if (const char* e = std::getenv("KNNSJ_TILE_QPT")) qpt = std::atoi(e);
#define KNNSJ_TILE_LAUNCH(QPT)                                                                 \
  do {                                                                                        \
    if (a.K <= 16)                                                                            \
      d3 ? launch_tile_kernel<3, 16, QPT>(p, sm_count, s) : launch_tile_kernel<2, 16, QPT>(p, sm_count, s); \
    else if (a.K <= 33)                                                                       \
      d3 ? launch_tile_kernel<3, 33, QPT>(p, sm_count, s) : launch_tile_kernel<2, 33, QPT>(p, sm_count, s); \
    else                                                                                      \
      d3 ? launch_tile_kernel<3, 65, QPT>(p, sm_count, s) : launch_tile_kernel<2, 65, QPT>(p, sm_count, s); \
  } while (0)
    if (qpt == 16)
      KNNSJ_TILE_LAUNCH(16);
    else if (qpt == 4)
      KNNSJ_TILE_LAUNCH(4);
    else
      KNNSJ_TILE_LAUNCH(8);
#undef KNNSJ_TILE_LAUNCH
  }
}

template void launch_tile_search<float>(const SearchLaunch<float>&, uint32_t*, uint32_t*, int, cudaStream_t);
template void launch_tile_search<double>(const SearchLaunch<double>&, uint32_t*, uint32_t*, int, cudaStream_t);

}  // namespace knnsj
