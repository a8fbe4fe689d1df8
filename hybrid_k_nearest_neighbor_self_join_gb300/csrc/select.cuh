// select.cuh -- the k+1 nearest of a stream of candidates, kept by one warp in
// a shared-memory buffer of keys (squared distance, id): a reduction that
// keeps the buffer's K best when it fills, and the sorted row's write.
// Shared by the ring search (k_search.cu) and the box-tree search
// (tree_search.cuh).
#pragma once

#include "knnsj_device.cuh"

namespace knnsj {

namespace {

constexpr uint32_t HIST_MAX_B = 256;  // histogram reduce for buffers up to this size

__device__ __forceinline__ unsigned long long shfl_key(unsigned long long v, int src) {
  return __shfl_sync(FULL, v, src);
}
__device__ __forceinline__ KeyF64 shfl_key(KeyF64 v, int src) {
  KeyF64 r;
  r.a = __shfl_sync(FULL, v.a, src);
  r.id = __shfl_sync(FULL, v.id, src);
  r.pad = 0;
  return r;
}
__device__ __forceinline__ unsigned long long key_min() { return 0ull; }
__device__ __forceinline__ KeyF64 key_min_f64() {
  KeyF64 k;
  k.a = 0;
  k.id = 0;
  k.pad = 0;
  return k;
}

__device__ __forceinline__ float to_float_up(float x) { return x; }
__device__ __forceinline__ float to_float_up(double x) { return __double2float_ru(x); }

template <typename T>
struct Sel {
  using K = Key<T>;
  using KT = typename K::type;
  uint32_t len;
  KT tau;     // pass iff key < tau
  bool tight; // tau came from a reduce (an upper bound of the K-th best)
};

template <typename T>
__device__ __forceinline__ void sort_reduce(typename Key<T>::type* buf, Sel<T>& st, uint32_t K, uint32_t B,
                                            int lane) {
  __syncwarp();
  for (uint32_t i = st.len + lane; i < B; i += 32) buf[i] = Key<T>::maxv();
  __syncwarp();
  warp_bitonic_sort<T>(buf, (int)B, lane);
  st.len = K;
  st.tau = buf[K - 1];
  st.tight = true;
  __syncwarp();
}

// Monotone bin of a squared distance, round(a * scale) clamped to top, on
// the FMA pipe (a float-to-int conversion runs on a narrower pipe): with
// 1.5 * 2^23 added, the integer lands in the low mantissa bits.  Both users
// only need a monotone map that sends the largest kept key to a bin <= top.
__device__ __forceinline__ int acc_bin(float a, float scale, int top) {
  return min(__float_as_int(__fmaf_rn(a, scale, 12582912.0f)) - 0x4b400000, top);
}
// scale that maps [0, tacc] onto [0, nb] (0 when tacc is 0 or huge)
__device__ __forceinline__ float bin_scale(float nb, float tacc) {
  return (tacc > 0.0f && tacc < 3.0e38f) ? __fdividef(nb, tacc) : 0.0f;
}

// Keeps the keys of the lowest histogram bins that hold at least K keys
// (bins split [0, acc(tau)] evenly); the new threshold is the largest kept
// key.  Needs st.len >= K and B <= HIST_MAX_B.
template <typename T>
__device__ void hist_reduce(typename Key<T>::type* buf, uint32_t* hist, Sel<T>& st, uint32_t K, uint32_t B,
                            int lane) {
  using Kt = Key<T>;
  using KT = typename Kt::type;
  // bins by a monotone float map of the distance: equal distances share a bin
  const float tacc = to_float_up(Kt::acc(st.tau));
  const float scale = bin_scale(32.0f, tacc);
  __syncwarp();
  hist[lane] = 0;
  __syncwarp();
  for (uint32_t i = lane; i < st.len; i += 32) {
    const int b = acc_bin((float)Kt::acc(buf[i]), scale, 31);
    atomicAdd(&hist[b], 1u);
  }
  __syncwarp();
  uint32_t cum = hist[lane];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, cum, off);
    if (lane >= off) cum += t;
  }
  const int bst = __ffs(__ballot_sync(FULL, cum >= K)) - 1;
  const uint32_t kept = __shfl_sync(FULL, cum, bst);
  if (kept + 32 > B) {  // one bin holds too much: exact reduce
    sort_reduce<T>(buf, st, K, B, lane);
    return;
  }
  // in-place compaction: a round writes only below the end of what has been
  // read, so reading the round before writing it is enough
  uint32_t nl = 0;
  KT mx;
  if constexpr (sizeof(KT) == 8)
    mx = key_min();
  else
    mx = key_min_f64();
  for (uint32_t base = 0; base < st.len; base += 32) {
    const uint32_t i = base + lane;
    KT v = Kt::maxv();
    if (i < st.len) v = buf[i];
    const bool keep = i < st.len && acc_bin((float)Kt::acc(v), scale, 31) <= bst;
    const unsigned m = __ballot_sync(FULL, keep);
    __syncwarp();
    if (keep) {
      buf[nl + __popc(m & lanemask_lt())] = v;
      if (Kt::less(mx, v)) mx = v;
    }
    nl += __popc(m);
    __syncwarp();
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const KT o = shfl_key(mx, lane ^ off);
    if (Kt::less(mx, o)) mx = o;
  }
  st.len = nl;
  st.tau = mx;
  st.tight = true;
  __syncwarp();
}

// Rare paths are kept out of line so the hot loop stays small in the
// instruction cache.
#ifndef KNNSJ_REDUCE_CALLED
#define KNNSJ_REDUCE_CALLED 1
#endif
#if KNNSJ_REDUCE_CALLED
#define KNNSJ_REDUCE_LINKAGE __noinline__
#else
#define KNNSJ_REDUCE_LINKAGE __forceinline__
#endif
template <typename T>
__device__ KNNSJ_REDUCE_LINKAGE Sel<T> reduce(typename Key<T>::type* buf, uint32_t* hist, Sel<T> st, uint32_t K, uint32_t B,
                                      int lane) {
  if (B <= HIST_MAX_B)
    hist_reduce<T>(buf, hist, st, K, B, lane);
  else
    sort_reduce<T>(buf, st, K, B, lane);
  return st;
}

// the output sort is inlined (0: measured faster) or a called function (1)
#ifndef KNNSJ_WRITE_CALLED
#define KNNSJ_WRITE_CALLED 0
#endif
#if KNNSJ_WRITE_CALLED
#define KNNSJ_WRITE_LINKAGE __noinline__
#else
#define KNNSJ_WRITE_LINKAGE __forceinline__
#endif

// Writes the K smallest of buf[0..len) in ascending (distance, id) order by a
// counting sort over 256 bins of a monotone map of the distance (all keys are
// <= acc(top)), ranking keys that share a bin among themselves.  len <= 256.
template <typename T>
__device__ KNNSJ_WRITE_LINKAGE void write_sorted_row(typename Key<T>::type* buf, uint32_t* cnt, uint32_t len,
                                              typename Key<T>::type top, uint32_t K, int32_t* __restrict__ out_ids,
                                              T* __restrict__ out_d, uint64_t row_out, int lane,
                                              double* __restrict__ rowsum) {
  using Kt = Key<T>;
  using KT = typename Kt::type;
  constexpr int R = HIST_MAX_B / 32;
  const float tacc = to_float_up(Kt::acc(top));
  const float scale = bin_scale(256.0f, tacc);
  __syncwarp();
  reinterpret_cast<uint4*>(cnt)[lane] = make_uint4(0u, 0u, 0u, 0u);
  reinterpret_cast<uint4*>(cnt)[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
  KT v[R];
  uint32_t slot[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const uint32_t i = r * 32 + lane;
    v[r] = Kt::maxv();
    slot[r] = 0;
    if (r * 32 < (int)len && i < len) {
      v[r] = buf[i];
      const int b = acc_bin((float)Kt::acc(v[r]), scale, 255);
      slot[r] = atomicAdd(&cnt[b], 1u);
    }
  }
  __syncwarp();
  // exclusive scan of the 256 bin counts, 8 consecutive bins per lane
  uint32_t c[8], s = 0;
  {
    const uint4 c0 = reinterpret_cast<const uint4*>(cnt)[lane * 2];
    const uint4 c1 = reinterpret_cast<const uint4*>(cnt)[lane * 2 + 1];
    c[0] = c0.x, c[1] = c0.y, c[2] = c0.z, c[3] = c0.w;
    c[4] = c1.x, c[5] = c1.y, c[6] = c1.z, c[7] = c1.w;
  }
#pragma unroll
  for (int t = 0; t < 8; t++) s += c[t];
  uint32_t incl = s;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, incl, off);
    if (lane >= off) incl += t;
  }
  uint32_t run = incl - s;
  __syncwarp();
  {
    uint32_t o[8];
#pragma unroll
    for (int t = 0; t < 8; t++) {
      o[t] = run;
      run += c[t];
    }
    reinterpret_cast<uint4*>(cnt)[lane * 2] = make_uint4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<uint4*>(cnt)[lane * 2 + 1] = make_uint4(o[4], o[5], o[6], o[7]);
  }
  __syncwarp();
  // scatter by bin (order inside a bin still arbitrary)
  uint32_t pos[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const uint32_t i = r * 32 + lane;
    pos[r] = 0xffffffffu;
    if (r * 32 < (int)len && i < len) {
      const int b = acc_bin((float)Kt::acc(v[r]), scale, 255);
      pos[r] = cnt[b] + slot[r];
      buf[pos[r]] = v[r];
    }
  }
  __syncwarp();
  // buf is now in bin order, and the K smallest keys lie in the bins that
  // start below K: only positions below the end of the bin holding position
  // K-1 are ranked inside their bin and written
  uint32_t end = 0;
  {
    uint32_t st = incl - s;  // start of this lane's first bin
    uint32_t e = 0;
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const uint32_t nx = st + c[t];
      if (st < K && K <= nx) e = nx;  // bin t holds position K-1
      st = nx;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) e = max(e, __shfl_xor_sync(FULL, e, off));
    end = e ? e : len;
  }
  T rsq = 0;
  for (uint32_t p0 = 0; p0 < end; p0 += 32) {
    const uint32_t pp = p0 + lane;
    if (pp < end) {
      const KT w = buf[pp];
      const int b = acc_bin((float)Kt::acc(w), scale, 255);
      const uint32_t first = cnt[b];
      const uint32_t last = b < 255 ? cnt[b + 1] : len;
      uint32_t rank = 0;
      if (last - first > 1)  // a key alone in its bin is ranked by the bin
        for (uint32_t j = first; j < last; j++) rank += Kt::less(buf[j], w) ? 1u : 0u;
      const uint32_t fin = first + rank;
      if (fin < K) {
        const T dist = Num<T>::sqrt(Kt::acc(w));
        out_ids[row_out + fin] = (int32_t)Kt::id(w);
        out_d[row_out + fin] = dist;
        rsq = Num<T>::add(rsq, Num<T>::mul(dist, dist));
      }
    }
  }
  if (rowsum) store_row_sum<T>(rowsum, row_out / K, rsq, lane);
  __syncwarp();
}

// Writes the K smallest of buf[0..len) by a full bitonic sort (any len <= B).
template <typename T>
__device__ __noinline__ void write_sorted_row_bitonic(typename Key<T>::type* buf, uint32_t len, uint32_t K,
                                                      int32_t* __restrict__ out_ids, T* __restrict__ out_d,
                                                      uint64_t row_out, int lane, double* __restrict__ rowsum) {
  using Kt = Key<T>;
  const uint32_t n2 = len <= 1 ? 1u : (1u << (32 - __clz(len - 1)));
  __syncwarp();
  for (uint32_t i = len + lane; i < n2; i += 32) buf[i] = Kt::maxv();
  __syncwarp();
  warp_bitonic_sort<T>(buf, (int)n2, lane);
  T rsq = 0;
  for (uint32_t i = lane; i < K; i += 32) {
    const typename Kt::type kk = buf[i];
    const T dist = Num<T>::sqrt(Kt::acc(kk));
    out_ids[row_out + i] = (int32_t)Kt::id(kk);
    out_d[row_out + i] = dist;
    rsq = Num<T>::add(rsq, Num<T>::mul(dist, dist));
  }
  if (rowsum) store_row_sum<T>(rowsum, row_out / K, rsq, lane);
  __syncwarp();
}

}  // namespace

}  // namespace knnsj
