// k_prep.cu -- input preparation on the device.
//
//  * transpose_reorder: row-major N x d input -> d column arrays in the
//    variance order chosen by ReorderByDimension (main.cu:2521-2615; the
//    reference permutes its host vectors, main.cu:2596-2605), flagging NaN /
//    infinite coordinates on the way.
//  * minmax: per-dimension minimum and maximum of the indexed dimensions, the
//    first half of generateNDGridDimensions (main.cu:2425-2460).

#include <algorithm>
#include <cfloat>

#include "exact_sqrt.cuh"
#include "knnsj_internal.h"

namespace knnsj {

namespace {

struct DimOrder {
  uint16_t p[MAX_D];
};

template <typename T>
__global__ void transpose_reorder_kernel(const T* __restrict__ aos, T* __restrict__ soa, float* __restrict__ soaf,
                                         uint64_t n, uint32_t d, const DimOrder perm,
                                         uint32_t* __restrict__ nonfinite) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  bool bad = false;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    for (uint32_t j = 0; j < d; j++) {
      const T v = aos[i * d + perm.p[j]];
      bad |= !isfinite(v);
      soa[(uint64_t)j * n + i] = v;
      if (soaf) soaf[(uint64_t)j * n + i] = (float)v;
    }
  }
  if (__any_sync(FULL, bad) && (threadIdx.x & 31) == 0) atomicOr(nonfinite, 1u);
}

template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ aos, uint64_t count, uint64_t step, uint32_t d,
                                   T* __restrict__ out) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < count * d;
       e += (uint64_t)gridDim.x * blockDim.x)
    out[e] = aos[e / d * step * d + e % d];
}

template <typename T>
__device__ __forceinline__ T tmin(T a, T b) { return b < a ? b : a; }
template <typename T>
__device__ __forceinline__ T tmax(T a, T b) { return b > a ? b : a; }

// Minimum and maximum over a block's threads, in thread 0.
template <typename T>
__device__ __forceinline__ void block_minmax(T& mn, T& mx) {
  __shared__ T smin[32], smax[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int off = 16; off > 0; off >>= 1) {
    mn = tmin(mn, __shfl_xor_sync(FULL, mn, off));
    mx = tmax(mx, __shfl_xor_sync(FULL, mx, off));
  }
  if (lane == 0) {
    smin[w] = mn;
    smax[w] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 1; k < (int)(blockDim.x >> 5); k++) {
      mn = tmin(mn, smin[k]);
      mx = tmax(mx, smax[k]);
    }
}

// Stage 1: min/max of column blockIdx.y over a block's points into
// part[column][2 * block].
template <typename T>
__global__ void minmax_kernel(const T* __restrict__ soa, uint64_t n, T* __restrict__ part) {
  const T* col = soa + (uint64_t)blockIdx.y * n;
  T mn = col[0], mx = mn;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const T v = col[i];
    mn = tmin(mn, v);
    mx = tmax(mx, v);
  }
  block_minmax(mn, mx);
  if (threadIdx.x == 0) {
    T* o = part + 2 * ((uint64_t)blockIdx.y * gridDim.x + blockIdx.x);
    o[0] = mn;
    o[1] = mx;
  }
}

// Stage 2: one block per column over its blocks' extremes.  (One thread per
// column walked the up to 1024 partial results one after the other: 93 us of
// a 1M-point join, 236 us of a 10M-point double one; now 3 us.)
template <typename T>
__global__ void minmax_final_kernel(const T* __restrict__ part, uint32_t nblocks, T* __restrict__ out) {
  const T* p = part + 2 * (uint64_t)blockIdx.x * nblocks;
  T mn = p[0], mx = p[1];
  for (uint32_t b = threadIdx.x; b < nblocks; b += blockDim.x) {
    mn = tmin(mn, p[2 * b]);
    mx = tmax(mx, p[2 * b + 1]);
  }
  block_minmax(mn, mx);
  if (threadIdx.x == 0) {
    out[2 * blockIdx.x] = mn;
    out[2 * blockIdx.x + 1] = mx;
  }
}

constexpr unsigned CHECKSUM_BLOCKS = 1024;

// Squared distance in DTYPE, widened and added in double (GPU.cu:3690-3693);
// fixed grid, fixed per-thread order and a fixed tree, so the figure is the
// same on every run.
// exact widening to double (float: assembled from bits, off the FP64 pipe)
__device__ __forceinline__ double widen(float x) { return es_f2d(x); }
__device__ __forceinline__ double widen(double x) { return x; }

template <typename T>
__global__ void checksum_kernel(const T* __restrict__ v, uint64_t count, double* __restrict__ part) {
  __shared__ double ws[32];
  double s = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const T x = v[i];
    s = __dadd_rn(s, widen(Num<T>::mul(x, x)));
  }
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(FULL, s, off);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += ws[k];
    part[blockIdx.x] = t;
  }
}

// One block: the block partials in a fixed tree.  (One thread adding the 1024
// of them in a row took 61 us.)
__global__ void __launch_bounds__(CHECKSUM_BLOCKS) checksum_final_kernel(const double* __restrict__ part,
                                                                        double* __restrict__ out) {
  __shared__ double ws[32];
  double s = part[threadIdx.x];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(FULL, s, off);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = ws[threadIdx.x];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(FULL, s, off);
    if (threadIdx.x == 0) *out = s;
  }
}

// Sum of n doubles in a fixed order: grid-stride partial sums per thread,
// warp butterflies, block partials summed in block order.
__global__ void sum_f64_kernel(const double* __restrict__ v, uint64_t count, double* __restrict__ part) {
  __shared__ double ws[32];
  double s = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x)
    s = __dadd_rn(s, v[i]);
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(FULL, s, off);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += ws[k];
    part[blockIdx.x] = t;
  }
}

}  // namespace

void launch_sum_f64(const double* v, uint64_t count, double* d_partial, double* d_out, cudaStream_t s) {
  sum_f64_kernel<<<CHECKSUM_BLOCKS, 256, 0, s>>>(v, count, d_partial);
  KNNSJ_CHECK_LAUNCH();
  checksum_final_kernel<<<1, CHECKSUM_BLOCKS, 0, s>>>(d_partial, d_out);
  KNNSJ_CHECK_LAUNCH();
}

template <typename T>
void launch_checksum(const T* dists, uint64_t count, double* d_partial, double* d_out, cudaStream_t s) {
  checksum_kernel<T><<<CHECKSUM_BLOCKS, 256, 0, s>>>(dists, count, d_partial);
  KNNSJ_CHECK_LAUNCH();
  checksum_final_kernel<<<1, CHECKSUM_BLOCKS, 0, s>>>(d_partial, d_out);
  KNNSJ_CHECK_LAUNCH();
}
template void launch_checksum<float>(const float*, uint64_t, double*, double*, cudaStream_t);
template void launch_checksum<double>(const double*, uint64_t, double*, double*, cudaStream_t);

constexpr uint32_t MINMAX_BLOCKS = 1024;

template <typename T>
void launch_transpose_reorder(const T* aos, T* soa, float* soaf, uint64_t n, uint32_t d, const uint32_t* perm,
                              cudaStream_t s, uint32_t* d_nonfinite) {
  DimOrder order{};
  for (uint32_t j = 0; j < d; j++) order.p[j] = (uint16_t)perm[j];
  uint64_t blocks = (n + 255) / 256;
  if (blocks > 152ull * 32) blocks = 152ull * 32;
  transpose_reorder_kernel<T><<<(unsigned)blocks, 256, 0, s>>>(aos, soa, soaf, n, d, order, d_nonfinite);
  KNNSJ_CHECK_LAUNCH();
}

template <typename T>
void launch_gather_rows(const T* aos, uint64_t count, uint64_t step, uint32_t d, T* out, cudaStream_t s) {
  const uint64_t blocks = std::min<uint64_t>((count * d + 255) / 256, 152ull * 8);
  gather_rows_kernel<T><<<(unsigned)std::max<uint64_t>(blocks, 1), 256, 0, s>>>(aos, count, step, d, out);
  KNNSJ_CHECK_LAUNCH();
}

template <typename T>
void launch_minmax(const T* soa, uint64_t n, uint32_t di, T* d_minmax, T* scratch, cudaStream_t s) {
  uint32_t blocks = (uint32_t)((n + 255) / 256);
  if (blocks > MINMAX_BLOCKS) blocks = MINMAX_BLOCKS;
  if (blocks < 1) blocks = 1;
  minmax_kernel<T><<<dim3(blocks, di), 256, 0, s>>>(soa, n, scratch);
  KNNSJ_CHECK_LAUNCH();
  minmax_final_kernel<T><<<di, 256, 0, s>>>(scratch, blocks, d_minmax);
  KNNSJ_CHECK_LAUNCH();
}

template void launch_transpose_reorder<float>(const float*, float*, float*, uint64_t, uint32_t, const uint32_t*,
                                              cudaStream_t, uint32_t*);
template void launch_transpose_reorder<double>(const double*, double*, float*, uint64_t, uint32_t,
                                               const uint32_t*, cudaStream_t, uint32_t*);
template void launch_gather_rows<float>(const float*, uint64_t, uint64_t, uint32_t, float*, cudaStream_t);
template void launch_gather_rows<double>(const double*, uint64_t, uint64_t, uint32_t, double*, cudaStream_t);
template void launch_minmax<float>(const float*, uint64_t, uint32_t, float*, float*, cudaStream_t);
template void launch_minmax<double>(const double*, uint64_t, uint32_t, double*, double*, cudaStream_t);

}  // namespace knnsj
