// k_mlp.cu -- training of the radius MLP (radius_model.cuh) on the GPU with
// hand-written kernels: forward + backward of the pinball (quantile) loss,
// a deterministic gradient reduction and Adam.  No reference counterpart.
//
// A block walks over tiles of TR_TILE samples.  Forward and backward keep the
// tile's activations in shared memory, sample-fastest, and every thread
// computes 2 samples x 16 units (one pair of activations and four weight
// vectors per 32 multiply-adds); the parameter gradients are sums over samples
// that stay in registers (32 of the 64 x 64 layer per thread) until the
// block's last tile.  One partial per block is then summed over blocks in a
// fixed tree -- every run gives the same bits.
//
// What bounds it: shared-memory reads (about one per three multiply-adds), at
// 8 warps per SM.  One thread per sample with rows of 64 floats put all 32
// lanes of a warp on one bank: 1.23 ms for the gradient of 200 003 samples,
// and 0.13 ms for the sum of 3126 partials (call with its host copies: 1.49 ms,
// now 0.42 ms).

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>
#include <vector>

#include "knnsj_internal.h"
#include "radius_model.cuh"

namespace knnsj {

constexpr int NPARAM = MODEL_FLOATS - M_W1;  // trainable: W1..b3 (5825)

namespace {

constexpr int TR_TILE = 64;            // samples per tile
constexpr int TR_THREADS = 128;
constexpr int TR_LD = TR_TILE + 4;     // row stride: 16-byte reads of 8 neighbouring rows hit 8 bank groups
constexpr int TR_MAX_BLOCKS = 2 * 152; // two blocks per SM
constexpr int TR_FLOATS = (NFEAT + 2 * NHID) * TR_LD + TR_TILE + NFEAT * NHID + 2 * NHID * NHID + 3 * NHID + 4;

// out[16][2] of units u0..u0+15 for the samples 2*lane, 2*lane+1: chains over
// `rows` inputs in ascending order, from init[u].
__device__ __forceinline__ void units16(const float* __restrict__ in, const float* __restrict__ w, int rows, int u0,
                                        int lane, float (&a)[16][2]) {
#pragma unroll 4
  for (int i = 0; i < rows; i++) {
    const float2 x = *reinterpret_cast<const float2*>(in + i * TR_LD + 2 * lane);
    const float4* wr = reinterpret_cast<const float4*>(w + i * NHID + u0);
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const float4 wv = wr[v];
      a[4 * v + 0][0] = fmaf(x.x, wv.x, a[4 * v + 0][0]);
      a[4 * v + 0][1] = fmaf(x.y, wv.x, a[4 * v + 0][1]);
      a[4 * v + 1][0] = fmaf(x.x, wv.y, a[4 * v + 1][0]);
      a[4 * v + 1][1] = fmaf(x.y, wv.y, a[4 * v + 1][1]);
      a[4 * v + 2][0] = fmaf(x.x, wv.z, a[4 * v + 2][0]);
      a[4 * v + 2][1] = fmaf(x.y, wv.z, a[4 * v + 2][1]);
      a[4 * v + 3][0] = fmaf(x.x, wv.w, a[4 * v + 3][0]);
      a[4 * v + 3][1] = fmaf(x.y, wv.w, a[4 * v + 3][1]);
    }
  }
}

// acc[i][o] += sum over the tile's samples of p[i0 + i * si][r] * q[o0 + o * so][r]
template <int NI, int NO>
__device__ __forceinline__ void outer_sums(const float* __restrict__ p, int i0, int si, const float* __restrict__ q,
                                           int o0, int so, float (&acc)[NI][NO]) {
#pragma unroll 2
  for (int r = 0; r < TR_TILE; r += 4) {
    float4 pv[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) pv[i] = *reinterpret_cast<const float4*>(p + (i0 + i * si) * TR_LD + r);
#pragma unroll
    for (int o = 0; o < NO; o++) {
      const float4 qv = *reinterpret_cast<const float4*>(q + (o0 + o * so) * TR_LD + r);
#pragma unroll
      for (int i = 0; i < NI; i++) {
        float a = acc[i][o];
        a = fmaf(pv[i].x, qv.x, a);
        a = fmaf(pv[i].y, qv.y, a);
        a = fmaf(pv[i].z, qv.z, a);
        acc[i][o] = fmaf(pv[i].w, qv.w, a);
      }
    }
  }
}

__device__ __forceinline__ float row_sum(const float* __restrict__ row, float a) {
#pragma unroll 4
  for (int r = 0; r < TR_TILE; r += 4) {
    const float4 v = *reinterpret_cast<const float4*>(row + r);
    a = ((a + v.x) + v.y) + v.z;
    a += v.w;
  }
  return a;
}

// grads: per-block partial [gridDim.x][NPARAM]; loss: per-block partial sum
__global__ void __launch_bounds__(TR_THREADS, 2) mlp_fwd_bwd_kernel(const float* __restrict__ model,
                                                                    const float* __restrict__ X,
                                                                    const float* __restrict__ Y,
                                                                    const uint32_t* __restrict__ idx, uint64_t n,
                                                                    float quantile, float inv_batch,
                                                                    float* __restrict__ part_grad,
                                                                    double* __restrict__ part_loss) {
  extern __shared__ __align__(16) float shm[];
  float* xs = shm;                        // [NFEAT][TR_LD] normalised inputs
  float* h1 = xs + NFEAT * TR_LD;         // [NHID][TR_LD]  post-ReLU layer 1, then dL/d(pre-activation 1)
  float* h2 = h1 + NHID * TR_LD;          // [NHID][TR_LD]  post-ReLU layer 2, then dL/d(pre-activation 2)
  float* g3 = h2 + NHID * TR_LD;          // [TR_TILE]      dL/dy
  float* w1 = g3 + TR_TILE;               // [NFEAT][NHID]
  float* w2 = w1 + NFEAT * NHID;          // [NHID in][NHID out]
  float* w2t = w2 + NHID * NHID;          // [NHID out][NHID in]
  float* b1 = w2t + NHID * NHID;
  float* b2 = b1 + NHID;
  float* w3 = b2 + NHID;
  __shared__ double lsum[TR_TILE];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int i = t; i < NFEAT * NHID; i += TR_THREADS) w1[i] = model[M_W1 + i];
  for (int i = t; i < NHID * NHID; i += TR_THREADS) {
    const float v = model[M_W2 + i];
    w2[i] = v;
    w2t[(i % NHID) * NHID + i / NHID] = v;
  }
  if (t < NHID) {
    b1[t] = model[M_B1 + t];
    b2[t] = model[M_B2 + t];
    w3[t] = model[M_W3 + t];
  }
  const float b3 = model[M_B3];
  const int u0 = warp * 16;                     // this warp's units
  const int i2 = t >> 3, o2 = t & 7;            // layer 2: inputs i2 + 16 k, outputs o2 + 8 k
  const int i1 = t & 7, o1 = t >> 3;            // layer 1: inputs i1 + 8 k, outputs o1 + 16 k
  float a2[4][8] = {}, a1[3][4] = {};
  float ab = 0.0f, aw3 = 0.0f, ab3 = 0.0f;      // b1 (threads 0-63) or b2 (64-127); W3; b3
  double loss_sum = 0.0;
  const uint64_t tiles = (n + TR_TILE - 1) / TR_TILE;
  for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    __syncthreads();  // the last tile's gradients are summed (and the weights are in place)
    const uint64_t s0 = tile * TR_TILE;
    for (int e = t; e < TR_TILE * NFEAT; e += TR_THREADS) {
      const int r = e / NFEAT, i = e % NFEAT;
      const bool valid = s0 + r < n;
      const uint64_t row = valid ? (idx ? idx[s0 + r] : s0 + r) : 0;
      xs[i * TR_LD + r] = valid ? (X[row * NFEAT + i] - model[M_MEAN + i]) * model[M_ISTD + i] : 0.0f;
    }
    __syncthreads();
    float a[16][2];
#pragma unroll
    for (int u = 0; u < 16; u++) a[u][0] = a[u][1] = b1[u0 + u];
    units16(xs, w1, NFEAT, u0, lane, a);
#pragma unroll
    for (int u = 0; u < 16; u++)
      *reinterpret_cast<float2*>(h1 + (u0 + u) * TR_LD + 2 * lane) =
          make_float2(fmaxf(a[u][0], 0.0f), fmaxf(a[u][1], 0.0f));
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; u++) a[u][0] = a[u][1] = b2[u0 + u];
    units16(h1, w2, NHID, u0, lane, a);
#pragma unroll
    for (int u = 0; u < 16; u++)
      *reinterpret_cast<float2*>(h2 + (u0 + u) * TR_LD + 2 * lane) =
          make_float2(fmaxf(a[u][0], 0.0f), fmaxf(a[u][1], 0.0f));
    __syncthreads();
    if (t < TR_TILE) {
      // output, and the pinball loss at `quantile`: max(q e, (q - 1) e),
      // e = target - y
      const bool valid = s0 + t < n;
      float y = b3;
#pragma unroll 8
      for (int o = 0; o < NHID; o++) y = fmaf(h2[o * TR_LD + t], w3[o], y);
      float loss = 0.0f, dy = 0.0f;
      if (valid) {
        const float e = Y[idx ? idx[s0 + t] : s0 + t] - y;
        loss = e > 0.0f ? quantile * e : (quantile - 1.0f) * e;
        dy = (e > 0.0f ? -quantile : (1.0f - quantile)) * inv_batch;
      }
      g3[t] = dy;
      lsum[t] = (double)loss;
    }
    __syncthreads();
    if (t < NHID) {  // W3
#pragma unroll 4
      for (int r = 0; r < TR_TILE; r++) aw3 = fmaf(h2[t * TR_LD + r], g3[r], aw3);
    } else if (t == NHID) {
      ab3 = row_sum(g3, ab3);
    } else if (t == NHID + 1) {
      for (int r = 0; r < TR_TILE; r++) loss_sum += lsum[r];
    }
    __syncthreads();
    // dL/d(pre-activation 2), in place
    {
      const float2 dy = *reinterpret_cast<const float2*>(g3 + 2 * lane);
#pragma unroll
      for (int u = 0; u < 16; u++) {
        float2* p = reinterpret_cast<float2*>(h2 + (u0 + u) * TR_LD + 2 * lane);
        const float2 h = *p;
        *p = make_float2(h.x > 0.0f ? dy.x * w3[u0 + u] : 0.0f, h.y > 0.0f ? dy.y * w3[u0 + u] : 0.0f);
      }
    }
    __syncthreads();
    outer_sums<4, 8>(h1, i2, 16, h2, o2, 8, a2);
    if (t >= NHID) ab = row_sum(h2 + (t - NHID) * TR_LD, ab);
    // dL/d(pre-activation 1): in registers, then over h1
#pragma unroll
    for (int u = 0; u < 16; u++) a[u][0] = a[u][1] = 0.0f;
    units16(h2, w2t, NHID, u0, lane, a);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 16; u++) {
      float2* p = reinterpret_cast<float2*>(h1 + (u0 + u) * TR_LD + 2 * lane);
      const float2 h = *p;
      *p = make_float2(h.x > 0.0f ? a[u][0] : 0.0f, h.y > 0.0f ? a[u][1] : 0.0f);
    }
    __syncthreads();
    outer_sums<3, 4>(xs, i1, 8, h1, o1, 16, a1);
    if (t < NHID) ab = row_sum(h1 + t * TR_LD, ab);
  }
  float* pg = part_grad + (uint64_t)blockIdx.x * NPARAM - M_W1;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int o = 0; o < 8; o++) pg[M_W2 + (i2 + 16 * i) * NHID + o2 + 8 * o] = a2[i][o];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int o = 0; o < 4; o++) pg[M_W1 + (i1 + 8 * i) * NHID + o1 + 16 * o] = a1[i][o];
  pg[t < NHID ? M_B1 + t : M_B2 + t - NHID] = ab;
  if (t < NHID) pg[M_W3 + t] = aw3;
  if (t == NHID) pg[M_B3] = ab3;
  if (t == NHID + 1) part_loss[blockIdx.x] = loss_sum;
}

// Sums the blocks' partials: 32 parameters per block, 8 interleaved sums of
// each, added in order.
__global__ void __launch_bounds__(256) grad_reduce_kernel(const float* __restrict__ part, uint32_t nblocks,
                                                          float* __restrict__ grad) {
  __shared__ float ws[8][32];
  const int p = blockIdx.x * 32 + (threadIdx.x & 31), k = threadIdx.x >> 5;
  float a = 0.0f;
  if (p < NPARAM)
    for (uint32_t b = k; b < nblocks; b += 8) a += part[(uint64_t)b * NPARAM + p];
  ws[k][threadIdx.x & 31] = a;
  __syncthreads();
  if (k == 0 && p < NPARAM) {
    for (int j = 1; j < 8; j++) a += ws[j][threadIdx.x];
    grad[p] = a;
  }
}

__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m1,
                            float* __restrict__ m2, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= NPARAM) return;
  const float gp = g[p];
  const float a = b1 * m1[p] + (1.0f - b1) * gp;
  const float v = b2 * m2[p] + (1.0f - b2) * gp * gp;
  m1[p] = a;
  m2[p] = v;
  const float mh = a / c1, vh = v / c2;
  w[p] -= lr * mh / (sqrtf(vh) + eps);
}

}  // namespace

uint32_t mlp_grad_blocks(uint64_t n) {
  return (uint32_t)std::min<uint64_t>((n + TR_TILE - 1) / TR_TILE, TR_MAX_BLOCKS);
}
size_t mlp_grad_partials(uint64_t n) { return (size_t)mlp_grad_blocks(n) * NPARAM; }

// Full gradient (sum over the batch of the pinball loss / n) and loss (one
// partial sum per block) of `model` on n samples already on the device.
void mlp_grad_device(const float* d_model, const float* d_X, const float* d_Y, const uint32_t* d_idx, uint64_t n,
                     float quantile, float inv_batch, float* d_part, double* d_part_loss, float* d_grad,
                     cudaStream_t s) {
  const uint32_t nb = mlp_grad_blocks(n);
  constexpr int sm = TR_FLOATS * (int)sizeof(float);
  KNNSJ_CUDA(cudaFuncSetAttribute(mlp_fwd_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  mlp_fwd_bwd_kernel<<<nb, TR_THREADS, sm, s>>>(d_model, d_X, d_Y, d_idx, n, quantile, inv_batch, d_part, d_part_loss);
  KNNSJ_CHECK_LAUNCH();
  grad_reduce_kernel<<<(NPARAM + 31) / 32, 256, 0, s>>>(d_part, nb, d_grad);
  KNNSJ_CHECK_LAUNCH();
}

struct TrainBuffers {
  DevBuf model, X, Y, idx, part, ploss, grad, m1, m2;
};

// Seeded initial model: feature standardisation from the data, He-normal
// weights, zero biases, output bias at the target's `quantile` quantile.
void init_model(const float* X, const float* Y, uint64_t n, float quantile, uint64_t seed, float* model) {
  std::memset(model, 0, sizeof(float) * MODEL_FLOATS);
  for (int i = 0; i < NFEAT; i++) {
    double s = 0, s2 = 0;
    for (uint64_t r = 0; r < n; r++) {
      const double v = X[r * NFEAT + i];
      s += v;
      s2 += v * v;
    }
    const double mean = n ? s / n : 0.0;
    const double var = n ? std::max(0.0, s2 / n - mean * mean) : 0.0;
    model[M_MEAN + i] = (float)mean;
    model[M_ISTD + i] = (float)(var > 1e-12 ? 1.0 / std::sqrt(var) : 1.0);
  }
  std::mt19937_64 rng(seed);
  std::normal_distribution<double> nd(0.0, 1.0);
  for (int i = 0; i < NFEAT * NHID; i++) model[M_W1 + i] = (float)(nd(rng) * std::sqrt(2.0 / NFEAT));
  for (int i = 0; i < NHID * NHID; i++) model[M_W2 + i] = (float)(nd(rng) * std::sqrt(2.0 / NHID));
  for (int i = 0; i < NHID; i++) model[M_W3 + i] = (float)(nd(rng) * std::sqrt(1.0 / NHID) * 0.1);
  if (n) {
    std::vector<float> ys(Y, Y + n);
    const size_t at = std::min<size_t>(n - 1, (size_t)(quantile * (n - 1)));
    std::nth_element(ys.begin(), ys.begin() + at, ys.end());
    model[M_B3] = ys[at];
  }
}

void train_model(const float* hX, const float* hY, uint64_t n, int epochs, uint32_t batch, float lr,
                 float quantile, uint64_t seed, float* model_out, float* loss_out, cudaStream_t s) {
  static TrainBuffers b;
  std::vector<float> model(MODEL_FLOATS);
  init_model(hX, hY, n, quantile, seed, model.data());
  float* d_model = (float*)b.model.get(MODEL_FLOATS * 4);
  float* d_X = (float*)b.X.get(n * NFEAT * 4);
  float* d_Y = (float*)b.Y.get(n * 4);
  uint32_t* d_idx = (uint32_t*)b.idx.get(n * 4);
  const uint32_t nbmax = mlp_grad_blocks(batch);
  float* d_part = (float*)b.part.get((size_t)nbmax * NPARAM * 4);
  double* d_pl = (double*)b.ploss.get((size_t)nbmax * 8);
  float* d_grad = (float*)b.grad.get(NPARAM * 4);
  float* d_m1 = (float*)b.m1.get(NPARAM * 4);
  float* d_m2 = (float*)b.m2.get(NPARAM * 4);
  KNNSJ_CUDA(cudaMemcpyAsync(d_model, model.data(), MODEL_FLOATS * 4, cudaMemcpyHostToDevice, s));
  KNNSJ_CUDA(cudaMemcpyAsync(d_X, hX, n * NFEAT * 4, cudaMemcpyHostToDevice, s));
  KNNSJ_CUDA(cudaMemcpyAsync(d_Y, hY, n * 4, cudaMemcpyHostToDevice, s));
  KNNSJ_CUDA(cudaMemsetAsync(d_m1, 0, NPARAM * 4, s));
  KNNSJ_CUDA(cudaMemsetAsync(d_m2, 0, NPARAM * 4, s));
  std::vector<uint32_t> perm(n);
  std::iota(perm.begin(), perm.end(), 0u);
  std::mt19937_64 rng(seed ^ 0x9e3779b97f4a7c15ull);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  int step = 0;
  std::vector<double> pl(nbmax);
  for (int e = 0; e < epochs; e++) {
    std::shuffle(perm.begin(), perm.end(), rng);
    KNNSJ_CUDA(cudaMemcpyAsync(d_idx, perm.data(), n * 4, cudaMemcpyHostToDevice, s));
    KNNSJ_CUDA(cudaStreamSynchronize(s));
    double epoch_loss = 0.0;
    for (uint64_t off = 0; off < n; off += batch) {
      const uint64_t nb = std::min<uint64_t>(batch, n - off);
      mlp_grad_device(d_model, d_X, d_Y, d_idx + off, nb, quantile, 1.0f / (float)nb, d_part, d_pl, d_grad, s);
      step++;
      const float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
      adam_kernel<<<(NPARAM + 255) / 256, 256, 0, s>>>(d_model + M_W1, d_grad, d_m1, d_m2, lr, b1, b2, eps, c1, c2);
      KNNSJ_CHECK_LAUNCH();
      const uint32_t nblk = mlp_grad_blocks(nb);
      KNNSJ_CUDA(cudaMemcpyAsync(pl.data(), d_pl, nblk * 8, cudaMemcpyDeviceToHost, s));
      KNNSJ_CUDA(cudaStreamSynchronize(s));
      for (uint32_t i = 0; i < nblk; i++) epoch_loss += pl[i];
    }
    if (loss_out) loss_out[e] = (float)(epoch_loss / (double)n);
  }
  KNNSJ_CUDA(cudaMemcpyAsync(model_out, d_model, MODEL_FLOATS * 4, cudaMemcpyDeviceToHost, s));
  KNNSJ_CUDA(cudaStreamSynchronize(s));
}

}  // namespace knnsj
