// Learned work predictor and the learned scheduler (no counterpart in the reference).
//
// A small MLP (8 features -> 32 -> 32 -> 1, FP32, ReLU) predicts log(1 + subtree size) of a
// root task, where the subtree size is the number of subgraphs the task counts (the log the
// plain engine writes through dm_opts.subtree_counts). Training, gradients and inference
// are this file's own CUDA kernels: a per-sample forward/backward whose activations stay in
// shared memory, a per-parameter reduction over each block's samples, and an Adam step.
//
// Features of root v for a k query (all FP32):
//   f0 log1p(deg v)            f1 log1p(core number of v)
//   f2 log1p(|C_0|)            candidate-set size: out-degree in the degree-ordered DAG for
//                              cliques, neighbours above v for motifs
//   f3 k / 8                   f4 (k - 2) / 8: DFS depth below a root task
//   f5 log1p(DAG out-degree)   f6 log1p(2-hop size: sum over C_0 of DAG out-degrees for
//                              cliques, of degrees for motifs)
//   f7 log1p(triangles whose lowest-ranked vertex is v)
//
// The learned scheduler orders root tasks by predicted cost (longest first) and splits a
// root whose predicted cost exceeds the per-warp share into P parts up front, so heavy
// subtrees start on several warps at once instead of waiting for reactive donation.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "engine.hpp"

// MLP geometry
constexpr int MLP_F = 8, MLP_H = 32;
constexpr int OFF_W1 = 0;                       // [H][F]
constexpr int OFF_B1 = OFF_W1 + MLP_H * MLP_F;  // [H]
constexpr int OFF_W2 = OFF_B1 + MLP_H;          // [H][H] (row = output unit)
constexpr int OFF_B2 = OFF_W2 + MLP_H * MLP_H;  // [H]
constexpr int OFF_W3 = OFF_B2 + MLP_H;          // [H]
constexpr int OFF_B3 = OFF_W3 + MLP_H;          // [1]
constexpr int MLP_NP = OFF_B3 + 1;              // 1377

struct dm_predictor {
  int device = -1;
  uint64_t uid = 0;           // identity for schedule caches
  uint64_t version = 0;       // bumped whenever the parameters change
  std::vector<float> params;  // host copy (authoritative between calls)
  uint64_t seed = 0;
  int steps = 0;
  std::vector<float> adam_m, adam_v;
};

namespace dmb {

static std::atomic<uint64_t> g_pred_uid{1};

// (identity, parameter version) of a predictor, the key of cached learned schedules.
void predictor_key(const void* pv, uint64_t* uid, uint64_t* version) {
  const dm_predictor* p = reinterpret_cast<const dm_predictor*>(pv);
  *uid = p->uid;
  *version = p->version;
}

// MLP forward of one feature row, parameters in shared memory.
__device__ __forceinline__ float mlp_eval(const float* sp, const float* x) {
  float h1[MLP_H];
#pragma unroll
  for (int h = 0; h < MLP_H; ++h) {
    float a = sp[OFF_B1 + h];
#pragma unroll
    for (int f = 0; f < MLP_F; ++f) a = fmaf(sp[OFF_W1 + h * MLP_F + f], x[f], a);
    h1[h] = fmaxf(a, 0.f);
  }
  float out = sp[OFF_B3];
  for (int h = 0; h < MLP_H; ++h) {
    float a = sp[OFF_B2 + h];
#pragma unroll
    for (int j = 0; j < MLP_H; ++j) a = fmaf(sp[OFF_W2 + h * MLP_H + j], h1[j], a);
    out = fmaf(sp[OFF_W3 + h], fmaxf(a, 0.f), out);
  }
  return out;
}

__global__ void mlp_forward_kernel(const float* __restrict__ P, const float* __restrict__ X, int n,
                                   float* __restrict__ y) {
  __shared__ float sp[MLP_NP];
  for (int i = threadIdx.x; i < MLP_NP; i += blockDim.x) sp[i] = P[i];
  __syncthreads();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  float x[MLP_F];
#pragma unroll
  for (int f = 0; f < MLP_F; ++f) x[f] = X[(size_t)s * MLP_F + f];
  y[s] = mlp_eval(sp, x);
}

// Gradients of mean squared error over the samples idx[0..n) (or 0..n when idx is null).
// One block takes TB samples: each thread runs one sample forward and back to the
// pre-activation gradients, keeping inputs, activations and those gradients in shared
// memory; then the block reduces every parameter's gradient over its samples and adds it
// to `grad` (zeroed by the caller) with one atomic per parameter. loss_sum receives the sum
// of squared errors.
constexpr int TB = 128;
constexpr int ROW = MLP_F + 4 * MLP_H + 1;  // x | h1 | h2 | dz1 | dz2 | dy

__global__ void __launch_bounds__(TB) mlp_backward_kernel(const float* __restrict__ P, const float* __restrict__ X,
                                                          const float* __restrict__ T, const int* __restrict__ idx,
                                                          int n, float inv_n, float* __restrict__ grad,
                                                          float* __restrict__ loss_sum) {
  extern __shared__ float sm[];
  float* sp = sm;               // MLP_NP
  float* rows = sm + MLP_NP + 3;  // TB x ROW
  for (int i = threadIdx.x; i < MLP_NP; i += blockDim.x) sp[i] = P[i];
  __syncthreads();
  const int t = blockIdx.x * TB + threadIdx.x;
  float* r = rows + threadIdx.x * ROW;
  float* rx = r;
  float* rh1 = r + MLP_F;
  float* rh2 = rh1 + MLP_H;
  float* rd1 = rh2 + MLP_H;
  float* rd2 = rd1 + MLP_H;
  float sq = 0.f;
  if (t < n) {
    const int s = idx ? idx[t] : t;
#pragma unroll
    for (int f = 0; f < MLP_F; ++f) rx[f] = X[(size_t)s * MLP_F + f];
    for (int h = 0; h < MLP_H; ++h) {
      float a = sp[OFF_B1 + h];
#pragma unroll
      for (int f = 0; f < MLP_F; ++f) a = fmaf(sp[OFF_W1 + h * MLP_F + f], rx[f], a);
      rh1[h] = fmaxf(a, 0.f);
    }
    float out = sp[OFF_B3];
    for (int h = 0; h < MLP_H; ++h) {
      float a = sp[OFF_B2 + h];
      for (int j = 0; j < MLP_H; ++j) a = fmaf(sp[OFF_W2 + h * MLP_H + j], rh1[j], a);
      rh2[h] = fmaxf(a, 0.f);
      out = fmaf(sp[OFF_W3 + h], rh2[h], out);
    }
    const float err = out - T[s];
    sq = err * err;
    const float dy = 2.f * err * inv_n;
    r[ROW - 1] = dy;
    for (int h = 0; h < MLP_H; ++h) rd2[h] = rh2[h] > 0.f ? dy * sp[OFF_W3 + h] : 0.f;
    for (int j = 0; j < MLP_H; ++j) {
      float a = 0.f;
      for (int h = 0; h < MLP_H; ++h) a = fmaf(rd2[h], sp[OFF_W2 + h * MLP_H + j], a);
      rd1[j] = rh1[j] > 0.f ? a : 0.f;
    }
  } else {
    for (int i = 0; i < ROW; ++i) r[i] = 0.f;
  }
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if ((threadIdx.x & 31) == 0 && sq != 0.f) atomicAdd(loss_sum, sq);
  __syncthreads();
  // per-parameter reductions over the block's samples
  for (int i = threadIdx.x; i < MLP_NP; i += blockDim.x) {
    float acc = 0.f;
    if (i < OFF_B1) {  // W1[h][f] = sum dz1[h] x[f]
      const int h = i / MLP_F, f = i % MLP_F;
      for (int q = 0; q < TB; ++q) acc = fmaf(rows[q * ROW + MLP_F + 2 * MLP_H + h], rows[q * ROW + f], acc);
    } else if (i < OFF_W2) {  // b1[h] = sum dz1[h]
      const int h = i - OFF_B1;
      for (int q = 0; q < TB; ++q) acc += rows[q * ROW + MLP_F + 2 * MLP_H + h];
    } else if (i < OFF_B2) {  // W2[h][j] = sum dz2[h] h1[j]
      const int h = (i - OFF_W2) / MLP_H, j = (i - OFF_W2) % MLP_H;
      for (int q = 0; q < TB; ++q)
        acc = fmaf(rows[q * ROW + MLP_F + 3 * MLP_H + h], rows[q * ROW + MLP_F + j], acc);
    } else if (i < OFF_W3) {  // b2[h] = sum dz2[h]
      const int h = i - OFF_B2;
      for (int q = 0; q < TB; ++q) acc += rows[q * ROW + MLP_F + 3 * MLP_H + h];
    } else if (i < OFF_B3) {  // W3[h] = sum dy h2[h]
      const int h = i - OFF_W3;
      for (int q = 0; q < TB; ++q) acc = fmaf(rows[q * ROW + ROW - 1], rows[q * ROW + MLP_F + MLP_H + h], acc);
    } else {  // b3 = sum dy
      for (int q = 0; q < TB; ++q) acc += rows[q * ROW + ROW - 1];
    }
    if (acc != 0.f) atomicAdd(grad + i, acc);
  }
}

constexpr size_t BACKWARD_SMEM = sizeof(float) * (MLP_NP + 3 + TB * ROW);

__global__ void adam_kernel(float* __restrict__ P, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= MLP_NP) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  P[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// A whole epoch of minibatches in one launch: a cluster of EP_CTAS blocks takes every step's
// samples interleaved (sample q of the batch on block q mod EP_CTAS), each block runs its samples
// forward and back through register tiles over shared memory and leaves its partial gradient in
// its shared memory; after a cluster barrier each block sums one slice of the parameters over the
// blocks' partial gradients through distributed shared memory (in block order, so a run is
// reproducible), takes the Adam step for the slice (its moments stay in registers for the epoch)
// and stores the new parameters into every block's copy. The next tile's samples and the indices
// after it are loaded while the current tile is computed.
//
// A step is a chain of small dependent pieces, bound by latency: with three launches per step
// (clear, backward, Adam) the launches and one thread per sample took about 29 us per step of 256
// samples; four epochs over the subtree log of a graph of 18,700 vertices and a count scheduled
// with the result took 9.29 ms, with a cluster of 8 blocks 1.88 ms and of 16 about 1.6 ms (a step is
// then 4.5 us). Batches above EP_BATCH_MAX keep those launches, which use every SM.
constexpr int EP_THREADS = 256, EP_TILE = 32;  // samples per block and tile
constexpr int EP_LD = MLP_H + 4;                            // padded row of 32 floats (16-byte rows)
constexpr int EP_BATCH_MAX = 4096;
static_assert((MLP_NP + 7) / 8 <= EP_THREADS && EP_TILE * MLP_F == EP_THREADS, "thread maps of the epoch kernel");

struct EpochArgs {
  float* P;
  float* M;
  float* V;
  const float* X;
  const float* T;
  const int* idx;          // the epoch's sample order
  const float2* bias;      // per step: 1 - b1^t, 1 - b2^t
  float* loss_sum;
  int n, batch;
  float lr, b1, b2, eps;
};

// Tile t0 of the minibatch starting at `off`.
template <int EP_CTAS>
struct EpochTile {
  int off, t0;
  __device__ __forceinline__ int size(const EpochArgs& a) const { return min(a.batch, a.n - off); }
  __device__ __forceinline__ bool last(const EpochArgs& a) const { return t0 + EP_CTAS * EP_TILE >= size(a); }
  __device__ __forceinline__ void next(const EpochArgs& a) {
    if (last(a)) {
      off += a.batch;
      t0 = 0;
    } else {
      t0 += EP_CTAS * EP_TILE;
    }
  }
  // global place of sample q of this block's share (-1: none)
  __device__ __forceinline__ int place(const EpochArgs& a, int cta, int q) const {
    const int i = t0 + q * EP_CTAS + cta;
    return off < a.n && i < size(a) ? off + i : -1;
  }
};

template <int EP_CTAS>
__global__ void __cluster_dims__(EP_CTAS, 1, 1) __launch_bounds__(EP_THREADS) mlp_epoch_kernel(const __grid_constant__ EpochArgs a) {
  namespace cg = cooperative_groups;
  constexpr int EP_SLICE = (MLP_NP + EP_CTAS - 1) / EP_CTAS;
  cg::cluster_group cl = cg::this_cluster();
  const int cta = (int)cl.block_rank(), t = threadIdx.x;
  __shared__ __align__(16) float W1[MLP_H * MLP_F], W2[MLP_H * EP_LD];
  __shared__ float B1[MLP_H], B2[MLP_H], W3[MLP_H], B3[1];
  __shared__ __align__(16) float x[EP_TILE * MLP_F], h1[EP_TILE * EP_LD], h2[EP_TILE * EP_LD], d1[EP_TILE * EP_LD],
      d2[EP_TILE * EP_LD];
  __shared__ float tgt[EP_TILE], dy[EP_TILE], grad[MLP_NP];
  // shared-memory home of parameter i
  auto home = [&](int i) -> float* {
    if (i < OFF_B1) return W1 + i;
    if (i < OFF_W2) return B1 + (i - OFF_B1);
    if (i < OFF_B2) return W2 + (i - OFF_W2) / MLP_H * EP_LD + (i - OFF_W2) % MLP_H;
    if (i < OFF_W3) return B2 + (i - OFF_B2);
    if (i < OFF_B3) return W3 + (i - OFF_W3);
    return B3;
  };
  for (int i = t; i < MLP_NP; i += EP_THREADS) *home(i) = a.P[i];
  // this thread's parameter of the block's slice
  const int mine = cta * EP_SLICE + t;
  const bool owner = t < EP_SLICE && mine < MLP_NP;
  float pm = 0.f, pv = 0.f, pp = 0.f;
  if (owner) {
    pm = a.M[mine];
    pv = a.V[mine];
    pp = a.P[mine];
  }
  const int s8 = t >> 3, q8 = t & 7;     // 8 threads per sample (or unit of W1)
  const int hi = t >> 4, lo = t & 15;    // 2 x 2 tiles: rows hi, hi + 16, columns lo, lo + 16
  float gw2[4], gw1, gb;                 // the batch's gradients this thread holds
  float loss = 0.f;
  EpochTile<EP_CTAS> cur{0, 0}, nxt{0, 0};
  // samples of the first tile, and the indices of the second
  int at = cur.place(a, cta, s8);
  int sidx = at >= 0 ? a.idx[at] : -1;
  float xr = sidx >= 0 ? a.X[(size_t)sidx * MLP_F + q8] : 0.f;
  float tr = sidx >= 0 && q8 == 0 ? a.T[sidx] : 0.f;
  nxt.next(a);
  at = nxt.place(a, cta, s8);
  sidx = at >= 0 ? a.idx[at] : -1;
  cl.sync();
  for (int step = 0; cur.off < a.n;) {
    const int bn = cur.size(a);
    const int ns = min(EP_TILE, max(0, (bn - cur.t0 - cta + EP_CTAS - 1) / EP_CTAS));  // samples here
    if (cur.t0 == 0) {
      gw1 = gb = 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) gw2[q] = 0.f;
    }
    x[t] = xr;
    if (q8 == 0) tgt[s8] = tr;
    __syncthreads();
    // the next tile's samples, and the indices of the one after it
    xr = sidx >= 0 ? a.X[(size_t)sidx * MLP_F + q8] : 0.f;
    tr = sidx >= 0 && q8 == 0 ? a.T[sidx] : 0.f;
    nxt.next(a);
    at = nxt.place(a, cta, s8);
    sidx = at >= 0 ? a.idx[at] : -1;
    // h1 = relu(W1 x + b1): four units of one sample
    if (s8 < ns) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int h = q8 + 8 * q;
        float v = B1[h];
#pragma unroll
        for (int f = 0; f < MLP_F; ++f) v = fmaf(W1[h * MLP_F + f], x[s8 * MLP_F + f], v);
        h1[s8 * EP_LD + h] = fmaxf(v, 0.f);
      }
    }
    __syncthreads();
    // h2 = relu(W2 h1 + b2): samples hi, hi + 16 by units lo, lo + 16
    if (hi < ns) {
      const bool two = hi + 16 < ns;
      float v00 = B2[lo], v01 = B2[lo + 16], v10 = v00, v11 = v01;
#pragma unroll
      for (int j = 0; j < MLP_H; j += 4) {
        const float4 w0 = *reinterpret_cast<const float4*>(W2 + lo * EP_LD + j);
        const float4 w1 = *reinterpret_cast<const float4*>(W2 + (lo + 16) * EP_LD + j);
        const float4 a0 = *reinterpret_cast<const float4*>(h1 + hi * EP_LD + j);
        v00 = fmaf(w0.w, a0.w, fmaf(w0.z, a0.z, fmaf(w0.y, a0.y, fmaf(w0.x, a0.x, v00))));
        v01 = fmaf(w1.w, a0.w, fmaf(w1.z, a0.z, fmaf(w1.y, a0.y, fmaf(w1.x, a0.x, v01))));
        if (two) {
          const float4 a1 = *reinterpret_cast<const float4*>(h1 + (hi + 16) * EP_LD + j);
          v10 = fmaf(w0.w, a1.w, fmaf(w0.z, a1.z, fmaf(w0.y, a1.y, fmaf(w0.x, a1.x, v10))));
          v11 = fmaf(w1.w, a1.w, fmaf(w1.z, a1.z, fmaf(w1.y, a1.y, fmaf(w1.x, a1.x, v11))));
        }
      }
      h2[hi * EP_LD + lo] = fmaxf(v00, 0.f);
      h2[hi * EP_LD + lo + 16] = fmaxf(v01, 0.f);
      if (two) {
        h2[(hi + 16) * EP_LD + lo] = fmaxf(v10, 0.f);
        h2[(hi + 16) * EP_LD + lo + 16] = fmaxf(v11, 0.f);
      }
    }
    __syncthreads();
    // output, error, and the gradient at the second pre-activation: four units of one sample
    {
      float o = 0.f;
      if (s8 < ns) {
#pragma unroll
        for (int q = 0; q < 4; ++q) o = fmaf(W3[q8 + 8 * q], h2[s8 * EP_LD + q8 + 8 * q], o);
      }
      o += __shfl_xor_sync(0xffffffffu, o, 1);
      o += __shfl_xor_sync(0xffffffffu, o, 2);
      o += __shfl_xor_sync(0xffffffffu, o, 4);
      if (s8 < ns) {
        const float err = o + B3[0] - tgt[s8];
        const float g = 2.f * err * (1.f / (float)bn);
        if (q8 == 0) {
          dy[s8] = g;
          loss += err * err;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int h = q8 + 8 * q;
          d2[s8 * EP_LD + h] = h2[s8 * EP_LD + h] > 0.f ? g * W3[h] : 0.f;
        }
      }
    }
    __syncthreads();
    // the gradient at the first pre-activation
    if (hi < ns) {
      const bool two = hi + 16 < ns;
      float v00 = 0.f, v01 = 0.f, v10 = 0.f, v11 = 0.f;
#pragma unroll
      for (int h = 0; h < MLP_H; ++h) {
        const float w0 = W2[h * EP_LD + lo], w1 = W2[h * EP_LD + lo + 16];
        const float a0 = d2[hi * EP_LD + h];
        v00 = fmaf(a0, w0, v00);
        v01 = fmaf(a0, w1, v01);
        if (two) {
          const float a1 = d2[(hi + 16) * EP_LD + h];
          v10 = fmaf(a1, w0, v10);
          v11 = fmaf(a1, w1, v11);
        }
      }
      d1[hi * EP_LD + lo] = h1[hi * EP_LD + lo] > 0.f ? v00 : 0.f;
      d1[hi * EP_LD + lo + 16] = h1[hi * EP_LD + lo + 16] > 0.f ? v01 : 0.f;
      if (two) {
        d1[(hi + 16) * EP_LD + lo] = h1[(hi + 16) * EP_LD + lo] > 0.f ? v10 : 0.f;
        d1[(hi + 16) * EP_LD + lo + 16] = h1[(hi + 16) * EP_LD + lo + 16] > 0.f ? v11 : 0.f;
      }
    }
    __syncthreads();
    // parameter gradients over the tile's samples: a 2 x 2 tile of W2, one of W1, one of the rest
    for (int q = 0; q < ns; ++q) {
      const float a0 = d2[q * EP_LD + hi], a1 = d2[q * EP_LD + hi + 16];
      const float c0 = h1[q * EP_LD + lo], c1 = h1[q * EP_LD + lo + 16];
      gw2[0] = fmaf(a0, c0, gw2[0]);
      gw2[1] = fmaf(a0, c1, gw2[1]);
      gw2[2] = fmaf(a1, c0, gw2[2]);
      gw2[3] = fmaf(a1, c1, gw2[3]);
      gw1 = fmaf(d1[q * EP_LD + s8], x[q * MLP_F + q8], gw1);
    }
    if (t < 32) {
      for (int q = 0; q < ns; ++q) gb += d1[q * EP_LD + t];
    } else if (t < 64) {
      for (int q = 0; q < ns; ++q) gb += d2[q * EP_LD + t - 32];
    } else if (t < 96) {
      for (int q = 0; q < ns; ++q) gb = fmaf(dy[q], h2[q * EP_LD + t - 64], gb);
    } else if (t == 96) {
      for (int q = 0; q < ns; ++q) gb += dy[q];
    }
    if (cur.last(a)) {
      grad[OFF_W2 + hi * MLP_H + lo] = gw2[0];
      grad[OFF_W2 + hi * MLP_H + lo + 16] = gw2[1];
      grad[OFF_W2 + (hi + 16) * MLP_H + lo] = gw2[2];
      grad[OFF_W2 + (hi + 16) * MLP_H + lo + 16] = gw2[3];
      grad[OFF_W1 + t] = gw1;
      if (t < 32) grad[OFF_B1 + t] = gb;
      else if (t < 64) grad[OFF_B2 + t - 32] = gb;
      else if (t < 96) grad[OFF_W3 + t - 64] = gb;
      else if (t == 96) grad[OFF_B3] = gb;
      cl.sync();
      if (owner) {
        float g = 0.f;
#pragma unroll
        for (int c = 0; c < EP_CTAS; ++c) g += *cl.map_shared_rank(grad + mine, c);
        const float2 bc = a.bias[step];
        pm = a.b1 * pm + (1.f - a.b1) * g;
        pv = a.b2 * pv + (1.f - a.b2) * g * g;
        pp -= a.lr * (pm / bc.x) / (sqrtf(pv / bc.y) + a.eps);
        float* h = home(mine);
#pragma unroll
        for (int c = 0; c < EP_CTAS; ++c) *cl.map_shared_rank(h, c) = pp;
      }
      ++step;
      cl.sync();
    } else {
      __syncthreads();  // x, h1, ... are rewritten by the next tile
    }
    cur.next(a);
  }
  if (owner) {
    a.P[mine] = pp;
    a.M[mine] = pm;
    a.V[mine] = pv;
  }
  for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  if ((t & 31) == 0 && loss != 0.f) atomicAdd(a.loss_sum, loss);
}

// Blocks of the epoch kernel's cluster: 16 (beyond the portable eight, half a tile each at 256
// samples) where the device can place them, else 8.
static int epoch_ctas(int dev) {
  static std::atomic<int> known[LAUNCH_CACHE_DEVICES];
  int c = dev >= 0 && dev < LAUNCH_CACHE_DEVICES ? known[dev].load() : 0;
  if (c) return c;
  c = 8;
  auto kern = mlp_epoch_kernel<16>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cfg.gridDim = 16;
    cfg.blockDim = EP_THREADS;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 16;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1) c = 16;
  }
  cudaGetLastError();
  if (dev >= 0 && dev < LAUNCH_CACHE_DEVICES) known[dev].store(c);
  return c;
}

static int pred_device(int* dev) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    return fail(DM_ENODEVICE, "no usable CUDA device");
  }
  DM_CUDA(cudaGetDevice(dev));
  return DM_OK;
}

// Batagelj-Zaversnik core decomposition, O(m).
static std::vector<int32_t> core_numbers(const dm_graph* g) {
  const int32_t n = g->n;
  std::vector<int32_t> deg(n), bin(g->max_degree + 2, 0), pos(n), vert(n);
  for (int32_t v = 0; v < n; ++v) {
    deg[v] = (int32_t)(g->row[v + 1] - g->row[v]);
    bin[deg[v]]++;
  }
  int32_t start = 0;
  for (int d = 0; d <= g->max_degree; ++d) {
    const int32_t num = bin[d];
    bin[d] = start;
    start += num;
  }
  for (int32_t v = 0; v < n; ++v) {
    pos[v] = bin[deg[v]];
    vert[pos[v]] = v;
    bin[deg[v]]++;
  }
  for (int d = g->max_degree; d >= 1; --d) bin[d] = bin[d - 1];
  bin[0] = 0;
  for (int32_t i = 0; i < n; ++i) {
    const int32_t v = vert[i];
    for (int64_t e = g->row[v]; e < g->row[v + 1]; ++e) {
      const int32_t u = g->adj[e];
      if (deg[u] > deg[v]) {
        const int32_t du = deg[u], pu = pos[u], pw = bin[du], w = vert[pw];
        if (u != w) {
          pos[u] = pw;
          vert[pu] = w;
          pos[w] = pu;
          vert[pw] = u;
        }
        bin[du]++;
        deg[u]--;
      }
    }
  }
  return deg;
}

constexpr int BASE_F = 6;  // f0 f1 f2 f5 f6 f7 per vertex; f3, f4 depend on k only

// Caches the k-independent features of every vertex. Counts triangles with the clique
// engine, so it must be called without the graph's mutex held.
int ensure_features(dm_graph* g, bool clique) {
  {
    std::lock_guard<std::mutex> lk(g->mu);
    ensure_oriented(g);
    if (!g->feat[clique ? 1 : 0].empty()) return DM_OK;
  }
  const int32_t n = g->n;
  std::vector<int32_t> core = core_numbers(g);
  // triangles per lowest-ranked vertex, counted by the clique engine (k = 3 subtree log)
  std::vector<uint64_t> tri(n, 0);
  {
    dm_opts o{};
    o.struct_size = sizeof(dm_opts);
    o.device = -1;
    o.subtree_counts = tri.data();
    uint64_t total = 0;
    int rc = dm_count_cliques(g, 3, &o, &total, nullptr);
    if (rc) return rc;
  }
  std::vector<float> F((size_t)n * BASE_F, 0.f);
  for (int32_t v = 0; v < n; ++v) {
    const int32_t deg = (int32_t)(g->row[v + 1] - g->row[v]);
    const int32_t r = g->rank[v];
    const int32_t outd = (int32_t)(g->orow[r + 1] - g->orow[r]);
    int32_t c0 = 0;
    double hop2 = 0;
    if (clique) {
      // C_0 = out-neighbours in the DAG; 2-hop size = their out-degrees
      c0 = outd;
      for (int64_t e = g->orow[r]; e < g->orow[r + 1]; ++e) {
        const int32_t ur = g->oadj[e];
        hop2 += (double)(g->orow[ur + 1] - g->orow[ur]);
      }
    } else {
      // C_0 = neighbours above v; 2-hop size = their degrees
      const int32_t* b = g->adj.data() + g->row[v];
      const int32_t* e = g->adj.data() + g->row[v + 1];
      const int32_t* s = std::upper_bound(b, e, v);
      c0 = (int32_t)(e - s);
      for (const int32_t* p = s; p < e; ++p) hop2 += (double)(g->row[*p + 1] - g->row[*p]);
    }
    float* x = F.data() + (size_t)v * BASE_F;
    x[0] = std::log1p((float)deg);
    x[1] = std::log1p((float)core[v]);
    x[2] = std::log1p((float)c0);
    x[3] = std::log1p((float)outd);
    x[4] = std::log1p((float)hop2);
    x[5] = std::log1p((float)tri[v]);
  }
  std::lock_guard<std::mutex> lk(g->mu);
  g->feat[clique ? 1 : 0].swap(F);
  return DM_OK;
}

// Full 8-feature row of vertex v for a k query from the cached base features.
static void feature_row(const dm_graph* g, bool clique, int k, int32_t v, float* x) {
  const float* b = g->feat[clique ? 1 : 0].data() + (size_t)v * BASE_F;
  x[0] = b[0];
  x[1] = b[1];
  x[2] = b[2];
  x[3] = k / 8.f;
  x[4] = (k - 2) / 8.f;
  x[5] = b[3];
  x[6] = b[4];
  x[7] = b[5];
}

static uint64_t g_pred_seed_mix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Runs inference for n feature rows on the current device.
static int predict_rows(const dm_predictor* p, const float* X, int64_t n, float* y) {
  if (n == 0) return DM_OK;
  float *dP = nullptr, *dX = nullptr, *dY = nullptr;
  DM_CUDA(cudaMalloc(&dP, sizeof(float) * MLP_NP));
  DM_CUDA(cudaMalloc(&dX, sizeof(float) * n * MLP_F));
  DM_CUDA(cudaMalloc(&dY, sizeof(float) * n));
  cudaMemcpy(dP, p->params.data(), sizeof(float) * MLP_NP, cudaMemcpyHostToDevice);
  cudaMemcpy(dX, X, sizeof(float) * n * MLP_F, cudaMemcpyHostToDevice);
  mlp_forward_kernel<<<(unsigned)((n + 255) / 256), 256>>>(dP, dX, (int)n, dY);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(y, dY, sizeof(float) * n, cudaMemcpyDeviceToHost);
  cudaFree(dP);
  cudaFree(dX);
  cudaFree(dY);
  if (e != cudaSuccess) return fail(DM_ECUDA, std::string("predictor inference failed: ") + cudaGetErrorString(e));
  return DM_OK;
}

// ---------------- the learned schedule on the device ----------------
//
// For the n_in root entries of a launch (the plain order, or one shard of it): the feature
// row of each root is assembled from the cached per-vertex base features, the MLP predicts
// log(1 + subtree size), and
//   cost = expm1(prediction) and a descending log-cost bucket (1/64 per bucket);
//   P = parts of the root: 1, or min(64, ceil(4 cost / share)) when the cost exceeds one
//       warp's share (total cost / warps);
//   the entries are written longest-first by a counting sort over the buckets (order inside
//   a bucket is arbitrary), each root as P consecutive entries (p | P << 16), flagged
//   PART_EAGER when its predicted cost is above EAGER_SHARE x share, so that the counting
//   kernel donates from it without waiting for the minimum task age.
// No allocation per call: the scratch lives in the caller's workspace.
constexpr int SCHED_BINS = 2048;
constexpr float EAGER_SHARE = 0.25f;

struct SchedArgs {
  const float* feat;        // n x BASE_F base features by original id
  const float* params;      // MLP_NP
  const int32_t* roots;     // n_in entries: rank space (cliques) or vertex ids (motifs)
  const int32_t* orig;      // rank -> original id (cliques), else null
  int n_in, k, warps, cap;
  float* cost;              // n_in
  int* bin;                 // n_in
  int* nparts;              // n_in
  double* total;            // 1
  unsigned* bins;           // SCHED_BINS
  int* n_out;               // 1
  int* err;                 // 1 (set when the output capacity would be exceeded)
  int32_t* out_roots;       // cap
  int32_t* out_parts;       // cap
  RootDesc* out_desc;       // cap, or null (cliques on the index)
  const int32_t* odeg;      // rank-space out-degrees (out_desc)
  const uint32_t* boff;     // index block offsets (out_desc)
};

__global__ void __launch_bounds__(256) sched_predict_kernel(SchedArgs a) {
  __shared__ float sp[MLP_NP];
  __shared__ double red[8];
  for (int i = threadIdx.x; i < MLP_NP; i += blockDim.x) sp[i] = a.params[i];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double c = 0.0;
  if (i < a.n_in) {
    const int32_t r = a.roots[i];
    const int32_t v = a.orig ? a.orig[r] : r;
    const float* b = a.feat + (size_t)v * BASE_F;
    const float x[MLP_F] = {b[0], b[1], b[2], a.k / 8.f, (a.k - 2) / 8.f, b[3], b[4], b[5]};
    const float y = fminf(fmaxf(mlp_eval(sp, x), 0.f), 40.f);
    c = (double)expm1f(y);
    a.cost[i] = (float)c;
    a.bin[i] = SCHED_BINS - 1 - min(SCHED_BINS - 1, (int)(y * 64.f));
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    atomicAdd(a.total, t);
  }
}

__global__ void __launch_bounds__(256) sched_parts_kernel(SchedArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n_in) return;
  const double share = *a.total / (double)max(1, a.warps);
  const double c = (double)a.cost[i];
  int P = 1;
  if (share > 0 && c > share) P = (int)fmin(64.0, ceil(4.0 * c / share));
  a.nparts[i] = P;
  atomicAdd(a.bins + a.bin[i], (unsigned)P);
}

// Exclusive scan of the bucket counts (one block of 1024 threads, two buckets per thread).
__global__ void __launch_bounds__(1024) sched_scan_kernel(SchedArgs a) {
  __shared__ unsigned part[1024];
  const int t = threadIdx.x;
  const unsigned c0 = a.bins[2 * t], c1 = a.bins[2 * t + 1];
  part[t] = c0 + c1;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const unsigned y = t >= o ? part[t - o] : 0u;
    __syncthreads();
    part[t] += y;
    __syncthreads();
  }
  const unsigned excl = part[t] - (c0 + c1);
  a.bins[2 * t] = excl;
  a.bins[2 * t + 1] = excl + c0;
  if (t == 1023) *a.n_out = (int)part[t];
}

__global__ void __launch_bounds__(256) sched_scatter_kernel(SchedArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n_in) return;
  const int P = a.nparts[i];
  const unsigned pos = atomicAdd(a.bins + a.bin[i], (unsigned)P);
  if ((long long)pos + P > a.cap) {
    atomicExch(a.err, 1);
    return;
  }
  const int32_t r = a.roots[i];
  const double share = *a.total / (double)max(1, a.warps);
  const int eager = share > 0 && (double)a.cost[i] > EAGER_SHARE * share ? PART_EAGER : 0;
  for (int q = 0; q < P; ++q) {
    const int32_t pw = (P > 1 ? (q | (P << 16)) : 0) | eager;
    a.out_roots[pos + q] = r;
    a.out_parts[pos + q] = pw;
    if (a.out_desc) a.out_desc[pos + q] = RootDesc{r, a.odeg[r], a.boff ? a.boff[r] : INDEX_NONE, pw};
  }
}

// Runs the schedule of `in` (device root entries) on ctx.stream into the scratch `w`, and
// returns the number of output entries (a 4-byte read-back). Output capacity: n_in + 4 x
// warps + 64 entries (the parts of the roots above one share sum to at most 4 x warps +
// their count).
int learned_schedule_device(const void* pv, const SchedIO& io, LaunchCtx& ctx, int* n_out) {
  const dm_predictor* p = reinterpret_cast<const dm_predictor*>(pv);
  SchedArgs a;
  a.feat = io.feat;
  a.params = io.params;
  a.roots = io.roots;
  a.orig = io.orig;
  a.n_in = io.n_in;
  a.k = io.k;
  a.warps = io.warps;
  a.cap = io.cap;
  char* w = reinterpret_cast<char*>(io.scratch);
  auto take = [&](size_t bytes) {
    char* q = w;
    w += (bytes + 255) / 256 * 256;
    return q;
  };
  a.total = reinterpret_cast<double*>(take(sizeof(double)));
  a.n_out = reinterpret_cast<int*>(take(sizeof(int)));
  a.err = reinterpret_cast<int*>(take(sizeof(int)));
  a.bins = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * SCHED_BINS));
  a.cost = reinterpret_cast<float*>(take(sizeof(float) * std::max(io.n_in, 1)));
  a.bin = reinterpret_cast<int*>(take(sizeof(int) * std::max(io.n_in, 1)));
  a.nparts = reinterpret_cast<int*>(take(sizeof(int) * std::max(io.n_in, 1)));
  a.out_roots = io.out_roots;
  a.out_parts = io.out_parts;
  a.out_desc = io.out_desc;
  a.odeg = io.odeg;
  a.boff = io.boff;
  // the scratch header (total, n_out, err, bins) starts at zero
  DM_CUDA(cudaMemsetAsync(io.scratch, 0, (size_t)(reinterpret_cast<char*>(a.cost) - reinterpret_cast<char*>(io.scratch)),
                          ctx.stream));
  if (!io.params_current)
    DM_CUDA(cudaMemcpyAsync(io.params, p->params.data(), sizeof(float) * MLP_NP, cudaMemcpyHostToDevice,
                            ctx.stream));
  const unsigned grid = (unsigned)std::max(1, (io.n_in + 255) / 256);
  sched_predict_kernel<<<grid, 256, 0, ctx.stream>>>(a);
  sched_parts_kernel<<<grid, 256, 0, ctx.stream>>>(a);
  sched_scan_kernel<<<1, 1024, 0, ctx.stream>>>(a);
  sched_scatter_kernel<<<grid, 256, 0, ctx.stream>>>(a);
  ctx.launches += 4;
  DM_CUDA(cudaGetLastError());
  // the task count and the error flag, through a page-locked pair (asynchronous copies)
  int* hdr = io.h_hdr;
  DM_CUDA(cudaMemcpyAsync(&hdr[0], a.n_out, sizeof(int), cudaMemcpyDeviceToHost, ctx.stream));
  DM_CUDA(cudaMemcpyAsync(&hdr[1], a.err, sizeof(int), cudaMemcpyDeviceToHost, ctx.stream));
  DM_CUDA(cudaStreamSynchronize(ctx.stream));
  if (hdr[1]) return fail(DM_EINTERNAL, "learned schedule exceeded its output capacity");
  *n_out = hdr[0];
  return DM_OK;
}

int predictor_num_params() { return MLP_NP; }

size_t learned_schedule_scratch_bytes(int n_in) {
  const size_t n = (size_t)std::max(n_in, 1);
  return 4 * 256 + (sizeof(unsigned) * SCHED_BINS + 255) / 256 * 256 + 3 * ((n * 4 + 255) / 256 * 256);
}

// Host version of the same schedule, for planning (dm_plan_roots): same costs, parts and
// flags, with ties inside a bucket in input order.
int predictor_schedule(const void* pv, dm_graph* g, int k, bool clique, int total_warps, std::vector<int32_t>& roots,
                       std::vector<int32_t>& parts) {
  const dm_predictor* p = reinterpret_cast<const dm_predictor*>(pv);
  if (g->feat[clique ? 1 : 0].empty()) return fail(DM_EINVAL, "predictor features were not prepared");
  int rc = DM_OK;
  // features are per original vertex; clique roots arrive in rank space
  std::vector<int32_t> orig(roots.size());
  if (clique) {
    std::vector<int32_t> inv(g->n);
    for (int32_t v = 0; v < g->n; ++v) inv[g->rank[v]] = v;
    for (size_t i = 0; i < roots.size(); ++i) orig[i] = inv[roots[i]];
  } else {
    orig = roots;
  }
  std::vector<float> Xr(roots.size() * MLP_F);
  for (size_t i = 0; i < roots.size(); ++i) feature_row(g, clique, k, orig[i], Xr.data() + i * MLP_F);
  std::vector<float> pred(roots.size());
  if ((rc = predict_rows(p, Xr.data(), (int64_t)roots.size(), pred.data()))) return rc;
  std::vector<double> cost(roots.size());
  std::vector<int> bin(roots.size());
  double total = 0;
  for (size_t i = 0; i < roots.size(); ++i) {
    const float y = std::min(std::max(pred[i], 0.f), 40.f);
    cost[i] = (double)std::expm1(y);
    bin[i] = SCHED_BINS - 1 - std::min(SCHED_BINS - 1, (int)(y * 64.f));
    total += cost[i];
  }
  std::vector<size_t> order(roots.size());
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return bin[a] < bin[b]; });
  const double share = total / std::max(1, total_warps);
  std::vector<int32_t> out_roots, out_parts;
  out_roots.reserve(roots.size());
  out_parts.reserve(roots.size());
  for (size_t i : order) {
    int P = 1;
    if (share > 0 && cost[i] > share) P = (int)std::min<double>(64.0, std::ceil(4.0 * cost[i] / share));
    const int eager = share > 0 && cost[i] > EAGER_SHARE * share ? PART_EAGER : 0;
    for (int q = 0; q < P; ++q) {
      out_roots.push_back(roots[i]);
      out_parts.push_back((P > 1 ? (q | (P << 16)) : 0) | eager);
    }
  }
  roots.swap(out_roots);
  parts.swap(out_parts);
  return DM_OK;
}

}  // namespace dmb

using namespace dmb;

extern "C" {

int dm_predictor_create(uint64_t seed, dm_predictor** out) {
  if (!out) return fail(DM_EINVAL, "dm_predictor_create: null argument");
  auto* p = new dm_predictor();
  p->uid = g_pred_uid++;
  p->seed = seed;
  p->params.assign(MLP_NP, 0.f);
  // He-uniform initialisation from a splitmix stream
  uint64_t s = seed;
  auto uni = [&]() {
    s = g_pred_seed_mix(s);
    return (float)((s >> 11) * (1.0 / 9007199254740992.0)) * 2.f - 1.f;
  };
  const float a1 = std::sqrt(6.f / MLP_F), a2 = std::sqrt(6.f / MLP_H);
  for (int i = 0; i < MLP_H * MLP_F; ++i) p->params[OFF_W1 + i] = a1 * uni();
  for (int i = 0; i < MLP_H * MLP_H; ++i) p->params[OFF_W2 + i] = a2 * uni();
  for (int i = 0; i < MLP_H; ++i) p->params[OFF_W3 + i] = a2 * uni() * 0.5f;
  for (int i = 0; i < MLP_H; ++i) p->params[OFF_B1 + i] = 0.01f;
  for (int i = 0; i < MLP_H; ++i) p->params[OFF_B2 + i] = 0.01f;
  p->adam_m.assign(MLP_NP, 0.f);
  p->adam_v.assign(MLP_NP, 0.f);
  *out = p;
  return DM_OK;
}

void dm_predictor_free(dm_predictor* p) { delete p; }

int dm_predictor_num_params(void) { return MLP_NP; }

int dm_predictor_get_params(const dm_predictor* p, float* params) {
  if (!p || !params) return fail(DM_EINVAL, "dm_predictor_get_params: null argument");
  std::memcpy(params, p->params.data(), sizeof(float) * MLP_NP);
  return DM_OK;
}

int dm_predictor_set_params(dm_predictor* p, const float* params) {
  if (!p || !params) return fail(DM_EINVAL, "dm_predictor_set_params: null argument");
  std::memcpy(p->params.data(), params, sizeof(float) * MLP_NP);
  ++p->version;
  return DM_OK;
}

int dm_predictor_features(dm_graph* g, int32_t k, int32_t clique, float* features) {
  if (!g || !features) return fail(DM_EINVAL, "dm_predictor_features: null argument");
  if (k < 2 || k > 12) return fail(DM_EINVAL, "dm_predictor_features: k out of range");
  int rc = ensure_features(g, clique != 0);
  if (rc) return rc;
  for (int32_t v = 0; v < g->n; ++v) feature_row(g, clique != 0, k, v, features + (size_t)v * MLP_F);
  return DM_OK;
}

int dm_predictor_predict(const dm_predictor* p, const float* X, int64_t n, float* y) {
  if (!p || (n && (!X || !y)) || n < 0) return fail(DM_EINVAL, "dm_predictor_predict: bad arguments");
  int dev = 0;
  int rc = pred_device(&dev);
  if (rc) return rc;
  return predict_rows(p, X, n, y);
}

// One full-batch gradient of the mean squared error (for checking against a CPU model).
int dm_predictor_gradients(const dm_predictor* p, const float* X, const float* T, int64_t n, float* grad,
                           float* loss) {
  if (!p || !X || !T || !grad || n <= 0) return fail(DM_EINVAL, "dm_predictor_gradients: bad arguments");
  int dev = 0;
  int rc = pred_device(&dev);
  if (rc) return rc;
  float *dP, *dX, *dT, *dG, *dL;
  DM_CUDA(cudaMalloc(&dP, sizeof(float) * MLP_NP));
  DM_CUDA(cudaMalloc(&dX, sizeof(float) * n * MLP_F));
  DM_CUDA(cudaMalloc(&dT, sizeof(float) * n));
  DM_CUDA(cudaMalloc(&dG, sizeof(float) * MLP_NP));
  DM_CUDA(cudaMalloc(&dL, sizeof(float)));
  cudaMemcpy(dP, p->params.data(), sizeof(float) * MLP_NP, cudaMemcpyHostToDevice);
  cudaMemcpy(dX, X, sizeof(float) * n * MLP_F, cudaMemcpyHostToDevice);
  cudaMemcpy(dT, T, sizeof(float) * n, cudaMemcpyHostToDevice);
  cudaMemset(dG, 0, sizeof(float) * MLP_NP);
  cudaMemset(dL, 0, sizeof(float));
  cudaFuncSetAttribute(mlp_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BACKWARD_SMEM);
  mlp_backward_kernel<<<(unsigned)((n + TB - 1) / TB), TB, BACKWARD_SMEM>>>(dP, dX, dT, nullptr, (int)n,
                                                                          1.f / (float)n, dG, dL);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(grad, dG, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost);
  float ls = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&ls, dL, sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(dP);
  cudaFree(dX);
  cudaFree(dT);
  cudaFree(dG);
  cudaFree(dL);
  if (e != cudaSuccess) return fail(DM_ECUDA, std::string("predictor gradients failed: ") + cudaGetErrorString(e));
  if (loss) *loss = ls / (float)n;
  return DM_OK;
}

// Adam on minibatches for `epochs` passes over (X, T); writes the final epoch's mean loss.
int dm_predictor_train(dm_predictor* p, const float* X, const float* T, int64_t n, int32_t epochs, int32_t batch,
                       float lr, float* final_loss) {
  if (!p || !X || !T || n <= 0 || epochs <= 0 || batch <= 0 || !(lr > 0))
    return fail(DM_EINVAL, "dm_predictor_train: bad arguments");
  int dev = 0;
  int rc = pred_device(&dev);
  if (rc) return rc;
  // one buffer from the library's pool: P, M, V, gradient, loss | X | T | two index buffers | bias
  const bool fused = batch <= EP_BATCH_MAX;
  const int ctas = fused ? epoch_ctas(dev) : 0;
  const int64_t steps = (n + batch - 1) / batch;
  const size_t pad = 64;  // floats: every part starts on 256 bytes
  auto room = [&](size_t floats) { return (floats + pad - 1) / pad * pad; };
  const size_t np = room(MLP_NP), nx = room((size_t)n * MLP_F), nt = room((size_t)n), nb = room(2 * (size_t)steps);
  float* buf = nullptr;
  DM_CUDA(gbuf_alloc(reinterpret_cast<void**>(&buf), sizeof(float) * (4 * np + pad + nx + 3 * nt + 2 * nb)));
  float *dP = buf, *dM = dP + np, *dV = dM + np, *dG = dV + np, *dL = dG + np, *dX = dL + pad, *dT = dX + nx;
  int* dIdx[2] = {reinterpret_cast<int*>(dT + nt), reinterpret_cast<int*>(dT + 2 * nt)};
  float* dBias[2] = {dT + 3 * nt, dT + 3 * nt + nb};
  cudaMemcpyAsync(dP, p->params.data(), sizeof(float) * MLP_NP, cudaMemcpyHostToDevice);
  cudaMemcpyAsync(dM, p->adam_m.data(), sizeof(float) * MLP_NP, cudaMemcpyHostToDevice);
  cudaMemcpyAsync(dV, p->adam_v.data(), sizeof(float) * MLP_NP, cudaMemcpyHostToDevice);
  cudaMemcpyAsync(dX, X, sizeof(float) * n * MLP_F, cudaMemcpyHostToDevice);
  cudaMemcpyAsync(dT, T, sizeof(float) * n, cudaMemcpyHostToDevice);
  cudaFuncSetAttribute(mlp_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BACKWARD_SMEM);
  std::vector<int> idx(n);
  std::iota(idx.begin(), idx.end(), 0);
  uint64_t s = p->seed ^ 0x5DEECE66Dull;
  const float b1 = 0.9f, b2 = 0.999f;
  std::vector<float> bias(2 * (size_t)steps);
  for (int ep = 0; ep < epochs; ++ep) {
    // (while the device still runs the previous epoch, whose indices are in the other device buffer. idx
    // and bias may change: a copy from pageable memory returns once it has left for the driver's own
    // staging memory. Page-locked buffers of ours with an event each made the host wait for the epoch
    // before: 300 rows, 4 epochs 132 -> 196 us.)
    for (int64_t i = n - 1; i > 0; --i) {
      s = g_pred_seed_mix(s);
      std::swap(idx[i], idx[s % (uint64_t)(i + 1)]);
    }
    for (int64_t q = 0; q < steps; ++q) {
      ++p->steps;
      bias[2 * q] = 1.f - std::pow(b1, (float)p->steps);
      bias[2 * q + 1] = 1.f - std::pow(b2, (float)p->steps);
    }
    int* di = dIdx[ep & 1];
    cudaMemcpyAsync(di, idx.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
    cudaMemsetAsync(dL, 0, sizeof(float));
    if (fused) {
      float* db = dBias[ep & 1];
      cudaMemcpyAsync(db, bias.data(), sizeof(float) * bias.size(), cudaMemcpyHostToDevice);
      const EpochArgs a{dP, dM, dV, dX, dT, di, reinterpret_cast<const float2*>(db), dL, (int)n, batch, lr, b1, b2, 1e-8f};
      if (ctas == 16) mlp_epoch_kernel<16><<<16, EP_THREADS>>>(a);
      else mlp_epoch_kernel<8><<<8, EP_THREADS>>>(a);
    } else {
      for (int64_t q = 0; q < steps; ++q) {
        const int64_t off = q * batch;
        const int bn = (int)std::min<int64_t>(batch, n - off);
        cudaMemsetAsync(dG, 0, sizeof(float) * MLP_NP);
        mlp_backward_kernel<<<(bn + TB - 1) / TB, TB, BACKWARD_SMEM>>>(dP, dX, dT, di + off, bn, 1.f / (float)bn, dG, dL);
        adam_kernel<<<(MLP_NP + 255) / 256, 256>>>(dP, dG, dM, dV, lr, b1, b2, 1e-8f, bias[2 * q], bias[2 * q + 1]);
      }
    }
  }
  cudaError_t e = cudaGetLastError();
  float ls = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&ls, dL, sizeof(float), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpyAsync(p->params.data(), dP, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpyAsync(p->adam_m.data(), dM, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpyAsync(p->adam_v.data(), dV, sizeof(float) * MLP_NP, cudaMemcpyDeviceToHost);
  const cudaError_t es = cudaStreamSynchronize(nullptr);  // before the buffer goes back to the pool
  if (e == cudaSuccess) e = es;
  ++p->version;
  gbuf_free(buf, dev);
  if (e != cudaSuccess) return fail(DM_ECUDA, std::string("predictor training failed: ") + cudaGetErrorString(e));
  if (final_loss) *final_loss = (float)((double)ls / (double)n);
  return DM_OK;
}

}  // extern "C"
