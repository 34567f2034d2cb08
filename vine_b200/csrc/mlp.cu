// Learned bucket scheduler: a 16-64-64-2 ReLU MLP in FP32, trained on the
// GPU by the kernels below (forward, backward, Adam).  The reference chooses
// its bucket width only through the AR model (algorithm/cspp.cuh:254-284);
// the network augments that policy.  It only changes how work is ordered, so
// exactness never depends on it (its outputs are clamped and a non-finite
// output falls back to the AR rule inside the search kernel).
//
// The contraction is 5.3 kFLOP per row in FP32 (the tensor cores have no FP32
// inputs, and the weights and sums stay in 32 bits): the kernels run it as
// register-tiled matrix products over 64-row tiles (mlp_tile).  Training
// batches run in one launch an epoch on a cluster of eight CTAs that
// exchange gradients and parameters through distributed shared memory.

#include "engine_host.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <random>
#include <string>
#include <vector>

namespace vine {
namespace {

constexpr int kTile = 64;       // rows of a tile
constexpr int kThreads = 256;   // 16 x 16 threads, 4 x 4 outputs each
constexpr int kPitch = kTile + 4;  // row pitch: 16-byte aligned, columns spread over the banks
constexpr int kXPitch = kFeat + 4;
constexpr int kWPitch = kHid + 4;  // transposed writes then meet 8 banks, not one
constexpr int kW1 = 0, kB1 = kW1 + kHid * kFeat, kW2 = kB1 + kHid, kB2 = kW2 + kHid * kHid,
              kW3 = kB2 + kHid, kB3 = kW3 + kOut * kHid;
static_assert(kHid == 64 && kThreads == 256, "the 16 x 16 thread grid covers 64 x 64 outputs");

// Shared memory of a tile.  Weights lie so that every inner loop reads four
// neighbouring values of the output dimension; activations are kept by
// column (operand of the next product) and by row (operand of the gradients).
struct __align__(16) MlpShared {
  float w1t[kFeat * kWPitch];  // [i][j] = W1[j][i]
  float w2t[kHid * kWPitch];   // [i][j] = W2[j][i]
  float w2[kHid * kWPitch];    // [j][i]
  float w3[kOut * kHid];
  float b1[kHid], b2[kHid], b3[4];
  float xt[kFeat * kPitch];    // inputs by column
  float xr[kTile * kXPitch];   // inputs by row
  float ct[kHid * kPitch];     // layer 1 by column, then the layer-2 gradients
  float r1[kTile * kPitch];    // layer 1 by row, then its gradients
  float r2[kTile * kPitch];    // layer-2 gradients by row
};

// Parameter p of the flat layout, into its place(s).
__device__ __forceinline__ void put_param(MlpShared &S, int p, float v) {
  if (p < kB1) {
    S.w1t[(p % kFeat) * kWPitch + p / kFeat] = v;
  } else if (p < kW2) {
    S.b1[p - kB1] = v;
  } else if (p < kB2) {
    const int q = p - kW2;
    S.w2[(q / kHid) * kWPitch + q % kHid] = v;
    S.w2t[(q % kHid) * kWPitch + q / kHid] = v;
  } else if (p < kW3) {
    S.b2[p - kB2] = v;
  } else if (p < kB3) {
    S.w3[p - kW3] = v;
  } else {
    S.b3[p - kB3] = v;
  }
}

// A thread's share of the gradient, summed over tiles: W2 block (rows
// 4 ty.., columns 4 tx..), four W1 entries (row tid / 4), and its rows'
// contributions to W3 and the biases (summed over ty at the end).
struct MlpGrad {
  float w2[4][4], w1[4], w3[kOut][4], b1[4], b2[4], b3[kOut];
};

// acc[r][c] += sum over k of a[k][4 ty + r] * b[k][4 tx + c]
template <int K, int kPitchA>
__device__ __forceinline__ void tile_product(const float *a, const float *b, int ty, int tx, float (&acc)[4][4]) {
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    const float4 x = *reinterpret_cast<const float4 *>(a + k * kPitchA + 4 * ty);
    const float4 y = *reinterpret_cast<const float4 *>(b + k * kWPitch + 4 * tx);
    const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(xs[r], ys[c], acc[r][c]);
  }
}

// What a thread brings into a tile: a quarter row of inputs and the targets of
// its four rows (the same for all 16 tx).  Loaded apart from the tile's work,
// so that a caller can have the next tile's reads in flight.
struct TileIn {
  float4 x;
  float2 t[4];
};

// Row r of the tile is row idx[r0 + r] (or r0 + r) of X and T; rows <= 64.
__device__ __forceinline__ void load_tile(TileIn &in, const float *__restrict__ X, const float *__restrict__ T,
                                          const int32_t *__restrict__ idx, int r0, int rows) {
  const int tid = threadIdx.x, r = tid >> 2, q = (tid & 3) * 4;
  in.x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (r < rows) in.x = *reinterpret_cast<const float4 *>(X + (size_t)(idx ? idx[r0 + r] : r0 + r) * kFeat + q);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int row = 4 * (tid >> 4) + k;
    in.t[k] = make_float2(0.0f, 0.0f);
    if (T && row < rows)
      in.t[k] = *reinterpret_cast<const float2 *>(T + (size_t)(idx ? idx[r0 + row] : r0 + row) * kOut);
  }
}

// Forward (and with kBackward the gradients) of a loaded tile of `rows` <= 64
// rows whose outputs are rows r0.. of Y.  All threads call.
//
// Bound by FP32 multiply-adds with two 16-byte shared reads for 16 of them.
// The former kernel read the weights with a stride of 64 words between the
// lanes, a 32-way bank conflict an operand.  65,536 rows with gradients: 86 us
// (24 TFLOP/s), 100,000 rows forward: 49 us.
template <bool kBackward>
__device__ __forceinline__ void mlp_tile(MlpShared &S, MlpGrad &g, const TileIn &in, bool targets, int r0,
                                         int rows, float inv_norm, float *Y, float &loss) {
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  {
    const int r = tid >> 2, q = (tid & 3) * 4;  // a quarter row a thread
    S.xt[(q + 0) * kPitch + r] = in.x.x;
    S.xt[(q + 1) * kPitch + r] = in.x.y;
    S.xt[(q + 2) * kPitch + r] = in.x.z;
    S.xt[(q + 3) * kPitch + r] = in.x.w;
    if (kBackward) *reinterpret_cast<float4 *>(S.xr + r * kXPitch + q) = in.x;
  }
  __syncthreads();
  float h1[4][4], h2[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      h1[r][c] = S.b1[4 * tx + c];
      h2[r][c] = S.b2[4 * tx + c];
    }
  tile_product<kFeat, kPitch>(S.xt, S.w1t, ty, tx, h1);
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) h1[r][c] = fmaxf(h1[r][c], 0.0f);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<float4 *>(S.ct + (4 * tx + c) * kPitch + 4 * ty) =
        make_float4(h1[0][c], h1[1][c], h1[2][c], h1[3][c]);
  if (kBackward)
#pragma unroll
    for (int r = 0; r < 4; ++r)
      *reinterpret_cast<float4 *>(S.r1 + (4 * ty + r) * kPitch + 4 * tx) =
          make_float4(h1[r][0], h1[r][1], h1[r][2], h1[r][3]);
  __syncthreads();
  tile_product<kHid, kPitch>(S.ct, S.w2t, ty, tx, h2);
  float dy[4][kOut];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
#pragma unroll
    for (int k = 0; k < kOut; ++k) {
      float p = 0.0f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (k == 0) h2[r][c] = fmaxf(h2[r][c], 0.0f);
        p = fmaf(h2[r][c], S.w3[k * kHid + 4 * tx + c], p);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
      const float y = p + S.b3[k];
      const int row = 4 * ty + r;
      dy[r][k] = 0.0f;
      if (row < rows) {
        if (Y && tx == 0) Y[(size_t)(r0 + row) * kOut + k] = y;
        if (targets) {
          const float e = y - (k == 0 ? in.t[r].x : in.t[r].y);
          if (tx == 0) loss += e * e;
          dy[r][k] = 2.0f * e * inv_norm;
        }
      }
    }
  }
  if (!kBackward) {
    __syncthreads();  // the tile is read before the next one is loaded
    return;
  }
  float d2[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float v = fmaf(dy[r][0], S.w3[4 * tx + c], dy[r][1] * S.w3[kHid + 4 * tx + c]);
      d2[r][c] = h2[r][c] > 0.0f ? v : 0.0f;
      g.b2[c] += d2[r][c];
      g.w3[0][c] = fmaf(dy[r][0], h2[r][c], g.w3[0][c]);
      g.w3[1][c] = fmaf(dy[r][1], h2[r][c], g.w3[1][c]);
    }
  if (tx == 0)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      g.b3[0] += dy[r][0];
      g.b3[1] += dy[r][1];
    }
  __syncthreads();  // layer 1 by column is read: the gradients take its place
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<float4 *>(S.ct + (4 * tx + c) * kPitch + 4 * ty) =
        make_float4(d2[0][c], d2[1][c], d2[2][c], d2[3][c]);
#pragma unroll
  for (int r = 0; r < 4; ++r)
    *reinterpret_cast<float4 *>(S.r2 + (4 * ty + r) * kPitch + 4 * tx) =
        make_float4(d2[r][0], d2[r][1], d2[r][2], d2[r][3]);
  __syncthreads();
  // W2 gradient [j][i]: sum over rows of d2[row][j] * h1[row][i]
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    const float4 x = *reinterpret_cast<const float4 *>(S.r2 + r * kPitch + 4 * ty);
    const float4 y = *reinterpret_cast<const float4 *>(S.r1 + r * kPitch + 4 * tx);
    const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) g.w2[a][b] = fmaf(xs[a], ys[b], g.w2[a][b]);
  }
  float d1[4][4] = {};
  tile_product<kHid, kPitch>(S.ct, S.w2, ty, tx, d1);
  __syncthreads();  // layer 1 by row is read: its gradients take its place
#pragma unroll
  for (int r = 0; r < 4; ++r) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      d1[r][c] = h1[r][c] > 0.0f ? d1[r][c] : 0.0f;
      g.b1[c] += d1[r][c];
    }
    *reinterpret_cast<float4 *>(S.r1 + (4 * ty + r) * kPitch + 4 * tx) =
        make_float4(d1[r][0], d1[r][1], d1[r][2], d1[r][3]);
  }
  __syncthreads();
  // W1 gradient: row j = tid / 4, columns 4 (tid % 4) ..
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    const float d = S.r1[r * kPitch + (tid >> 2)];
    const float4 x = *reinterpret_cast<const float4 *>(S.xr + r * kXPitch + (tid & 3) * 4);
    g.w1[0] = fmaf(d, x.x, g.w1[0]);
    g.w1[1] = fmaf(d, x.y, g.w1[1]);
    g.w1[2] = fmaf(d, x.z, g.w1[2]);
    g.w1[3] = fmaf(d, x.w, g.w1[3]);
  }
  __syncthreads();
}

// Sums what the 16 ty of a block hold of the W3 and bias gradients and hands
// every parameter's block total to `put(p, value)` once.  `sum`: 16 rows of
// kSmallPitch floats of shared memory.
constexpr int kSmallGrads = kOut * kHid + 2 * kHid + kOut;
constexpr int kSmallPitch = (kSmallGrads + 3) & ~3;
static_assert(16 * kSmallPitch <= 2 * kTile * kPitch, "the sums fit the activation buffers ct and r1");
template <typename Put>
__device__ __forceinline__ void reduce_grads(const MlpGrad &g, float *sum, Put put) {
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  float *row = sum + ty * kSmallPitch + 4 * tx;
  *reinterpret_cast<float4 *>(row) = make_float4(g.w3[0][0], g.w3[0][1], g.w3[0][2], g.w3[0][3]);
  *reinterpret_cast<float4 *>(row + kHid) = make_float4(g.w3[1][0], g.w3[1][1], g.w3[1][2], g.w3[1][3]);
  *reinterpret_cast<float4 *>(row + 2 * kHid) = make_float4(g.b1[0], g.b1[1], g.b1[2], g.b1[3]);
  *reinterpret_cast<float4 *>(row + 3 * kHid) = make_float4(g.b2[0], g.b2[1], g.b2[2], g.b2[3]);
  if (tx == 0) *reinterpret_cast<float2 *>(row + 4 * kHid) = make_float2(g.b3[0], g.b3[1]);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) put(kW2 + (4 * ty + a) * kHid + 4 * tx + b, g.w2[a][b]);
#pragma unroll
  for (int b = 0; b < 4; ++b) put(kW1 + (tid >> 2) * kFeat + (tid & 3) * 4 + b, g.w1[b]);
  __syncthreads();
  for (int i = tid; i < kSmallGrads; i += kThreads) {
    float v = 0.0f;
#pragma unroll
    for (int r = 0; r < 16; ++r) v += sum[r * kSmallPitch + i];
    const int p = i < 2 * kHid ? kW3 + i
                : i < 3 * kHid ? kB1 + i - 2 * kHid
                : i < 4 * kHid ? kB2 + i - 3 * kHid
                               : kB3 + i - 4 * kHid;
    put(p, v);
  }
}

// Forward (and optionally backward) over rows idx[0..n) (or 0..n when idx is
// null).  Loss = (1/norm) * sum over rows and outputs of (y - t)^2.
template <bool kBackward>
__global__ void __launch_bounds__(kThreads, 2) mlp_fb_kernel(const float *__restrict__ params,
                                                             const float *__restrict__ X,
                                                             const float *__restrict__ T,
                                                             const int32_t *__restrict__ idx, int n,
                                                             float inv_norm, float *grad, float *loss, float *Y) {
  extern __shared__ __align__(16) unsigned char mlp_smem[];
  MlpShared &S = *reinterpret_cast<MlpShared *>(mlp_smem);
  const int tid = threadIdx.x;
  for (int p = tid; p < kMlpParams; p += kThreads) put_param(S, p, params[p]);
  MlpGrad g = {};
  float loss_local = 0.0f;
  __syncthreads();
  const int ntiles = (n + kTile - 1) / kTile;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int r0 = tile * kTile, rows = min(kTile, n - r0);
    TileIn in;
    load_tile(in, X, T, idx, r0, rows);
    mlp_tile<kBackward>(S, g, in, T != nullptr, r0, rows, inv_norm, Y, loss_local);
  }
  if (kBackward) reduce_grads(g, S.ct, [grad](int p, float v) { atomicAdd(&grad[p], v); });
  if (loss) {  // one addition a block to the total
    for (int o = 16; o > 0; o >>= 1) loss_local += __shfl_down_sync(0xffffffffu, loss_local, o);
    float *part = S.xt;  // free after the last tile
    if ((tid & 31) == 0) part[tid >> 5] = loss_local;
    __syncthreads();
    if (tid == 0) {
      float total = 0.0f;
      for (int w = 0; w < kThreads / 32; ++w) total += part[w];
      atomicAdd(loss, total * inv_norm);
    }
  }
}

__device__ __forceinline__ void adam_step(float &p, float &m, float &v, float g, float lr, float b1, float b2,
                                          float c1, float c2, float eps) {
  m = b1 * m + (1.0f - b1) * g;
  v = b2 * v + (1.0f - b2) * g * g;
  p -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

// One epoch of mini-batch Adam on a cluster of kCluster CTAs, one launch.
// A batch's rows are dealt to the CTAs; each leaves its gradient in shared
// memory; CTA c then sums its slice of the parameters over the cluster
// (distributed shared memory) and steps it, and every CTA reads the new
// slices.  The next batch's rows are fetched meanwhile.
//
// Bound by latency: at 512 rows a batch each CTA has one tile and the cluster
// two barriers with an exchange of 21 KB each way.  Eight CTAs, the portable
// cluster size: a batch of the training recipe is eight tiles.  Measured at
// 512 rows a batch: 18 us a step, of which the tile takes 11 (a memset, a
// gradient and a step launch with the former tile took about 55).
constexpr int kCluster = 8;
constexpr int kSlice = ((kMlpParams + kCluster - 1) / kCluster + 3) & ~3;  // whole float4s
constexpr int kEpochMaxBatch = 4 * kCluster * kTile;  // above, more SMs than a cluster has pay
static_assert(kSlice / 4 <= kThreads, "one float4 of a slice a thread");

struct __align__(16) EpochShared {
  MlpShared t;
  float grad[kCluster * kSlice];
  float p[kSlice];
};

__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(kCluster, 1, 1)
mlp_epoch_kernel(float *params, float *am, float *av, const float *__restrict__ X, const float *__restrict__ T,
                 const int32_t *__restrict__ idx, int n, int batch, const float2 *__restrict__ corr, float lr,
                 float b1, float b2, float eps) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char mlp_smem[];
  EpochShared &S = *reinterpret_cast<EpochShared *>(mlp_smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, rank = (int)cluster.block_rank();
  const bool owner = tid < kSlice / 4;  // of parameters own .. own + 3
  const int own = rank * kSlice + 4 * tid;
  for (int p = tid; p < kMlpParams; p += kThreads) put_param(S.t, p, params[p]);
  for (int i = tid; i < kCluster * kSlice; i += kThreads) S.grad[i] = 0.0f;  // the padding stays 0
  float pp[4] = {}, pm[4] = {}, pv[4] = {};
  if (owner)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (own + k < kMlpParams) {
        pp[k] = params[own + k];
        pm[k] = am[own + k];
        pv[k] = av[own + k];
      }
  // rows of this CTA in the batch at b0: whole 4-row groups
  auto mine = [&](int b0, int *lo, int *hi) {
    const int nb = min(batch, n - b0), share = ((nb + kCluster - 1) / kCluster + 3) & ~3;
    *lo = min(nb, rank * share);
    *hi = min(nb, *lo + share);
    return nb;
  };
  int lo, hi, nb = mine(0, &lo, &hi);
  TileIn in;
  load_tile(in, X, T, idx, lo, min(kTile, hi - lo));
  __syncthreads();
  int step = 0;
  for (int b0 = 0; b0 < n; ++step) {
    MlpGrad g = {};
    float loss = 0.0f;
    const float inv = 1.0f / nb;
    for (int r = lo; r < hi; r += kTile) {
      mlp_tile<true>(S.t, g, in, true, 0, min(kTile, hi - r), inv, nullptr, loss);
      if (r + kTile < hi) load_tile(in, X, T, idx, b0 + r + kTile, min(kTile, hi - r - kTile));
    }
    const float2 c = corr[step];
    b0 += batch;
    if (b0 < n) {
      nb = mine(b0, &lo, &hi);
      load_tile(in, X, T, idx, b0 + lo, min(kTile, hi - lo));
    }
    float *out = S.grad;
    reduce_grads(g, S.t.ct, [out](int p, float v) { out[p] = v; });
    cluster.sync();  // every CTA's gradient is complete
    if (owner) {
      float4 part[kCluster];
#pragma unroll
      for (int k = 0; k < kCluster; ++k)
        part[k] = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(S.grad, k) + own);
      float s[4] = {};
#pragma unroll
      for (int k = 0; k < kCluster; ++k) {
        s[0] += part[k].x;
        s[1] += part[k].y;
        s[2] += part[k].z;
        s[3] += part[k].w;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) adam_step(pp[k], pm[k], pv[k], s[k], lr, b1, b2, c.x, c.y, eps);
      *reinterpret_cast<float4 *>(S.p + 4 * tid) = make_float4(pp[0], pp[1], pp[2], pp[3]);
    }
    cluster.sync();  // every slice has its new parameters
    for (int i = tid; i < kCluster * (kSlice / 4); i += kThreads) {
      const int k = i / (kSlice / 4), q = i % (kSlice / 4);
      const float4 v = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(S.p, k) + 4 * q);
      const float w[4] = {v.x, v.y, v.z, v.w};
      const int p = k * kSlice + 4 * q;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (p + j < kMlpParams) put_param(S.t, p + j, w[j]);
    }
    __syncthreads();
  }
  cluster.sync();  // no CTA leaves while its slice may still be read
  if (owner)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (own + k < kMlpParams) {
        params[own + k] = pp[k];
        am[own + k] = pm[k];
        av[own + k] = pv[k];
      }
}

__global__ void adam_kernel(float *p, float *m, float *v, const float *g, int n, float lr,
                            float b1, float b2, float c1, float c2, float eps) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  adam_step(p[i], m[i], v[i], g[i], lr, b1, b2, c1, c2, eps);
}

// The shared-memory opt-ins are per-device attributes: set once per device.
int set_attributes(int dev) {
  static std::mutex mu;
  static bool attr[64] = {};
  if (dev < 0 || dev >= 64) return fail(VINE_ERR_INVALID, "device out of range");
  std::lock_guard<std::mutex> lock(mu);
  if (attr[dev]) return VINE_OK;
  VINE_CUDA_TRY(cudaFuncSetAttribute(mlp_fb_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(MlpShared)));
  VINE_CUDA_TRY(cudaFuncSetAttribute(mlp_fb_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(MlpShared)));
  VINE_CUDA_TRY(cudaFuncSetAttribute(mlp_epoch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(EpochShared)));
  attr[dev] = true;
  return VINE_OK;
}

int fb_launch(const vine_mlp *m, const float *dX, const float *dT, const int32_t *didx, int n,
              float inv_norm, float *dgrad, float *dloss, float *dY, bool backward,
              cudaStream_t s) {
  VINE_TRY(set_attributes(m->device));
  const int ntiles = (n + kTile - 1) / kTile;
  const int grid = std::max(1, std::min(ntiles, 296));  // two CTAs an SM
  if (backward)
    mlp_fb_kernel<true><<<grid, kThreads, sizeof(MlpShared), s>>>(m->params, dX, dT, didx, n, inv_norm, dgrad,
                                                                  dloss, dY);
  else
    mlp_fb_kernel<false><<<grid, kThreads, sizeof(MlpShared), s>>>(m->params, dX, dT, didx, n, inv_norm, nullptr,
                                                                   dloss, dY);
  VINE_CUDA_TRY(cudaGetLastError());
  return VINE_OK;
}

// Device memory of one host-buffer call: the model's kept block, or its own
// allocation when it needs more than kScratchKeep (then freed at the end).
// Allocating and freeing four buffers took 0.1 ms of a call on few rows.
constexpr size_t kScratchKeep = size_t(32) << 20;

class Scratch {
 public:
  explicit Scratch(const vine_mlp *m) : m_(m), lock_(m->scratch_mu) {}
  ~Scratch() {
    if (own_) cudaFree(base_);
  }
  int reserve(size_t bytes) {
    bytes = std::max<size_t>(bytes, 256);
    if (bytes > kScratchKeep) {
      if (cudaMalloc(&base_, bytes) != cudaSuccess) return VINE_CUDA_FAIL("allocation failed");
      own_ = true;
      return VINE_OK;
    }
    if (bytes > m_->scratch_cap) {
      cudaFree(m_->scratch);
      m_->scratch = nullptr;
      m_->scratch_cap = 0;
      const size_t cap = std::min(kScratchKeep, bytes + bytes / 2);
      if (cudaMalloc(&m_->scratch, cap) != cudaSuccess) return VINE_CUDA_FAIL("allocation failed");
      m_->scratch_cap = cap;
    }
    base_ = m_->scratch;
    return VINE_OK;
  }
  // The next `count` values (256-byte aligned; reserve() gets the sum of size()).
  template <typename T>
  T *take(size_t count) {
    T *p = reinterpret_cast<T *>(base_ + used_);
    used_ += size<T>(count);
    return p;
  }
  template <typename T>
  static size_t size(size_t count) {
    return (sizeof(T) * std::max<size_t>(count, 1) + 255) & ~(size_t)255;
  }

 private:
  const vine_mlp *m_;
  std::lock_guard<std::mutex> lock_;
  char *base_ = nullptr;
  size_t used_ = 0;
  bool own_ = false;
};

}  // namespace
}  // namespace vine

using namespace vine;

extern "C" {

int vine_mlp_create(int32_t device, uint64_t seed, const float *params, vine_mlp **out) {
  if (!out) return fail(VINE_ERR_INVALID, "null output");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(VINE_ERR_NO_DEVICE, "no CUDA device");
  if (device < 0 || device >= ndev) return fail(VINE_ERR_INVALID, "device out of range");
  VINE_CUDA_TRY(cudaSetDevice(device));
  std::vector<float> p(kMlpParams, 0.0f);
  if (params) {
    std::memcpy(p.data(), params, sizeof(float) * kMlpParams);
  } else {
    // He-uniform weights, zero biases; one mt19937_64 stream in layout order
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int count, int fan_in) {
      const double a = std::sqrt(6.0 / fan_in);
      for (int i = 0; i < count; ++i) {
        const double u = (double)(rng() >> 11) * (1.0 / 9007199254740992.0);
        p[off + i] = (float)((2.0 * u - 1.0) * a);
      }
    };
    fill(kW1, kHid * kFeat, kFeat);
    fill(kW2, kHid * kHid, kHid);
    fill(kW3, kOut * kHid, kHid);
  }
  auto *m = new vine_mlp();
  m->device = device;
  if (cudaMalloc(&m->params, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaMalloc(&m->adam_m, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaMalloc(&m->adam_v, sizeof(float) * kMlpParams) != cudaSuccess) {
    vine_mlp_destroy(m);
    return VINE_CUDA_FAIL("parameter allocation failed");
  }
  if (cudaMemcpy(m->params, p.data(), sizeof(float) * kMlpParams, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(m->adam_m, 0, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaMemset(m->adam_v, 0, sizeof(float) * kMlpParams) != cudaSuccess ||
      cudaStreamSynchronize(0) != cudaSuccess) {  // the upload has landed before any stream uses it
    vine_mlp_destroy(m);
    return fail(VINE_ERR_CUDA, "parameter upload failed");
  }
  *out = m;
  return VINE_OK;
}

void vine_mlp_destroy(vine_mlp *m) {
  if (!m) return;
  cudaSetDevice(m->device);
  cudaFree(m->params);
  cudaFree(m->adam_m);
  cudaFree(m->adam_v);
  cudaFree(m->scratch);
  delete m;
}

int vine_mlp_get_params(const vine_mlp *m, float *params) {
  if (!m || !params) return fail(VINE_ERR_INVALID, "bad arguments");
  VINE_CUDA_TRY(cudaSetDevice(m->device));
  VINE_CUDA_TRY(cudaMemcpy(params, m->params, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost));
  return VINE_OK;
}

int vine_mlp_set_params(vine_mlp *m, const float *params) {
  if (!m || !params) return fail(VINE_ERR_INVALID, "bad arguments");
  VINE_CUDA_TRY(cudaSetDevice(m->device));
  VINE_CUDA_TRY(cudaMemcpy(m->params, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
  // a copy from pageable memory may return before the DMA lands; wait for the
  // legacy stream so a kernel on a non-blocking caller stream sees the values
  VINE_CUDA_TRY(cudaStreamSynchronize(0));
  return VINE_OK;
}

int vine_mlp_forward(const vine_mlp *m, int32_t n, const float *x, float *y) {
  if (!m || n < 0 || (n > 0 && (!x || !y))) return fail(VINE_ERR_INVALID, "bad arguments");
  if (n == 0) return VINE_OK;
  VINE_CUDA_TRY(cudaSetDevice(m->device));
  Scratch sc(m);
  VINE_TRY(sc.reserve(Scratch::size<float>((size_t)n * kFeat) + Scratch::size<float>((size_t)n * kOut)));
  float *dX = sc.take<float>((size_t)n * kFeat), *dY = sc.take<float>((size_t)n * kOut);
  VINE_CUDA_TRY(cudaMemcpy(dX, x, sizeof(float) * n * kFeat, cudaMemcpyHostToDevice));
  VINE_TRY(fb_launch(m, dX, nullptr, nullptr, n, 1.0f, nullptr, nullptr, dY, false, 0));
  VINE_CUDA_TRY(cudaMemcpy(y, dY, sizeof(float) * n * kOut, cudaMemcpyDeviceToHost));
  return VINE_OK;
}

int vine_mlp_loss_grad(const vine_mlp *m, int32_t n, const float *x, const float *y_target,
                       float *loss, float *grad) {
  if (!m || n <= 0 || !x || !y_target || !loss || !grad) return fail(VINE_ERR_INVALID, "bad arguments");
  VINE_CUDA_TRY(cudaSetDevice(m->device));
  Scratch sc(m);
  VINE_TRY(sc.reserve(Scratch::size<float>((size_t)n * kFeat) + Scratch::size<float>((size_t)n * kOut) +
                      Scratch::size<float>(kMlpParams + 1)));
  float *dX = sc.take<float>((size_t)n * kFeat), *dT = sc.take<float>((size_t)n * kOut),
        *dG = sc.take<float>(kMlpParams + 1);  // the gradient, then the loss
  VINE_CUDA_TRY(cudaMemcpy(dX, x, sizeof(float) * n * kFeat, cudaMemcpyHostToDevice));
  VINE_CUDA_TRY(cudaMemcpy(dT, y_target, sizeof(float) * n * kOut, cudaMemcpyHostToDevice));
  VINE_CUDA_TRY(cudaMemsetAsync(dG, 0, sizeof(float) * (kMlpParams + 1), 0));
  VINE_TRY(fb_launch(m, dX, dT, nullptr, n, 1.0f / n, dG, dG + kMlpParams, nullptr, true, 0));
  float host[kMlpParams + 1];
  VINE_CUDA_TRY(cudaMemcpy(host, dG, sizeof(host), cudaMemcpyDeviceToHost));
  std::memcpy(grad, host, sizeof(float) * kMlpParams);
  *loss = host[kMlpParams];
  return VINE_OK;
}

int vine_mlp_train(vine_mlp *m, int32_t n, const float *x, const float *y_target, int32_t epochs,
                   int32_t batch, float lr, uint64_t seed, float *final_loss) {
  if (!m || n <= 0 || !x || !y_target || epochs < 0 || batch <= 0 || !(lr > 0.0f))
    return fail(VINE_ERR_INVALID, "bad arguments");
  VINE_CUDA_TRY(cudaSetDevice(m->device));
  const int32_t steps = (int32_t)(((int64_t)n + batch - 1) / batch);
  const bool clustered = batch <= kEpochMaxBatch;
  Scratch sc(m);
  VINE_TRY(sc.reserve(Scratch::size<float>((size_t)n * kFeat) + Scratch::size<float>((size_t)n * kOut) +
                      Scratch::size<float>(kMlpParams) + Scratch::size<float>(1) +
                      Scratch::size<int32_t>((size_t)n) + Scratch::size<float2>((size_t)steps)));
  float *dX = sc.take<float>((size_t)n * kFeat), *dT = sc.take<float>((size_t)n * kOut),
        *dG = sc.take<float>(kMlpParams), *dL = sc.take<float>(1);
  int32_t *dI = sc.take<int32_t>((size_t)n);
  float2 *dC = sc.take<float2>((size_t)steps);  // bias corrections of an epoch's steps
  VINE_CUDA_TRY(cudaMemcpy(dX, x, sizeof(float) * n * kFeat, cudaMemcpyHostToDevice));
  VINE_CUDA_TRY(cudaMemcpy(dT, y_target, sizeof(float) * n * kOut, cudaMemcpyHostToDevice));
  std::vector<int32_t> perm(n);
  for (int32_t i = 0; i < n; ++i) perm[i] = i;
  std::mt19937_64 rng(seed);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  std::vector<float2> corr((size_t)steps);
  if (clustered) VINE_TRY(set_attributes(m->device));
  for (int e = 0; e < epochs; ++e) {
    for (int32_t i = n - 1; i > 0; --i) {  // Fisher-Yates with a fixed stream
      const int32_t j = (int32_t)(rng() % (uint64_t)(i + 1));
      std::swap(perm[i], perm[j]);
    }
    VINE_CUDA_TRY(cudaMemcpy(dI, perm.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice));
    if (clustered) {
      for (float2 &c : corr) {
        m->step++;
        c = make_float2(1.0f - std::pow(b1, (float)m->step), 1.0f - std::pow(b2, (float)m->step));
      }
      VINE_CUDA_TRY(cudaMemcpy(dC, corr.data(), sizeof(float2) * corr.size(), cudaMemcpyHostToDevice));
      mlp_epoch_kernel<<<kCluster, kThreads, sizeof(EpochShared)>>>(m->params, m->adam_m, m->adam_v, dX, dT,
                                                                    dI, n, batch, dC, lr, b1, b2, eps);
      VINE_CUDA_TRY(cudaGetLastError());
      continue;
    }
    for (int32_t b0 = 0; b0 < n; b0 += batch) {
      const int32_t nb = std::min(batch, n - b0);
      VINE_CUDA_TRY(cudaMemsetAsync(dG, 0, sizeof(float) * kMlpParams, 0));
      VINE_TRY(fb_launch(m, dX, dT, dI + b0, nb, 1.0f / nb, dG, nullptr, nullptr, true, 0));
      m->step++;
      const float c1 = 1.0f - std::pow(b1, (float)m->step);
      const float c2 = 1.0f - std::pow(b2, (float)m->step);
      adam_kernel<<<(kMlpParams + 255) / 256, 256>>>(m->params, m->adam_m, m->adam_v, dG,
                                                     kMlpParams, lr, b1, b2, c1, c2, eps);
      VINE_CUDA_TRY(cudaGetLastError());
    }
  }
  VINE_CUDA_TRY(cudaMemset(dL, 0, sizeof(float)));
  VINE_TRY(fb_launch(m, dX, dT, nullptr, n, 1.0f / n, nullptr, dL, nullptr, false, 0));
  float l = 0.0f;
  VINE_CUDA_TRY(cudaMemcpy(&l, dL, sizeof(float), cudaMemcpyDeviceToHost));
  if (final_loss) *final_loss = l;
  return VINE_OK;
}

// ------------------------------------------- no-allocation loss / gradient
//
// Callers that may not allocate device memory (a scheduler-refinement loop
// running beside a seconds-long batch solve, where cudaFree would wait for
// the whole device; a process whose HBM the label arena already holds) use
// vine_mlp_loss_grad_noalloc.  Its staging buffers live in one fixed array
// in the library image instead of cudaMalloc'd memory.
//
// Scratch layout (floats; every region starts on a 256-byte boundary):
//   [0]                          loss accumulator      (zeroed by each call)
//   [kNaGrad, +kMlpParams)       gradient accumulator  (zeroed by each call)
//   [kNaX, +maxrows * 16)        x rows                (overwritten by each call)
//   [kNaT, +maxrows * 2)         targets               (overwritten by each call)

}  // extern "C"

namespace vine {
namespace {

constexpr int kNaMaxRows = VINE_MLP_NOALLOC_MAX_ROWS;
constexpr size_t kNaAlign = 64;  // floats: 256 bytes
constexpr size_t kNaGrad = kNaAlign;
constexpr size_t kNaX = kNaGrad + ((kMlpParams + kNaAlign - 1) / kNaAlign) * kNaAlign;
constexpr size_t kNaT = kNaX + (size_t)kNaMaxRows * kFeat;
constexpr size_t kNaFloats = kNaT + (size_t)kNaMaxRows * kOut;  // 79,232 floats = 309.5 KiB
static_assert(kNaFloats == 79232, "no-allocation scratch size changed: update the documented size");

static __device__ __align__(256) float g_noalloc_scratch[kNaFloats];

constexpr int kNaMaxDevices = 64;
std::mutex g_na_mu;
float *g_na_ptr[kNaMaxDevices] = {};

// Device address of the scratch array on `device` (the current device),
// looked up once per device.
int noalloc_scratch(int device, float **out) {
  if (device < 0 || device >= kNaMaxDevices) return fail(VINE_ERR_INVALID, "device out of range");
  std::lock_guard<std::mutex> lock(g_na_mu);
  if (g_na_ptr[device] == nullptr) {
    float *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress((void **)&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr)
      return fail(VINE_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") +
                                     cudaGetErrorString(e));
    g_na_ptr[device] = p;
  }
  *out = g_na_ptr[device];
  return VINE_OK;
}

}  // namespace
}  // namespace vine

extern "C" {

int vine_mlp_loss_grad_noalloc(const vine_mlp *m, int32_t n, const float *x,
                               const float *y_target, float *loss, float *grad, void *stream) {
  if (!m || !x || !y_target || !loss || !grad) return fail(VINE_ERR_INVALID, "bad arguments");
  if (n < 1 || n > kNaMaxRows)
    return fail(VINE_ERR_INVALID, "vine_mlp_loss_grad_noalloc: n = " + std::to_string(n) +
                                      " rows, allowed 1.." + std::to_string(kNaMaxRows) +
                                      " (VINE_MLP_NOALLOC_MAX_ROWS)");
  VINE_CUDA_TRY(cudaSetDevice(m->device));
  float *scratch = nullptr;
  VINE_TRY(noalloc_scratch(m->device, &scratch));
  cudaStream_t s = (cudaStream_t)stream;
  float *dL = scratch, *dG = scratch + kNaGrad, *dX = scratch + kNaX, *dT = scratch + kNaT;
  VINE_CUDA_TRY(cudaMemsetAsync(scratch, 0, sizeof(float) * kNaX, s));  // loss + gradient
  VINE_CUDA_TRY(cudaMemcpyAsync(dX, x, sizeof(float) * (size_t)n * kFeat, cudaMemcpyHostToDevice, s));
  VINE_CUDA_TRY(cudaMemcpyAsync(dT, y_target, sizeof(float) * (size_t)n * kOut,
                                cudaMemcpyHostToDevice, s));
  VINE_TRY(fb_launch(m, dX, dT, nullptr, n, 1.0f / n, dG, dL, nullptr, true, s));
  VINE_CUDA_TRY(cudaMemcpyAsync(grad, dG, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, s));
  VINE_CUDA_TRY(cudaMemcpyAsync(loss, dL, sizeof(float), cudaMemcpyDeviceToHost, s));
  VINE_CUDA_TRY(cudaStreamSynchronize(s));
  return VINE_OK;
}

}  // extern "C"
