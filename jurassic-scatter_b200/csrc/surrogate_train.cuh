// Training step of the surrogate in three launches (FP32):
//
//   train_rows_kernel    a block per 32 samples: minibatch gather, forward,
//                        loss gradient and the gradients of every layer's
//                        outputs, activations in shared memory
//   train_weights_kernel partial weight gradients of a slice of the samples
//                        and a 64 x 64 tile, and the bias gradients
//   train_update_kernel  the slices added in order, then Adam
//
// Before them, once: train_stats_kernel, train_stats_sum_kernel and
// train_targets_kernel standardise the training set.
//
// Every sum runs in the order of a plain product (the inner index upwards,
// slices of the samples in order, bias sums over eight interleaved rows; the
// products of the contractions are fused into their sums), so training is
// deterministic and does not depend on the tiling.
#pragma once
#include <math.h>
#include <stdint.h>

#include "surrogate.h"

#define TR_ROWS 32               // samples per block
#define TR_LD 36                 // row of a transposed activation tile
#define TR_K 32                  // inner indices per weight tile
#define TR_THREADS 256
#define TR_KSPLIT_MAX 64         // slices of the samples for the weight gradients

struct TrainNet {
  int nout, in[4], out[4];
  float *w[4], *b[4];            // weights [out][in], biases
  float *wt[4];                  // weights [in][out]
  float *gw[4], *gb[4];          // gradients
  float *mw[4], *vw[4], *mb[4], *vb[4];  // Adam moments
  int off[5];                    // first weight of each layer in a slice
};

struct TrainBatch {
  int n;
  const int *idx;                // samples of the minibatch, or null: x, t as given
  const float *x, *t;            // [.][SUR_NF], [.][nout]
  const float *xm, *xs;          // standardisation of x (with idx)
  float *h[4];                   // inputs of the layers [n][in]
  float *dz[4];                  // gradients of their outputs [n][out]
  float *err;                    // [n][nout] output minus target
};

// Weight tile k0 .. k0 + 31 of B [K][N] for the 256 threads: four values of
// four columns each, zero beyond B.
__device__ __forceinline__ void tile_fetch(const float *B, int K, int N, int k0, float4 *r) {
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int e = threadIdx.x + j * TR_THREADS, k = k0 + e / 32, c = (e % 32) * 4;
    r[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < K && c < N) {
      const float *p = B + (size_t)k * N + c;
      if ((N & 3) == 0) {
        r[j] = *reinterpret_cast<const float4 *>(p);
      } else {
        r[j].x = p[0];
        if (c + 1 < N) r[j].y = p[1];
        if (c + 2 < N) r[j].z = p[2];
        if (c + 3 < N) r[j].w = p[3];
      }
    }
  }
}

__device__ __forceinline__ void tile_store(float (*wt)[SUR_W], const float4 *r) {
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int e = threadIdx.x + j * TR_THREADS;
    *reinterpret_cast<float4 *>(&wt[e / 32][(e % 32) * 4]) = r[j];
  }
}

// acc[row][col] = sum over k upwards of a[k][row] B[k][col]: rows 4 w .. 4 w
// + 3 of the warp w, columns 4 lane .. 4 lane + 3 (128 in all; idle past N).
__device__ __forceinline__ void rows_product(const float *a, const float *B, int K, int N,
                                             float (*wt)[TR_K][SUR_W], float (*acc)[4]) {
  const int w = threadIdx.x >> 5, c = (threadIdx.x & 31) * 4;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
  float4 r[4];
  tile_fetch(B, K, N, 0, r);
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += TR_K, buf ^= 1) {
    tile_store(wt[buf], r);
    __syncthreads();  // the tile is complete; the other one has been read
    if (k0 + TR_K < K) tile_fetch(B, K, N, k0 + TR_K, r);
    const int m = min(TR_K, K - k0);
    if (c < N) {
#pragma unroll 8
      for (int k = 0; k < m; k++) {
        const float4 av = *reinterpret_cast<const float4 *>(a + (k0 + k) * TR_LD + 4 * w);
        const float4 bv = *reinterpret_cast<const float4 *>(&wt[buf][k][c]);
        const float as[4] = {av.x, av.y, av.z, av.w}, bs[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) acc[i][j] = fmaf(as[i], bs[j], acc[i][j]);
      }
    }
  }
  __syncthreads();  // a and the tiles may be rewritten
}

// Bound by the latency of its shared-memory operands, eight warps on each of
// 128 SMs: 43 us of a step of 4096 samples, 15 us at the full FP32 rate; with
// a multiplication and an addition per product it took 51.  The step took 330
// us in 35 launches, most of it products of 64 x 64 tiles of which each layer
// fills a few blocks and bias sums in one to four blocks; now 75 us in three.
static __global__ void __launch_bounds__(TR_THREADS) train_rows_kernel(TrainNet net, TrainBatch b) {
  extern __shared__ __align__(16) float tr_sh[];
  float *ht[4];                                    // inputs of the layers, [in][TR_LD]
  ht[0] = tr_sh;
  ht[1] = ht[0] + SUR_NF * TR_LD;
  ht[2] = ht[1] + SUR_W * TR_LD;
  ht[3] = ht[2] + SUR_W * TR_LD;
  float *dz = ht[3] + SUR_W * TR_LD;               // [out][TR_LD]
  float (*wt)[TR_K][SUR_W] = reinterpret_cast<float (*)[TR_K][SUR_W]>(dz + SUR_W * TR_LD);
  const int row0 = blockIdx.x * TR_ROWS, rows = min(TR_ROWS, b.n - row0);
  const int w = threadIdx.x >> 5, c = (threadIdx.x & 31) * 4;
  const int nout = net.nout;
  {
    const int i = threadIdx.x / SUR_NF, k = threadIdx.x % SUR_NF;
    static_assert(TR_THREADS == TR_ROWS * SUR_NF, "one feature per thread");
    float v = 0.f;
    if (i < rows) {
      if (b.idx) {
        v = (b.x[(size_t)b.idx[row0 + i] * SUR_NF + k] - b.xm[k]) / b.xs[k];
        b.h[0][(size_t)(row0 + i) * SUR_NF + k] = v;
      } else {
        v = b.x[(size_t)(row0 + i) * SUR_NF + k];
      }
    }
    ht[0][k * TR_LD + i] = v;
  }
  __syncthreads();
  float acc[4][4];
#pragma unroll 1
  for (int l = 0; l < 3; l++) {
    rows_product(ht[l], net.wt[l], net.in[l], SUR_W, wt, acc);
    const float4 bias = *reinterpret_cast<const float4 *>(net.b[l] + c);
    const float bs[4] = {bias.x, bias.y, bias.z, bias.w};
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = tanhf(acc[i][j] + bs[j]);
#pragma unroll
    for (int j = 0; j < 4; j++)
      *reinterpret_cast<float4 *>(ht[l + 1] + (c + j) * TR_LD + 4 * w) =
          make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (4 * w + i < rows)
        *reinterpret_cast<float4 *>(b.h[l + 1] + (size_t)(row0 + 4 * w + i) * SUR_W + c) =
            make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
  }
  // Output layer, error and the loss gradient 2 (y - t) / n.
  rows_product(ht[3], net.wt[3], SUR_W, nout, wt, acc);
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (c + j < nout)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int row = row0 + 4 * w + i;
        float d = 0.f;
        if (row < b.n) {
          const float y = acc[i][j] + net.b[3][c + j];
          const int src = b.idx ? b.idx[row] : row;
          const float e = y - b.t[(size_t)src * nout + c + j];
          d = 2.f * e / (float)b.n;
          b.err[(size_t)row * nout + c + j] = e;
          b.dz[3][(size_t)row * nout + c + j] = d;
        }
        dz[(c + j) * TR_LD + 4 * w + i] = d;
      }
  __syncthreads();
  // dH_l = dZ_l W_l, dZ_(l-1) = dH_l (1 - H_l^2)
#pragma unroll 1
  for (int l = 3; l > 0; l--) {
    rows_product(dz, net.w[l], net.out[l], SUR_W, wt, acc);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float4 h = *reinterpret_cast<const float4 *>(ht[l] + (c + j) * TR_LD + 4 * w);
      acc[0][j] *= 1.f - h.x * h.x;
      acc[1][j] *= 1.f - h.y * h.y;
      acc[2][j] *= 1.f - h.z * h.z;
      acc[3][j] *= 1.f - h.w * h.w;
      *reinterpret_cast<float4 *>(dz + (c + j) * TR_LD + 4 * w) =
          make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (4 * w + i < rows)
        *reinterpret_cast<float4 *>(b.dz[l - 1] + (size_t)(row0 + 4 * w + i) * SUR_W + c) =
            make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
  }
}

#define TR_ROWS_SHMEM \
  ((int)sizeof(float) * ((SUR_NF + 4 * SUR_W) * TR_LD + 2 * TR_K * SUR_W))

// Tiles of the weight gradients: 64 outputs x 64 inputs (layer 0: its 8
// inputs).
#define TR_TILES 12

// Blocks 0 .. ncol-1: bias gradients, 32 columns each (eight threads per
// column take every eighth row, then their sums in order).  The others: the
// partial weight gradient of slice z of the samples and one tile, rows
// upwards, into ws[z].
static __global__ void __launch_bounds__(TR_THREADS)
train_weights_kernel(TrainNet net, TrainBatch b, int ncol, int kchunk, float *ws) {
  __shared__ __align__(16) float as[64][64], bs[64][64];
  if ((int)blockIdx.x < ncol) {
    int l = 0, c0 = (int)blockIdx.x * 32;
    while (c0 >= (net.out[l] + 31) / 32 * 32) c0 -= (net.out[l++] + 31) / 32 * 32;
    const int o = c0 + (threadIdx.x & 31), r0 = threadIdx.x >> 5, cols = net.out[l];
    const float *dz = b.dz[l];
    float sum = 0;
    if (o < cols) {
#pragma unroll 16
      for (int i = r0; i < b.n; i += 8) sum += dz[(size_t)i * cols + o];
    }
    as[r0][threadIdx.x & 31] = sum;
    __syncthreads();
    if (r0 == 0 && o < cols) {
      float t = 0;
      for (int j = 0; j < 8; j++) t += as[j][threadIdx.x];
      net.gb[l][o] = t;
    }
    return;
  }
  const int t = (int)blockIdx.x - ncol, z = t / TR_TILES, tile = t - z * TR_TILES;
  // tiles 0-3 layer 1, 4-7 layer 2, 8-9 layer 3, 10-11 layer 0
  const int l = tile < 4 ? 1 : tile < 8 ? 2 : tile < 10 ? 3 : 0;
  const int o0 = l == 0 ? (tile - 10) * 64 : l == 3 ? 0 : ((tile & 3) >> 1) * 64;
  const int i0 = l == 0 ? 0 : (tile & 1) * 64;
  const int no = min(64, net.out[l] - o0), ni = min(64, net.in[l] - i0);
  const int lo = net.out[l], li = net.in[l];
  const int kb = z * kchunk, ke = min(b.n, kb + kchunk);
  const float *dz = b.dz[l] + o0, *h = b.h[l] + i0;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  for (int k0 = kb; k0 < ke; k0 += 64) {
    const int m = min(64, ke - k0);
    __syncthreads();
    for (int e = threadIdx.x; e < m * 64; e += TR_THREADS) {
      const int k = e >> 6, j = e & 63;
      as[k][j] = j < no ? dz[(size_t)(k0 + k) * lo + j] : 0.f;
      bs[k][j] = j < ni ? h[(size_t)(k0 + k) * li + j] : 0.f;
    }
    __syncthreads();
    if (l == 0) {  // 64 outputs x 8 inputs: two a thread
      const int o = threadIdx.x >> 2, i = (threadIdx.x & 3) * 2;
      for (int k = 0; k < m; k++) {
        const float a = as[k][o];
        acc[0][0] = fmaf(a, bs[k][i], acc[0][0]);
        acc[0][1] = fmaf(a, bs[k][i + 1], acc[0][1]);
      }
    } else if (ty * 4 < no) {
#pragma unroll 4
      for (int k = 0; k < m; k++) {
        const float4 av = *reinterpret_cast<const float4 *>(&as[k][ty * 4]);
        const float4 bv = *reinterpret_cast<const float4 *>(&bs[k][tx * 4]);
        const float aa[4] = {av.x, av.y, av.z, av.w}, bb[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) acc[i][j] = fmaf(aa[i], bb[j], acc[i][j]);
      }
    }
  }
  float *out = ws + (size_t)z * net.off[4] + net.off[l];
  if (l == 0) {
    const int o = threadIdx.x >> 2, i = (threadIdx.x & 3) * 2;
    out[(size_t)(o0 + o) * li + i] = acc[0][0];
    out[(size_t)(o0 + o) * li + i + 1] = acc[0][1];
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (ty * 4 + i < no)
        *reinterpret_cast<float4 *>(out + (size_t)(o0 + ty * 4 + i) * li + i0 + tx * 4) =
            make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  }
}

struct TrainAdam {
  int on;                        // 0: leave the gradients in gw, gb
  float lr, b1, b2, c1, c2, eps;
};

__device__ __forceinline__ float adam_step(const TrainAdam &a, float *p, float *m, float *v, float g) {
  const float mi = a.b1 * *m + (1 - a.b1) * g;
  const float vi = a.b2 * *v + (1 - a.b2) * g * g;
  *m = mi;
  *v = vi;
  return *p -= a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
}

// A thread per weight, then per bias.
static __global__ void __launch_bounds__(TR_THREADS)
train_update_kernel(TrainNet net, TrainAdam a, int nz, const float *ws) {
  int i = blockIdx.x * TR_THREADS + threadIdx.x;
  const int total = net.off[4];
  if (i < total) {
    float g = 0;
#pragma unroll 16
    for (int z = 0; z < nz; z++) g += ws[(size_t)z * total + i];
    int l = 0;
    while (i >= net.off[l + 1]) l++;
    i -= net.off[l];
    if (!a.on) {
      net.gw[l][i] = g;
      return;
    }
    const float p = adam_step(a, net.w[l] + i, net.mw[l] + i, net.vw[l] + i, g);
    const int o = i / net.in[l];
    net.wt[l][(size_t)(i - o * net.in[l]) * net.out[l] + o] = p;
    return;
  }
  i -= total;
  for (int l = 0; l < 4; l++) {
    if (i < net.out[l]) {
      if (a.on) adam_step(a, net.b[l] + i, net.mb[l] + i, net.vb[l] + i, net.gb[l][i]);
      return;
    }
    i -= net.out[l];
  }
}

// Transposed copies of the weights.
static __global__ void __launch_bounds__(TR_THREADS) train_transpose_kernel(TrainNet net) {
  int i = blockIdx.x * TR_THREADS + threadIdx.x, l = 0;
  if (i >= net.off[4]) return;
  while (i >= net.off[l + 1]) l++;
  i -= net.off[l];
  const int o = i / net.in[l];
  net.wt[l][(size_t)(i - o * net.in[l]) * net.out[l] + o] = net.w[l][i];
}

// Per-block sums of the squared errors (the loss is their sum over n).
static __global__ void __launch_bounds__(TR_THREADS) train_loss_kernel(int64_t cnt, const float *err,
                                                                       float *part) {
  __shared__ float red[TR_THREADS];
  const int64_t i = (int64_t)blockIdx.x * TR_THREADS + threadIdx.x;
  float e2 = 0;
  if (i < cnt) e2 = err[i] * err[i];
  red[threadIdx.x] = e2;
  __syncthreads();
  for (int o = TR_THREADS / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

#define TR_STAT_BLOCKS 296       // two per SM
#define TR_STATS 4               // sum, sum of squares, lowest, highest

// Statistics of the nc <= 64 columns of v [n][nc], a part per block; LOG:
// each value is replaced by its logarithm first.  Lanes run over the columns
// and rows of a block's slice, so loads are contiguous; sums in FP64 in a
// fixed order.  Bound by the read and write, 10 us for 65536 samples x 16
// channels (sums over the blocks 20 us, targets 5); with two passes of logarithms on the host a training of 8
// epochs on that set took 39 ms, with this 22.
template <typename T, bool LOG>
static __global__ void __launch_bounds__(TR_THREADS)
train_stats_kernel(int64_t n, int nc, T *v, double *part) {
  __shared__ double red[TR_STATS][TR_THREADS];
  const int t = threadIdx.x, rows = TR_THREADS / nc, rl = t / nc, c = t - rl * nc;
  double s = 0, s2 = 0, lo = INFINITY, hi = -INFINITY;
  if (rl < rows)
    for (int64_t i = (int64_t)blockIdx.x * rows + rl; i < n; i += (int64_t)gridDim.x * rows) {
      double x = v[i * nc + c];
      if (LOG) v[i * nc + c] = x = log(fmax(x, 1e-300));
      s += x;
      s2 += x * x;
      if (x < lo) lo = x;
      if (x > hi) hi = x;
    }
  red[0][t] = s;
  red[1][t] = s2;
  red[2][t] = lo;
  red[3][t] = hi;
  __syncthreads();
  if (t >= nc) return;
  for (int r = 1; r < rows; r++) {
    s += red[0][r * nc + t];
    s2 += red[1][r * nc + t];
    lo = red[2][r * nc + t] < lo ? red[2][r * nc + t] : lo;
    hi = red[3][r * nc + t] > hi ? red[3][r * nc + t] : hi;
  }
  double *p = part + (size_t)blockIdx.x * TR_STATS * nc + t;
  p[0] = s;
  p[nc] = s2;
  p[2 * nc] = lo;
  p[3 * nc] = hi;
}

// The blocks' parts together: out [TR_STATS][nc], a thread per value.
static __global__ void __launch_bounds__(TR_STATS * SUR_NOUT_MAX)
train_stats_sum_kernel(int nblk, int nc, const double *part, double *out) {
  const int t = threadIdx.x, k = t / nc;
  if (k >= TR_STATS) return;
  double a = part[t];
#pragma unroll 8
  for (int b = 1; b < nblk; b++) {
    const double x = part[(size_t)b * TR_STATS * nc + t];
    a = k < 2 ? a + x : k == 2 ? (x < a ? x : a) : (x > a ? x : a);
  }
  out[t] = a;
}

// Standardised targets: (y - mean) / spread of each column.
static __global__ void __launch_bounds__(TR_THREADS)
train_targets_kernel(int64_t cnt, int nc, const double *y, const double *mean, const float *spread,
                     float *t) {
  const int64_t i = (int64_t)blockIdx.x * TR_THREADS + threadIdx.x;
  if (i >= cnt) return;
  const int c = (int)(i % nc);
  t[i] = (float)((y[i] - mean[c]) / spread[c]);
}
