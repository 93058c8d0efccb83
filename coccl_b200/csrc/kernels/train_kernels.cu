// Memory-bound training kernels of the GPT trainer (bf16 activations, fp32
// statistics): residual-add + LayerNorm / RMSNorm forward/backward, GELU backward,
// column sums (bias gradients), fused cross-entropy forward+backward, fused
// Adam with fp32 master weights, squared-norm reduction and clip coefficient.
//
// The reference ships no trainer (its training layer is an empty submodule,
// .gitmodules:1-3); these kernels belong to the framework layer that drives the
// compressed collectives. Each kernel touches every byte once.
#include "dependent_launch.h"
#include "launch_count.h"
#include "common.cuh"
#include "train_api.h"
#include "no_alloc_api.h"
#include <mutex>
#include <stdio.h>
#include <math.h>

namespace coccl {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float warpSum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ float warpMax(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
// Block-wide sum; `sm` holds 32 floats. All threads get the result.
__device__ __forceinline__ float blockSum(float x, float* sm) {
  x = warpSum(x);
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[w] = x;
  __syncthreads();
  float t = (threadIdx.x & 31) < nw ? sm[threadIdx.x & 31] : 0.f;
  return warpSum(t);
}
__device__ __forceinline__ float blockMax(float x, float* sm) {
  x = warpMax(x);
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[w] = x;
  __syncthreads();
  float t = (threadIdx.x & 31) < nw ? sm[threadIdx.x & 31] : -INFINITY;
  return warpMax(t);
}

// ---------------------------------------------------------------- LayerNorm and RMSNorm
constexpr int kLnThreads = 256;
constexpr int kLnMaxVec = 8;  // H <= 256*8*8 = 16384

// xs = x (+ res); xOut = xs (optional); y = (xs - mean) * rstd * gamma + beta. RMS: y = xs * rstd * gamma with
// rstd = 1 / sqrt(mean(xs^2) + eps), no mean and no beta.
// Memory-bound: every byte moves once, 24 us (LayerNorm) and 21 us (RMSNorm) for the 134 MB of 4096 x 4096 with a residual,
// 20.5 us to copy. A CTA has no more threads than the row has 16-byte vectors, so narrow rows do not carry idle warps through the block reductions.
template <int NV, bool RMS>
__global__ void __launch_bounds__(kLnThreads) normFwdKernel(const bf16* x, const bf16* res, const bf16* gamma,
                                                            const bf16* beta, bf16* y, bf16* xOut, float* mean,
                                                            float* rstd, int M, int H, float eps) {
  releaseNext();
  awaitPrevious();
  __shared__ float sm[32];
  const int nvec = H / 8;
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    const bf16* xr = x + (long)row * H;
    float v[NV][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int vi = threadIdx.x + i * kLnThreads;
      if (vi < nvec) {
        Vec8<bf16>::load(xr + vi * 8, 8, true, v[i]);
        if (res) {
          float r[8];
          Vec8<bf16>::load(res + (long)row * H + vi * 8, 8, true, r);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] += r[j];
        }
        if (xOut) {
          Vec8<bf16>::store(xOut + (long)row * H + vi * 8, 8, true, v[i]);
          // keep the statistics consistent with the rounded value that is saved
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = __bfloat162float(__float2bfloat16_rn(v[i][j]));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) s += RMS ? v[i][j] * v[i][j] : v[i][j];
      }
    }
    float mu = 0.f, q = 0.f;
    if (RMS) {
      q = blockSum(s, sm) / H;
    } else {
      mu = blockSum(s, sm) / H;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int vi = threadIdx.x + i * kLnThreads;
        if (vi < nvec) {
#pragma unroll
          for (int j = 0; j < 8; ++j) { const float d = v[i][j] - mu; q += d * d; }
        }
      }
      q = blockSum(q, sm) / H;
    }
    const float rs = rsqrtf(q + eps);
    if (threadIdx.x == 0) { if (!RMS) mean[row] = mu; rstd[row] = rs; }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int vi = threadIdx.x + i * kLnThreads;
      if (vi < nvec) {
        float g[8], b[8], o[8];
        Vec8<bf16>::load(gamma + vi * 8, 8, true, g);
        if (!RMS) Vec8<bf16>::load(beta + vi * 8, 8, true, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = RMS ? v[i][j] * rs * g[j] : (v[i][j] - mu) * rs * g[j] + b[j];
        Vec8<bf16>::store(y + (long)row * H + vi * 8, 8, true, o);
      }
    }
  }
}

__device__ __forceinline__ void unpackBf16x8(const uint4& a, float (&v)[8]) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// dx = rstd * (dy*gamma - mean(dy*gamma) - xhat * mean(dy*gamma*xhat)) (+ dres); RMS: without the mean(dy*gamma) term.
// partial[blockIdx.x][0][h] = sum_rows dy*xhat, partial[blockIdx.x][1][h] = sum_rows dy (RMS: only the first of the two)
//
// What bounds a row is the chain load -> block reduction -> store, not the arithmetic: with the row held as fp32 the
// kernel had two CTAs of one row each per SM in flight and ran at 0.41 of the copy rate. Here a row is held as it was
// loaded (packed bf16; xhat and dy*gamma are formed twice from it) and the loads of the CTA's NEXT row are issued before
// the reduction of the current one; the two sums share one reduction and one barrier (the two halves of `sm` alternate).
// 4096 x 4096 with a residual gradient: 50 -> 33.6 us (LayerNorm), 25 us (RMSNorm), of 134 MB that take 20.5 us to copy.
template <int NV, bool RMS>
__global__ void __launch_bounds__(kLnThreads) normBwdKernel(const bf16* dy, const bf16* x, const float* mean,
                                                            const float* rstd, const bf16* gamma, const bf16* dres,
                                                            bf16* dx, float* partial, int M, int H) {
  releaseNext();
  awaitPrevious();
  __shared__ float2 sm[2][8];
  const int nvec = H / 8, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float dg[NV][8], db[RMS ? 1 : NV][8];
  uint4 gm[NV], nd[NV], nx[NV], nr[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    gm[i] = vi < nvec ? loadOrdered(reinterpret_cast<const uint4*>(gamma) + vi) : make_uint4(0, 0, 0, 0);
    nd[i] = nx[i] = nr[i] = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 8; ++j) { dg[i][j] = 0.f; if (!RMS) db[i][j] = 0.f; }
  }
  float nmu = 0.f, nrs = 0.f;
  auto fetch = [&](int row) {
    const long base = (long)row * nvec;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int vi = threadIdx.x + i * blockDim.x;
      if (vi < nvec) {
        nd[i] = loadOrdered(reinterpret_cast<const uint4*>(dy) + base + vi);
        nx[i] = loadOrdered(reinterpret_cast<const uint4*>(x) + base + vi);
        if (dres) nr[i] = loadOrdered(reinterpret_cast<const uint4*>(dres) + base + vi);
      }
    }
    if (!RMS) nmu = mean[row];
    nrs = rstd[row];
  };
  if (blockIdx.x < M) fetch(blockIdx.x);
  int parity = 0;
  for (int row = blockIdx.x; row < M; row += gridDim.x, parity ^= 1) {
    uint4 cd[NV], cx[NV], cr[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) { cd[i] = nd[i]; cx[i] = nx[i]; cr[i] = nr[i]; }
    const float mu = nmu, rs = nrs;
    if (row + (int)gridDim.x < M) fetch(row + gridDim.x);
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {   // vectors past the row are zero in dy and gamma and add nothing
      float d[8], xv[8], g[8];
      unpackBf16x8(cd[i], d);
      unpackBf16x8(cx[i], xv);
      unpackBf16x8(gm[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = RMS ? xv[j] * rs : (xv[j] - mu) * rs, t = d[j] * g[j];
        if (!RMS) s1 += t;
        s2 += t * xh;
        dg[i][j] += d[j] * xh;
        if (!RMS) db[i][j] += d[j];
      }
    }
    if (!RMS) s1 = warpSum(s1);
    s2 = warpSum(s2);
    if ((threadIdx.x & 31) == 0) sm[parity][warp] = make_float2(s1, s2);
    __syncthreads();
    float c1 = 0.f, c2 = 0.f;
    for (int w = 0; w < nw; ++w) { const float2 t = sm[parity][w]; c1 += t.x; c2 += t.y; }
    c1 /= H;
    c2 /= H;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int vi = threadIdx.x + i * blockDim.x;
      if (vi < nvec) {
        float d[8], xv[8], g[8], r[8], o[8];
        unpackBf16x8(cd[i], d);
        unpackBf16x8(cx[i], xv);
        unpackBf16x8(gm[i], g);
        unpackBf16x8(cr[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = RMS ? xv[j] * rs : (xv[j] - mu) * rs, t = d[j] * g[j];
          o[j] = rs * (RMS ? t - xh * c2 : t - c1 - xh * c2);
          if (dres) o[j] += r[j];
        }
        Vec8<bf16>::store(dx + (long)row * H + vi * 8, 8, true, o);
      }
    }
  }
  float* pg = partial + (long)blockIdx.x * (RMS ? 1 : 2) * H;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi < nvec) {
      Vec8<float>::store(pg + vi * 8, 8, true, dg[i]);
      if (!RMS) Vec8<float>::store(pg + H + vi * 8, 8, true, db[RMS ? 0 : i]);
    }
  }
}

// The same for rows wider than 8192, where sums for two weights and a row of which some is prefetched do not fit the registers
// (eight vectors a thread spilled 5.6 KB: 4096 x 16384 1430 us). The sums stay in shared memory, where a thread adds to its own
// columns (131 KB at 16384, one CTA of 512 threads an SM), dy and x of the next row are on their way while this one is worked
// on, the weight comes from the L1 cache twice a row. With the fold of the sums 4096 x 12288 and 4096 x 16384 take 112 and
// 134 us (LayerNorm; with the row as fp32 in registers and no prefetch 275 and 374), 92 and 110 us (RMSNorm); 403 and 537 MB take
// 62 and 82 us to copy.
constexpr int kLnWideThreads = 512, kLnWideVec = 4;
template <bool RMS>
__global__ void __launch_bounds__(kLnWideThreads, 1) normBwdWideKernel(const bf16* dy, const bf16* x, const float* mean,
                                                                       const float* rstd, const bf16* gamma, const bf16* dres,
                                                                       bf16* dx, float* partial, int M, int H) {
  releaseNext();
  awaitPrevious();
  extern __shared__ float4 lnSums[];   // [dgamma | dbeta][vector of the thread][half][thread]
  __shared__ float2 sm[2][kLnWideThreads / 32];
  const int nvec = H / 8, warp = threadIdx.x >> 5, sums = (nvec + kLnWideThreads - 1) / kLnWideThreads * 2;
  auto sum = [&](int which, int i, int half) -> float4& { return lnSums[(which * sums + i * 2 + half) * kLnWideThreads + threadIdx.x]; };
  for (int k = 0; k < sums * (RMS ? 1 : 2); ++k) lnSums[k * kLnWideThreads + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
  const uint4* gv = reinterpret_cast<const uint4*>(gamma);
  uint4 nd[kLnWideVec], nx[kLnWideVec];
  float nmu = 0.f, nrs = 0.f;
  auto fetch = [&](int row) {
    const long base = (long)row * nvec;
#pragma unroll
    for (int i = 0; i < kLnWideVec; ++i) {
      const int vi = threadIdx.x + i * kLnWideThreads;
      if (vi < nvec) {
        nd[i] = loadOrdered(reinterpret_cast<const uint4*>(dy) + base + vi);
        nx[i] = loadOrdered(reinterpret_cast<const uint4*>(x) + base + vi);
      }
    }
    if (!RMS) nmu = mean[row];
    nrs = rstd[row];
  };
  auto add = [](float4& to, const float (&v)[8], int half) {
    float4 t = to;
    t.x += v[4 * half]; t.y += v[4 * half + 1]; t.z += v[4 * half + 2]; t.w += v[4 * half + 3];
    to = t;
  };
  if (blockIdx.x < M) fetch(blockIdx.x);
  int parity = 0;
  for (int row = blockIdx.x; row < M; row += gridDim.x, parity ^= 1) {
    uint4 cd[kLnWideVec], cx[kLnWideVec], cr[kLnWideVec];
    const long base = (long)row * nvec;
#pragma unroll
    for (int i = 0; i < kLnWideVec; ++i) {
      const int vi = threadIdx.x + i * kLnWideThreads;
      cd[i] = nd[i];
      cx[i] = nx[i];
      if (dres && vi < nvec) cr[i] = loadOrdered(reinterpret_cast<const uint4*>(dres) + base + vi);
    }
    const float mu = nmu, rs = nrs;
    if (row + (int)gridDim.x < M) fetch(row + gridDim.x);
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < kLnWideVec; ++i) {
      const int vi = threadIdx.x + i * kLnWideThreads;
      if (vi < nvec) {
        float d[8], xv[8], g[8], p[8];
        unpackBf16x8(cd[i], d);
        unpackBf16x8(cx[i], xv);
        unpackBf16x8(loadOrdered(gv + vi), g);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = RMS ? xv[j] * rs : (xv[j] - mu) * rs, t = d[j] * g[j];
          if (!RMS) s1 += t;
          s2 += t * xh;
          p[j] = d[j] * xh;
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          add(sum(0, i, half), p, half);
          if (!RMS) add(sum(1, i, half), d, half);
        }
      }
    }
    if (!RMS) s1 = warpSum(s1);
    s2 = warpSum(s2);
    if ((threadIdx.x & 31) == 0) sm[parity][warp] = make_float2(s1, s2);
    __syncthreads();
    float c1 = 0.f, c2 = 0.f;
    for (int w = 0; w < kLnWideThreads / 32; ++w) { const float2 t = sm[parity][w]; c1 += t.x; c2 += t.y; }
    c1 /= H;
    c2 /= H;
#pragma unroll
    for (int i = 0; i < kLnWideVec; ++i) {
      const int vi = threadIdx.x + i * kLnWideThreads;
      if (vi < nvec) {
        float d[8], xv[8], g[8], r[8], o[8];
        unpackBf16x8(cd[i], d);
        unpackBf16x8(cx[i], xv);
        unpackBf16x8(loadOrdered(gv + vi), g);
        if (dres) unpackBf16x8(cr[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = RMS ? xv[j] * rs : (xv[j] - mu) * rs, t = d[j] * g[j];
          o[j] = rs * (RMS ? t - xh * c2 : t - c1 - xh * c2);
          if (dres) o[j] += r[j];
        }
        Vec8<bf16>::store(dx + (long)row * H + vi * 8, 8, true, o);
      }
    }
  }
  float* pg = partial + (long)blockIdx.x * (RMS ? 1 : 2) * H;
  for (int i = 0; i < sums / 2; ++i) {
    const int vi = threadIdx.x + i * kLnWideThreads;
    if (vi >= nvec) break;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      reinterpret_cast<float4*>(pg + vi * 8)[half] = sum(0, i, half);
      if (!RMS) reinterpret_cast<float4*>(pg + H + vi * 8)[half] = sum(1, i, half);
    }
  }
}

// out[c] (+)= sum_r partial[r][c]; `cols` columns, `rows` partial rows; columns from `split` on go to out2[c - split].
// A CTA owns 32 columns; its WARPS warps take every WARPS-th row (a warp reads 128 contiguous bytes of a row), four in flight,
// and fold their sums through shared memory in a fixed order. Latency is all there is: with 32 warps 296 rows are three steps for
// a warp (ten with 8 warps: 3.2 us a fold, then 2.5). Few rows leave most of 32 warps idle, and more CTAs than the 296 of that size
// that the GPU holds are a second wave, so such folds have 8 (column sum of 1 x 16384 in all: 5.5 us with 32, 3.9 with 8).
constexpr int kColReduceCols = 32;
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) colReduceKernel(const float* partial, float* out, float* out2, long split, int rows,
                                                             long cols, long stride, int accumulate) {
  releaseNext();
  awaitPrevious();
  __shared__ float red[WARPS][33];
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const long c = (long)blockIdx.x * kColReduceCols + lane;
  float s = 0.f;
  if (c < cols) {
    int r = wy;
    for (; r + 3 * WARPS < rows; r += 4 * WARPS) {
      const float a0 = partial[(long)r * stride + c], a1 = partial[(long)(r + WARPS) * stride + c];
      const float a2 = partial[(long)(r + 2 * WARPS) * stride + c], a3 = partial[(long)(r + 3 * WARPS) * stride + c];
      s += (a0 + a1) + (a2 + a3);
    }
    float t[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) t[u] = r + u * WARPS < rows ? partial[(long)(r + u * WARPS) * stride + c] : 0.f;
    s += (t[0] + t[1]) + t[2];
  }
  red[wy][lane] = s;
  __syncthreads();
  if (wy == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) t += red[w][lane];
    float* o = c < split ? out + c : out2 + (c - split);
    *o = accumulate ? *o + t : t;
  }
}

// shared with llama_kernels.cu
void launchColReduce(const float* partial, float* out, float* out2, long split, int rows, long cols, long stride, int accumulate,
                     cudaStream_t s) {
  const unsigned grid = (unsigned)((cols + kColReduceCols - 1) / kColReduceCols);
  if (rows > 64 && grid <= 2 * 148) launchAfter(colReduceKernel<32>, grid, 32 * 32, 0, s, partial, out, out2, split, rows, cols, stride, accumulate);
  else launchAfter(colReduceKernel<8>, grid, 32 * 8, 0, s, partial, out, out2, split, rows, cols, stride, accumulate);
  cocclkCountLaunches(1);
}

// ---------------------------------------------------------------- column sum of a bf16 matrix
// partial[blockIdx.y][n] = sum over this block's rows of x[m][n]
// A CTA owns 256 columns (32 lanes x 8) and `rowsPerBlock` rows; its 8 warps take every 8th row, four rows in
// flight per thread, and fold their sums through shared memory. A warp reads 512 contiguous bytes of one row.
__global__ void __launch_bounds__(256) colSumPartialKernel(const bf16* x, float* partial, int M, int N, int rowsPerBlock) {
  releaseNext();
  awaitPrevious();
  __shared__ float red[8][32][9];
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int col = (blockIdx.x * 32 + lane) * 8;
  const int r0 = blockIdx.y * rowsPerBlock;
  const int r1 = min(M, r0 + rowsPerBlock);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (col < N) {
    const bf16* base = x + col;
    int r = r0 + wy;
    for (; r + 24 < r1; r += 32) {
      float v[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) Vec8<bf16>::load(base + (long)(r + 8 * u) * N, 8, true, v[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += v[u][j];
    }
    for (; r < r1; r += 8) {
      float v[8];
      Vec8<bf16>::load(base + (long)r * N, 8, true, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[wy][lane][j] = acc[j];
  __syncthreads();
  if (wy == 0 && col < N) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += red[w][lane][j];   // fixed order: the result does not depend on scheduling
      acc[j] = s;
    }
    Vec8<float>::store(partial + (long)blockIdx.y * N + col, 8, true, acc);
  }
}

// ---------------------------------------------------------------- GELU (tanh form)
__device__ __forceinline__ float geluF(float x) {
  const float u = 0.7978845608028654f * x * (1.f + 0.044715f * x * x);
  return 0.5f * x * (1.f + tanhf(u));
}
__device__ __forceinline__ float geluGrad(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float u = k0 * x * (1.f + k1 * x * x);
  const float t = tanhf(u);
  const float du = k0 * (1.f + 3.f * k1 * x * x);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}
// y = gelu(z (+ bias)); zOut = z + bias (optional)
__global__ void __launch_bounds__(256) geluFwdKernel(const bf16* z, const bf16* bias, bf16* y, bf16* zOut, long n, int N) {
  releaseNext();
  awaitPrevious();
  for (long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (long)gridDim.x * blockDim.x * 8) {
    float v[8];
    Vec8<bf16>::load(z + i, 8, true, v);
    if (bias) {
      float b[8];
      Vec8<bf16>::load(bias + (i % N), 8, true, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += b[j];
      if (zOut) {
        Vec8<bf16>::store(zOut + i, 8, true, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __bfloat162float(__float2bfloat16_rn(v[j]));
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = geluF(v[j]);
    Vec8<bf16>::store(y + i, 8, true, v);
  }
}
// dz = dy * gelu'(z)
__global__ void __launch_bounds__(256) geluBwdKernel(const bf16* dy, const bf16* z, bf16* dz, long n) {
  releaseNext();
  awaitPrevious();
  for (long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (long)gridDim.x * blockDim.x * 8) {
    float d[8], v[8];
    Vec8<bf16>::load(dy + i, 8, true, d);
    Vec8<bf16>::load(z + i, 8, true, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) d[j] *= geluGrad(v[j]);
    Vec8<bf16>::store(dz + i, 8, true, d);
  }
}

// ---------------------------------------------------------------- cross-entropy
constexpr int kCeThreads = 1024;
constexpr int kCeMaxVec = 7;  // V <= 1024*7*8 = 57344 held in registers
constexpr int kCeNarrow = 256 * 4 * 8;

__device__ __forceinline__ void cpAsync16(uint32_t smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(g) : "memory");
}

// loss[row] = logsumexp(logits[row]) - logits[row][target]; logits <- (softmax - onehot) * gscale
// rows with target < 0 get loss 0 and a zero gradient.
//
// A row of 50304 logits fills the registers of a CTA that fills the SM, so load, two reductions, exponentials and store of a
// row followed one another with the memory idle in between (4096 rows 324 us, 824 MB: 126 us to copy). The next row is now
// on its way into shared memory while this one is worked on; a thread copies exactly the vectors it reads back, so the copy
// needs no barrier, only the thread's own wait; and only the one vector that holds the target looks at it. 217 us, bound by
// the exponentials and the two block reductions of the one CTA an SM has room for. Rows of up to 8192 logits leave most of 1024
// threads without one and take 256, four CTAs an SM, so that one row's reductions run beside another's arithmetic: 4096 x 512
// 71 us with 1024 threads, 12.5 with 256, 4096 x 8192 85 and 26 us.
template <int THREADS, int VECS>
__global__ void __launch_bounds__(THREADS) crossEntropyKernel(bf16* logits, const long* targets, float* loss,
                                                                 int M, int V, long ld, float gscale) {
  releaseNext();
  awaitPrevious();
  extern __shared__ __align__(16) uint8_t ceRow[];
  __shared__ float sm[32];
  const int nvec = V / 8;
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(ceRow) + threadIdx.x * 16;
  auto fetch = [&](int row) {
    const bf16* src = logits + (long)row * ld;
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int vi = threadIdx.x + i * THREADS;
      if (vi < nvec) cpAsync16(mine + i * THREADS * 16, src + vi * 8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (blockIdx.x < M) fetch(blockIdx.x);
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    bf16* lr = logits + (long)row * ld;
    const long tgt = targets[row];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float v[VECS][8];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int vi = threadIdx.x + i * THREADS;
      if (vi < nvec) {
        unpackBf16x8(*reinterpret_cast<const uint4*>(ceRow + (size_t)vi * 16), v[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = fmaxf(mx, v[i][j]);
      }
    }
    if (row + (int)gridDim.x < M) fetch(row + gridDim.x);
    mx = blockMax(mx, sm);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int vi = threadIdx.x + i * THREADS;
      if (vi < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { v[i][j] = __expf(v[i][j] - mx); s += v[i][j]; }
      }
    }
    s = blockSum(s, sm);
    const float inv = 1.f / s;
    const bool ignore = tgt < 0;
    if (threadIdx.x == 0 && ignore) loss[row] = 0.f;
    const int tvec = ignore ? -1 : (int)(tgt >> 3), tj = (int)(tgt & 7);   // the one vector that holds the target
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int vi = threadIdx.x + i * THREADS;
      if (vi < nvec) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = ignore ? 0.f : v[i][j] * inv * gscale;
        if (vi == tvec) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j == tj) {
              const float p = v[i][j] * inv;
              loss[row] = -__logf(fmaxf(p, 1e-37f));
              o[j] = (p - 1.f) * gscale;
            }
          }
        }
        Vec8<bf16>::store(lr + vi * 8, 8, true, o);
      }
    }
  }
}

// ---------------------------------------------------------------- vocabulary-parallel cross-entropy
// The vocabulary is sharded over the tensor-parallel ranks: a rank holds columns [vocabOffset, vocabOffset + V) of
// every logit row. Pass 1 leaves per row {local max, sum of exp(logit - local max), target logit if the target lies
// in this shard, else 0}; the ranks exchange these 16 bytes per row (an all-gather of a few hundred KB, issued by the
// caller), and pass 2 combines them (global max, rescaled sums), writes the loss and overwrites the logits with
// (softmax - onehot) * gscale. Rows with target < 0 get loss 0 and a zero gradient.
__global__ void __launch_bounds__(kCeThreads) ceStatsKernel(const bf16* logits, const long* targets, float4* stats,
                                                            int M, int V, long ld, long vocabOffset) {
  releaseNext();
  awaitPrevious();
  __shared__ float sm[32];
  const int nvec = V / 8;
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    const bf16* lr = logits + (long)row * ld;
    const long tgt = targets[row] - vocabOffset;
    float v[kCeMaxVec][8];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < kCeMaxVec; ++i) {
      const int vi = threadIdx.x + i * kCeThreads;
      if (vi < nvec) {
        Vec8<bf16>::load(lr + vi * 8, 8, true, v[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = fmaxf(mx, v[i][j]);
      }
    }
    mx = blockMax(mx, sm);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < kCeMaxVec; ++i) {
      const int vi = threadIdx.x + i * kCeThreads;
      if (vi < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) s += __expf(v[i][j] - mx);
      }
    }
    s = blockSum(s, sm);
    if (threadIdx.x == 0) {
      const bool inside = tgt >= 0 && tgt < V;
      stats[row] = make_float4(mx, s, inside ? __bfloat162float(lr[tgt]) : 0.f, inside ? 1.f : 0.f);
    }
  }
}

// statsAll: [tp][M] entries of pass 1 from every rank (this rank's included).
__global__ void __launch_bounds__(kCeThreads) ceFinishKernel(bf16* logits, const long* targets, const float4* statsAll, int tp,
                                                             float* loss, int M, int V, long ld, long vocabOffset, float gscale) {
  releaseNext();
  awaitPrevious();
  const int nvec = V / 8;
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    bf16* lr = logits + (long)row * ld;
    const long tgtGlobal = targets[row];
    const long tgt = tgtGlobal - vocabOffset;
    float gm = -INFINITY;
    for (int r = 0; r < tp; ++r) gm = fmaxf(gm, statsAll[(long)r * M + row].x);
    float S = 0.f, tl = 0.f;
    for (int r = 0; r < tp; ++r) {
      const float4 st = statsAll[(long)r * M + row];
      S += st.y * __expf(st.x - gm);
      tl += st.z;
    }
    const bool ignore = tgtGlobal < 0;
    if (threadIdx.x == 0) loss[row] = ignore ? 0.f : (__logf(S) + gm - tl);
    const float inv = 1.f / S;
#pragma unroll
    for (int i = 0; i < kCeMaxVec; ++i) {
      const int vi = threadIdx.x + i * kCeThreads;
      if (vi < nvec) {
        float v[8], o[8];
        Vec8<bf16>::load(lr + vi * 8, 8, true, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float p = __expf(v[j] - gm) * inv;
          const bool hit = (long)(vi * 8 + j) == tgt;
          o[j] = ignore ? 0.f : (p - (hit ? 1.f : 0.f)) * gscale;
        }
        Vec8<bf16>::store(lr + vi * 8, 8, true, o);
      }
    }
  }
}

// ---------------------------------------------------------------- optimizer
// AdamW on a flat shard: fp32 master/m/v, fp32 or bf16 gradients, bf16 model copy.
// gradScale (device scalar, optional) multiplies every gradient (loss scaling x clip).
template <typename G>
__global__ void __launch_bounds__(256) adamKernel(float* master, float* m, float* v, const G* grad, bf16* param,
                                                  long n, float lr, float b1, float b2, float eps, float wd,
                                                  float bc1, float bc2, const float* gradScale) {
  releaseNext();
  awaitPrevious();
  const float gs = gradScale ? *gradScale : 1.f;
  for (long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (long)gridDim.x * blockDim.x * 8) {
    const long left = n - i;
    const bool vec = left >= 8;
    float w[8], mm[8], vv[8], g[8];
    Vec8<float>::load(master + i, left, vec, w);
    Vec8<float>::load(m + i, left, vec, mm);
    Vec8<float>::load(v + i, left, vec, vv);
    Vec8<G>::load(grad + i, left, vec && aligned16(grad + i), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gj = g[j] * gs;
      mm[j] = b1 * mm[j] + (1.f - b1) * gj;
      vv[j] = b2 * vv[j] + (1.f - b2) * gj * gj;
      const float mh = mm[j] / bc1, vh = vv[j] / bc2;
      w[j] = w[j] - lr * (mh / (sqrtf(vh) + eps) + wd * w[j]);
    }
    Vec8<float>::store(master + i, left, vec, w);
    Vec8<float>::store(m + i, left, vec, mm);
    Vec8<float>::store(v + i, left, vec, vv);
    if (param) Vec8<bf16>::store(param + i, left, vec && aligned16(param + i), w);
  }
}

template <typename G>
__global__ void __launch_bounds__(256) sumSqPartialKernel(const G* x, long n, float* partial) {
  releaseNext();
  awaitPrevious();
  __shared__ float sm[32];
  float s = 0.f;
  for (long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (long)gridDim.x * blockDim.x * 8) {
    float v[8];
    const long left = n - i;
    Vec8<G>::load(x + i, left, left >= 8 && aligned16(x + i), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v[j] * v[j];
  }
  s = blockSum(s, sm);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
// out[0] (+)= sum(partial)
__global__ void __launch_bounds__(256) sumFinalKernel(const float* partial, int n, float* out, int accumulate) {
  releaseNext();
  awaitPrevious();
  __shared__ float sm[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
  s = blockSum(s, sm);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + s : s;
}
// coef = gradScaleIn * min(1, maxNorm / (sqrt(sumsq) * gradScaleIn + 1e-6))
__global__ void clipCoefKernel(const float* sumsq, float maxNorm, float gradScaleIn, float* coef, float* normOut) {
  releaseNext();
  awaitPrevious();
  const float norm = sqrtf(sumsq[0]) * gradScaleIn;
  if (normOut) normOut[0] = norm;
  float c = 1.f;
  if (maxNorm > 0.f && norm > maxNorm) c = maxNorm / (norm + 1e-6f);
  coef[0] = c * gradScaleIn;
}

// dst(fp32) += src(bf16)  /  dst = src
__global__ void __launch_bounds__(256) accumBf16Kernel(float* dst, const bf16* src, long n, int accumulate) {
  releaseNext();
  awaitPrevious();
  for (long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n; i += (long)gridDim.x * blockDim.x * 8) {
    const long left = n - i;
    const bool vec = left >= 8;
    float a[8], b[8];
    Vec8<bf16>::load(src + i, left, vec && aligned16(src + i), b);
    if (accumulate) {
      Vec8<float>::load(dst + i, left, vec, a);
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j] += a[j];
    }
    Vec8<float>::store(dst + i, left, vec, b);
  }
}

static int gridForElems(long n, int per) {
  long b = (n + per - 1) / per;
  const long cap = 148L * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace coccl

using namespace coccl;

// Threads of a norm kernel's CTA: one per 16-byte vector of a row, whole warps, at most kLnThreads.
static int normThreads(int H) {
  const int t = (H / 8 + 31) / 32 * 32;
  return t < kLnThreads ? t : kLnThreads;
}

template <bool RMS>
static int launchNormFwd(const void* x, const void* res, const void* gamma, const void* beta, void* y, void* xOut, float* mean,
                         float* rstd, int M, int H, float eps, cudaStream_t s) {
  if (H % 8 || H <= 0 || H > kLnThreads * kLnMaxVec * 8 || M <= 0) return -1;
  const int threads = normThreads(H), cap = 148 * 8 * (kLnThreads / threads), grid = M < cap ? M : cap;
  const int nv = (H / 8 + threads - 1) / threads;
  // Wide rows with nothing added: in turn, for the reason at launchNormBwd (RMSNorm early and in turn: 4096 x 5120 17.5 and 16.6 us, 1024 x
  // 16384 16.5 and 15.8; with a residual 32.8 and 33.6, 36.3 and 37.4).
  const bool early = res != nullptr || H <= 4096;
#define NORM_FWD(NV) launchIfEarly(early, normFwdKernel<NV, RMS>, grid, threads, 0, s, (const bf16*)x, (const bf16*)res, (const bf16*)gamma, \
      (const bf16*)beta, (bf16*)y, (bf16*)xOut, mean, rstd, M, H, eps)
  if (nv <= 1) NORM_FWD(1); else if (nv <= 2) NORM_FWD(2); else if (nv <= 4) NORM_FWD(4); else NORM_FWD(8);
#undef NORM_FWD
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkLayerNormBwdGrid(int M) { return M < 148 * 2 ? M : 148 * 2; }

template <bool RMS>
static int launchNormBwd(const void* dy, const void* x, const float* mean, const float* rstd, const void* gamma,
                         const void* dres, void* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int M, int H,
                         cudaStream_t s) {
  if (H % 8 || H <= 0 || H > kLnThreads * kLnMaxVec * 8 || M <= 0) return -1;
  int grid = cocclkLayerNormBwdGrid(M);
  const int threads = normThreads(H), nv = (H / 8 + threads - 1) / threads;
  // Many rows for each of a fixed number of CTAs: those that move in early share an SM with the last ones of the kernel before, and the
  // slowest SM counts (in a graph of such calls, early and in turn: 4096 x 1024 LayerNorm 19.0 and 14.7 us, 4096 x 2048 RMSNorm 21.9
  // and 16.8, 1024 x 768 7.8 and 7.2). Few rows gain (512 x 512: 5.1 and 5.5 us), and so do wide ones, which take an SM's
  // registers anyway (4096 x 4096 with a residual: 36.2 and 37.0).
  const bool early = M <= 2 * grid || H > 2048;
#define NORM_BWD(NV) launchIfEarly(early, normBwdKernel<NV, RMS>, grid, threads, 0, s, (const bf16*)dy, (const bf16*)x, mean, rstd, \
      (const bf16*)gamma, (const bf16*)dres, (bf16*)dx, scratch, M, H)
  if (nv <= 1) NORM_BWD(1);
  else if (nv <= 2) NORM_BWD(2);
  else if (nv <= 4) NORM_BWD(4);
  else {
    const int rounds = (M + 147) / 148, smem = (H / 8 + kLnWideThreads - 1) / kLnWideThreads * kLnWideThreads * (RMS ? 32 : 64);
    grid = (M + rounds - 1) / rounds;   // one CTA an SM, as many rows for each
    const cudaError_t e = cudaFuncSetAttribute(normBwdWideKernel<RMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;   // per device: a process may use several
    launchAfter(normBwdWideKernel<RMS>, grid, kLnWideThreads, smem, s, (const bf16*)dy, (const bf16*)x, mean, rstd, (const bf16*)gamma,
                                                              (const bf16*)dres, (bf16*)dx, scratch, M, H);
  }
#undef NORM_BWD
  // a scratch row is [dgamma | dbeta] (RMS: dgamma only): one fold for both
  const long cols = (RMS ? 1L : 2L) * H;
  launchColReduce(scratch, dgamma, dbeta, H, grid, cols, cols, accumulate, s);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkLayerNormFwd(const void* x, const void* res, const void* gamma, const void* beta, void* y,
                                  void* xOut, float* mean, float* rstd, int M, int H, float eps, cudaStream_t s) {
  return launchNormFwd<false>(x, res, gamma, beta, y, xOut, mean, rstd, M, H, eps, s);
}
extern "C" int cocclkLayerNormBwd(const void* dy, const void* x, const float* mean, const float* rstd,
                                  const void* gamma, const void* dres, void* dx, float* dgamma, float* dbeta,
                                  int accumulate, float* scratch, int M, int H, cudaStream_t s) {
  return launchNormBwd<false>(dy, x, mean, rstd, gamma, dres, dx, dgamma, dbeta, accumulate, scratch, M, H, s);
}
extern "C" int cocclkRmsNormFwd(const void* x, const void* res, const void* gamma, void* y, void* xOut, float* rstd, int M, int H,
                                float eps, cudaStream_t s) {
  return launchNormFwd<true>(x, res, gamma, nullptr, y, xOut, nullptr, rstd, M, H, eps, s);
}
extern "C" int cocclkRmsNormBwd(const void* dy, const void* x, const float* rstd, const void* gamma, const void* dres, void* dx,
                                float* dgamma, int accumulate, float* scratch, int M, int H, cudaStream_t s) {
  return launchNormBwd<true>(dy, x, nullptr, rstd, gamma, dres, dx, dgamma, nullptr, accumulate, scratch, M, H, s);
}

// The most row blocks of a column sum (what its scratch holds): 32 rows a block up to 64 blocks.
extern "C" int cocclkColSumBlocks(int M) { int b = (M + 31) / 32; return b > 64 ? 64 : (b < 1 ? 1 : b); }

// Row blocks: 32 rows each (a warp then has its at most four rows in flight at once) while that leaves the GPU room, down to 128
// rows where the column blocks fill it: more partial rows are more to write and fold (4096 x 4096: 7.5 us with 64 blocks, 6.6 with
// 32; 512 x 16384: 7.7 with 16, 5.9 with 4).
static int colSumBlocks(int M, int N) {
  const int most = cocclkColSumBlocks(M), least = (M + 127) / 128 < most ? (M + 127) / 128 : most, colBlocks = (N / 8 + 31) / 32;
  const int fill = 2 * 148 / colBlocks;
  return fill < least ? least : (fill > most ? most : fill);
}

extern "C" int cocclkColSum(const void* x, float* out, int accumulate, float* scratch, int M, int N, cudaStream_t s) {
  if (N % 8 || M <= 0) return -1;
  const int by = colSumBlocks(M, N);
  const int rowsPer = (M + by - 1) / by;
  dim3 grid((N / 8 + 31) / 32, by);
  launchAfter(colSumPartialKernel, grid, 256, 0, s, (const bf16*)x, scratch, M, N, rowsPer);
  launchColReduce(scratch, out, nullptr, N, by, N, N, accumulate, s);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkGeluFwd(const void* z, const void* bias, void* y, void* zOut, long n, int N, cudaStream_t s) {
  if (n % 8 || N % 8) return -1;
  launchAfter(geluFwdKernel, gridForElems(n, 2048), 256, 0, s, (const bf16*)z, (const bf16*)bias, (bf16*)y, (bf16*)zOut, n, N);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}
extern "C" int cocclkGeluBwd(const void* dy, const void* z, void* dz, long n, cudaStream_t s) {
  if (n % 8) return -1;
  launchAfter(geluBwdKernel, gridForElems(n, 2048), 256, 0, s, (const bf16*)dy, (const bf16*)z, (bf16*)dz, n);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkCrossEntropy(void* logits, const long* targets, float* loss, int M, int V, long ld,
                                  float gscale, cudaStream_t s) {
  if (V % 8 || V > kCeThreads * kCeMaxVec * 8 || ld % 8 || M <= 0) return -1;
  // the resident CTAs walk the rows (the next one prefetched): as many rows for each
  const bool narrow = V <= kCeNarrow;
  const int resident = 148 * (narrow ? 4 : 1), rounds = (M + resident - 1) / resident, grid = (M + rounds - 1) / rounds;
  if (V * 2 > 40 * 1024) {   // per device: a process may use several
    const cudaError_t e = cudaFuncSetAttribute(crossEntropyKernel<kCeThreads, kCeMaxVec>, cudaFuncAttributeMaxDynamicSharedMemorySize, kCeThreads * kCeMaxVec * 16);
    if (e != cudaSuccess) return (int)e;
  }
  if (narrow) launchAfter(crossEntropyKernel<256, 4>, grid, 256, (size_t)V * 2, s, (bf16*)logits, targets, loss, M, V, ld, gscale);
  else launchAfter(crossEntropyKernel<kCeThreads, kCeMaxVec>, grid, kCeThreads, (size_t)V * 2, s, (bf16*)logits, targets, loss, M, V, ld, gscale);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkCrossEntropyStats(const void* logits, const long* targets, float* stats, int M, int V, long ld,
                                       long vocabOffset, cudaStream_t s) {
  if (V % 8 || V > kCeThreads * kCeMaxVec * 8 || ld % 8 || M <= 0) return -1;
  const int grid = M < 148 * 2 ? M : 148 * 2;
  launchAfter(ceStatsKernel, grid, kCeThreads, 0, s, (const bf16*)logits, targets, reinterpret_cast<float4*>(stats), M, V, ld, vocabOffset);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}
extern "C" int cocclkCrossEntropyFinish(void* logits, const long* targets, const float* statsAll, int tp, float* loss, int M,
                                        int V, long ld, long vocabOffset, float gscale, cudaStream_t s) {
  if (V % 8 || V > kCeThreads * kCeMaxVec * 8 || ld % 8 || M <= 0 || tp < 1) return -1;
  const int grid = M < 148 * 2 ? M : 148 * 2;
  launchAfter(ceFinishKernel, grid, kCeThreads, 0, s, (bf16*)logits, targets, reinterpret_cast<const float4*>(statsAll), tp, loss, M, V, ld,
                                             vocabOffset, gscale);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkAdam(float* master, float* m, float* v, const void* grad, int gradIsBf16, void* param, long n,
                          float lr, float b1, float b2, float eps, float wd, int step, const float* gradScale,
                          cudaStream_t s) {
  if (n <= 0) return -1;
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  const int grid = gridForElems(n, 2048);
  if (gradIsBf16)
    launchAfter(adamKernel<bf16>, grid, 256, 0, s, master, m, v, (const bf16*)grad, (bf16*)param, n, lr, b1, b2, eps, wd, bc1, bc2, gradScale);
  else
    launchAfter(adamKernel<float>, grid, 256, 0, s, master, m, v, (const float*)grad, (bf16*)param, n, lr, b1, b2, eps, wd, bc1, bc2, gradScale);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkSumSqBlocks(long n) { return gridForElems(n, 8192); }

extern "C" int cocclkSumSq(const void* x, int isBf16, long n, float* out, int accumulate, float* scratch,
                           cudaStream_t s) {
  if (n <= 0) return -1;
  const int grid = cocclkSumSqBlocks(n);
  if (isBf16) launchAfter(sumSqPartialKernel<bf16>, grid, 256, 0, s, (const bf16*)x, n, scratch);
  else launchAfter(sumSqPartialKernel<float>, grid, 256, 0, s, (const float*)x, n, scratch);
  launchAfter(sumFinalKernel, 1, 256, 0, s, scratch, grid, out, accumulate);
  cocclkCountLaunches(2);
  return (int)cudaGetLastError();
}

extern "C" int cocclkClipCoef(const float* sumsq, float maxNorm, float gradScaleIn, float* coef, float* normOut,
                              cudaStream_t s) {
  launchAfter(clipCoefKernel, 1, 1, 0, s, sumsq, maxNorm, gradScaleIn, coef, normOut);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkAccumBf16(float* dst, const void* src, long n, int accumulate, cudaStream_t s) {
  if (n <= 0) return -1;
  launchAfter(accumBf16Kernel, gridForElems(n, 2048), 256, 0, s, dst, (const bf16*)src, n, accumulate);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Allocation-free column sum (see no_alloc_api.h). The scratch lives in the library
// image; host code must not pass the symbol itself to a kernel (on the host the name
// is only a stand-in), so the device address is looked up once per device.
// ---------------------------------------------------------------------------
namespace coccl {
constexpr int kNoAllocRows = 64;  // == upper bound of cocclkColSumBlocks
static __device__ __align__(256) float gColSumScratch[kNoAllocRows * COCCLK_NOALLOC_MAX_COLS];
static float* gColSumScratchAddr[COCCLK_NOALLOC_MAX_DEVICES];
static std::mutex gNoAllocMutex;
static thread_local char gNoAllocError[256] = "";
}  // namespace coccl

extern "C" const char* cocclkNoAllocLastError(void) { return coccl::gNoAllocError; }

extern "C" int cocclkColSumNoAlloc(const void* x, float* out, int accumulate, int M, int N, cudaStream_t s) {
  using namespace coccl;
  gNoAllocError[0] = 0;
  if (M <= 0 || N <= 0 || (N % 8) != 0) {
    snprintf(gNoAllocError, sizeof(gNoAllocError), "cocclkColSumNoAlloc: need M > 0 and N a positive multiple of 8 (M=%d N=%d)", M, N);
    return COCCLK_NOALLOC_BAD_SHAPE;
  }
  if (N > COCCLK_NOALLOC_MAX_COLS) {
    snprintf(gNoAllocError, sizeof(gNoAllocError),
             "cocclkColSumNoAlloc: N=%d exceeds the built-in scratch (max %d columns); use cocclkColSum with caller scratch",
             N, COCCLK_NOALLOC_MAX_COLS);
    return COCCLK_NOALLOC_TOO_LARGE;
  }
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= COCCLK_NOALLOC_MAX_DEVICES) {
    snprintf(gNoAllocError, sizeof(gNoAllocError), "cocclkColSumNoAlloc: device index %d is outside the address cache (0..%d)", dev,
             COCCLK_NOALLOC_MAX_DEVICES - 1);
    return COCCLK_NOALLOC_BAD_SHAPE;
  }
  float* scratch;
  {
    std::lock_guard<std::mutex> lock(gNoAllocMutex);
    if (gColSumScratchAddr[dev] == nullptr) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, gColSumScratch);  // device `dev` is current
      if (e != cudaSuccess) {
        snprintf(gNoAllocError, sizeof(gNoAllocError), "cocclkColSumNoAlloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        return (int)e;
      }
      gColSumScratchAddr[dev] = static_cast<float*>(p);
    }
    scratch = gColSumScratchAddr[dev];
  }
  const int by = colSumBlocks(M, N);  // <= kNoAllocRows
  const int rowsPer = (M + by - 1) / by;
  dim3 grid((N / 8 + 31) / 32, by);
  launchAfter(colSumPartialKernel, grid, 256, 0, s, (const bf16*)x, scratch, M, N, rowsPer);
  launchColReduce(scratch, out, nullptr, N, by, N, N, accumulate, s);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}
