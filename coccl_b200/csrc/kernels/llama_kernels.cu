// Memory-bound kernels of the Llama / Qwen layers (bf16 tensors, fp32 arithmetic): the rotation of queries and keys with
// the optional RMSNorm per head before it, straight from the packed projection, and the SwiGLU gate, forward and backward.
//
// The reference ships no model; these belong to the framework layer that drives the compressed collectives. Each kernel
// moves every byte once. As PyTorch operations the same work was about fifty launches a layer and several fp32 passes over
// the activations: at 4096 wide, 32 + 8 heads of 128 with norms, ffn 12288 and 4096 tokens 5.3 ms of device time for two
// layers forward and backward, 0.42 ms here.
#include "dependent_launch.h"
#include "launch_count.h"
#include "common.cuh"
#include "train_api.h"

namespace coccl {

using bf16 = __nv_bfloat16;

// train_kernels.cu: out[c] / out2[c - split] (+)= sum over `rows` partial rows
void launchColReduce(const float* partial, float* out, float* out2, long split, int rows, long cols, long stride, int accumulate,
                     cudaStream_t s);

// ---------------------------------------------------------------- rotation (+ RMSNorm per head)
struct RotateArgs {
  const bf16* qkv;        // [tokens][(nh + 2 nkv) D]: q heads, k heads, v heads
  bf16* q;                // [tokens][nh][D] (backward: the incoming gradients of the three, read only)
  bf16* k;                // [tokens][nkv][D]
  bf16* v;                // [tokens][nkv][D]
  bf16* dqkv;             // backward: gradient of qkv
  const float* cosT;      // [seq][D], the second half of a row repeats the first
  const float* sinT;
  const bf16* qw;         // [D] norm weights (NORM only)
  const bf16* kw;
  float* partial;         // backward, NORM: [gridDim.x][2][D] sums for the two weights
  int tokens, seq, nh, nkv, iters, perIter;
  float eps;
};

__device__ __forceinline__ void unpack8(const uint4& a, float (&v)[8]) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
template <int G>
__device__ __forceinline__ float groupSum(float x) {
#pragma unroll
  for (int o = 1; o < G; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// A thread owns 16 values of a head, eight from each half (the rotation pairs i with i + D / 2), so a head is D / 16
// neighbouring lanes and its norm a few shuffles. A CTA takes one token at a time: `perIter` heads side by side, `iters`
// times, so that the token's sines and cosines are loaded once into registers and serve every head. 4096 tokens, 48 heads of
// 128 with norms: 20 us forward (100 MB, 15 us to copy), 46 us backward (151 MB, 23 us; 127 registers, two CTAs an SM).
template <int D, bool NORM, bool BWD>
__global__ void __launch_bounds__(256) rotateKernel(const RotateArgs a) {
  releaseNext();
  awaitPrevious();
  constexpr int G = D / 16, H2 = D / 2;
  __shared__ float red[BWD && NORM ? 2 * D * 8 : 1];
  const int slot = threadIdx.x % G, hl = threadIdx.x / G;
  const int heads = a.nh + 2 * a.nkv;
  float wq[16], wk[16], dwq[16], dwk[16];
  if (NORM) {
    float t[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      unpack8(loadOrdered(reinterpret_cast<const uint4*>(a.qw + h * H2) + slot), t);
#pragma unroll
      for (int i = 0; i < 8; ++i) wq[8 * h + i] = t[i];
      unpack8(loadOrdered(reinterpret_cast<const uint4*>(a.kw + h * H2) + slot), t);
#pragma unroll
      for (int i = 0; i < 8; ++i) wk[8 * h + i] = t[i];
    }
    if (BWD) {
#pragma unroll
      for (int i = 0; i < 16; ++i) dwq[i] = dwk[i] = 0.f;
    }
  }
  for (int t = blockIdx.x; t < a.tokens; t += gridDim.x) {
    const long tr = (long)(t % a.seq) * D + slot * 8;
    float cs[8], sn[8];
    Vec8<float>::load(a.cosT + tr, 8, true, cs);
    Vec8<float>::load(a.sinT + tr, 8, true, sn);
    for (int it = 0; it < a.iters; ++it) {   // uniform over the CTA: the shuffles below need whole warps
      const int head = it * a.perIter + hl;
      const bool valid = hl < a.perIter && head < heads;
      const bool isQ = head < a.nh, isV = head >= a.nh + a.nkv;
      const long packed = ((long)t * heads + head) * D + slot * 8;
      bf16* split = isQ ? a.q + ((long)t * a.nh + head) * D
                        : (isV ? a.v + ((long)t * a.nkv + head - a.nh - a.nkv) * D : a.k + ((long)t * a.nkv + head - a.nh) * D);
      split += slot * 8;
      uint4 lo = make_uint4(0, 0, 0, 0), hi = lo, glo = lo, ghi = lo;
      if (valid) {
        if (!BWD || (NORM && !isV)) {
          lo = loadOrdered(reinterpret_cast<const uint4*>(a.qkv + packed));
          hi = loadOrdered(reinterpret_cast<const uint4*>(a.qkv + packed + H2));
        }
        if (BWD) {
          glo = loadOrdered(reinterpret_cast<const uint4*>(split));
          ghi = loadOrdered(reinterpret_cast<const uint4*>(split + H2));
        }
      }
      float x[16];
      {
        float u[8];
        unpack8(lo, u);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = u[i];
        unpack8(hi, u);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[8 + i] = u[i];
      }
      float rs = 1.f;
      if (NORM) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) ss += x[i] * x[i];
        rs = rsqrtf(groupSum<G>(ss) / D + a.eps);
      }
      float o[16];
      if (!BWD) {
        float y[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = NORM ? x[i] * rs * (isQ ? wq[i] : wk[i]) : x[i];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          o[i] = y[i] * cs[i] - y[8 + i] * sn[i];
          o[8 + i] = y[8 + i] * cs[i] + y[i] * sn[i];
        }
      } else {
        float gl[8], gh[8], d[16];
        unpack8(glo, gl);
        unpack8(ghi, gh);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          d[i] = gl[i] * cs[i] + gh[i] * sn[i];
          d[8 + i] = gh[i] * cs[i] - gl[i] * sn[i];
        }
        if (NORM) {
          float m = 0.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            x[i] *= rs;   // the normalised value
            if (valid && !isV) {
              if (isQ) dwq[i] += d[i] * x[i]; else dwk[i] += d[i] * x[i];
            }
            d[i] *= isQ ? wq[i] : wk[i];
            m += d[i] * x[i];
          }
          m = groupSum<G>(m) / D;
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = rs * (d[i] - x[i] * m);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = d[i];
        }
      }
      if (valid) {
        bf16* dst = BWD ? a.dqkv + packed : split;
        if (isV) {   // values are not rotated
          *reinterpret_cast<uint4*>(dst) = BWD ? glo : lo;
          *reinterpret_cast<uint4*>(dst + H2) = BWD ? ghi : hi;
        } else {
          float u[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) u[i] = o[i];
          Vec8<bf16>::store(dst, 8, true, u);
#pragma unroll
          for (int i = 0; i < 8; ++i) u[i] = o[8 + i];
          Vec8<bf16>::store(dst + H2, 8, true, u);
        }
      }
    }
  }
  if (BWD && NORM) {
    // sum over the heads of a warp by shuffles, over the warps through shared memory, in a fixed order
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
#pragma unroll
      for (int s = G; s < 32; s <<= 1) {
        dwq[i] += __shfl_xor_sync(0xffffffffu, dwq[i], s);
        dwk[i] += __shfl_xor_sync(0xffffffffu, dwk[i], s);
      }
      const int c = (i < 8 ? 0 : H2) + slot * 8 + (i & 7);
      if (lane < G) {
        red[warp * 2 * D + c] = dwq[i];
        red[warp * 2 * D + D + c] = dwk[i];
      }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < 2 * D; c += blockDim.x) {
      float s = 0.f;
      for (int w = 0; w < nw; ++w) s += red[w * 2 * D + c];
      a.partial[(long)blockIdx.x * 2 * D + c] = s;
    }
  }
}

// ---------------------------------------------------------------- SwiGLU
// z = [gate | up] rows of 2 F. Forward: y = silu(gate) * up. Backward: dz = [dy * up * silu'(gate) | dy * silu(gate)].
// Streaming, two (three) reads and one (two) writes of F values a row: 4096 x 12288 forward 56 us for 302 MB (46 us to
// copy), backward 85 us for 503 MB (77 us).
template <bool BWD>
__global__ void __launch_bounds__(256) swigluKernel(const bf16* z, const bf16* dy, bf16* out, int M, int F) {
  releaseNext();
  awaitPrevious();
  const int nvec = F / 8;
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nvec) return;
  for (int row = blockIdx.y; row < M; row += gridDim.y) {
    const uint4* zr = reinterpret_cast<const uint4*>(z + (long)row * 2 * F);
    float g[8], u[8], d[8], a[8], b[8];
    const uint4 rg = loadOrdered(zr + v), ru = loadOrdered(zr + nvec + v);
    uint4 rd = make_uint4(0, 0, 0, 0);
    if (BWD) rd = loadOrdered(reinterpret_cast<const uint4*>(dy + (long)row * F) + v);
    unpack8(rg, g);
    unpack8(ru, u);
    unpack8(rd, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float e = 1.f + __expf(-g[j]);
      if (!BWD) {
        a[j] = g[j] / e * u[j];
      } else {
        const float sg = 1.f / e;
        a[j] = d[j] * u[j] * sg * (1.f + g[j] * (1.f - sg));
        b[j] = d[j] * (g[j] * sg);
      }
    }
    bf16* o = out + (long)row * (BWD ? 2 * F : F) + v * 8;
    Vec8<bf16>::store(o, 8, true, a);
    if (BWD) Vec8<bf16>::store(o + F, 8, true, b);
  }
}

}  // namespace coccl

using namespace coccl;

template <bool BWD>
static int launchSwiglu(const void* z, const void* dy, void* out, int M, int F, cudaStream_t s) {
  if (M <= 0 || F <= 0 || F % 8) return -1;
  const int bx = (F / 8 + 255) / 256;
  // two waves of resident CTAs (8 of 256 threads an SM) walk the rows; fewer rows: one CTA a row and column block
  const int by = 148 * 16 / bx > 0 ? 148 * 16 / bx : 1;
  launchAfter(swigluKernel<BWD>, dim3(bx, M < by ? M : by), 256, 0, s, (const bf16*)z, (const bf16*)dy, (bf16*)out, M, F);
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}
extern "C" int cocclkSwigluFwd(const void* z, void* y, int M, int F, cudaStream_t s) { return launchSwiglu<false>(z, nullptr, y, M, F, s); }
extern "C" int cocclkSwigluBwd(const void* dy, const void* z, void* dz, int M, int F, cudaStream_t s) {
  return launchSwiglu<true>(z, dy, dz, M, F, s);
}

// The backward's grid is the number of partial rows of the weight sums: 4 CTAs an SM.
extern "C" int cocclkRotateBwdGrid(int tokens) { return tokens < 148 * 4 ? tokens : 148 * 4; }

template <bool BWD>
static int launchRotate(RotateArgs a, int D, cudaStream_t s) {
  const bool norm = a.qw != nullptr;
  if (a.tokens <= 0 || a.seq <= 0 || a.nh <= 0 || a.nkv <= 0 || (norm && a.kw == nullptr)) return -1;
  const int G = D / 16, heads = a.nh + 2 * a.nkv;
  // the heads of a token spread evenly over as few passes of the CTA as 256 threads allow
  a.iters = (heads * G + 255) / 256;
  a.perIter = (heads + a.iters - 1) / a.iters;
  const int threads = (a.perIter * G + 31) / 32 * 32;
  const int grid = BWD ? cocclkRotateBwdGrid(a.tokens) : (a.tokens < 148 * 8 ? a.tokens : 148 * 8);
  // Without norms and with several tokens a CTA the kernel gains nothing from starting early, and the CTAs that do share an SM with the
  // last ones of the kernel before (4096 tokens, 16 + 4 heads of 64, early and in turn: 6.2 and 4.8 us forward, 8.4 and 5.8 backward).
  const bool early = a.tokens <= 2 * grid;
#define ROT(DD) (norm ? launchAfter(rotateKernel<DD, true, BWD>, grid, threads, 0, s, a) \
                      : launchIfEarly(early, rotateKernel<DD, false, BWD>, grid, threads, 0, s, a))
  switch (D) {
    case 32: ROT(32); break;
    case 64: ROT(64); break;
    case 128: ROT(128); break;
    case 256: ROT(256); break;
    default: return -1;
  }
#undef ROT
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkRotateFwd(const void* qkv, void* q, void* k, void* v, const float* cosT, const float* sinT, const void* qw,
                               const void* kw, int tokens, int seq, int nh, int nkv, int D, float eps, cudaStream_t s) {
  RotateArgs a{};
  a.qkv = (const bf16*)qkv; a.q = (bf16*)q; a.k = (bf16*)k; a.v = (bf16*)v; a.cosT = cosT; a.sinT = sinT;
  a.qw = (const bf16*)qw; a.kw = (const bf16*)kw;
  a.tokens = tokens; a.seq = seq; a.nh = nh; a.nkv = nkv; a.eps = eps;
  return launchRotate<false>(a, D, s);
}

extern "C" int cocclkRotateBwd(const void* dq, const void* dk, const void* dv, const void* qkv, void* dqkv, const float* cosT,
                               const float* sinT, const void* qw, const void* kw, float* dqw, float* dkw, int accumulate,
                               float* scratch, int tokens, int seq, int nh, int nkv, int D, float eps, cudaStream_t s) {
  RotateArgs a{};
  a.qkv = (const bf16*)qkv; a.q = (bf16*)const_cast<void*>(dq); a.k = (bf16*)const_cast<void*>(dk);
  a.v = (bf16*)const_cast<void*>(dv); a.dqkv = (bf16*)dqkv; a.cosT = cosT; a.sinT = sinT; a.qw = (const bf16*)qw;
  a.kw = (const bf16*)kw; a.partial = scratch;
  a.tokens = tokens; a.seq = seq; a.nh = nh; a.nkv = nkv; a.eps = eps;
  if (qw != nullptr && (scratch == nullptr || dqw == nullptr || dkw == nullptr)) return -1;
  const int rc = launchRotate<true>(a, D, s);
  if (rc != 0 || qw == nullptr) return rc;
  launchColReduce(scratch, dqw, dkw, D, cocclkRotateBwdGrid(tokens), 2L * D, 2L * D, accumulate, s);
  return (int)cudaGetLastError();
}
