// bf16 GEMM for outputs too small to fill the GPU with 256 x 256 tiles: 128 x 64 tiles, the contraction split over the CTAs
// of a thread-block cluster.
//
// What bounds a small product is not the tensor pipe but one SM's share of L2 bandwidth: a 512 x 512 output is four pair
// tiles, eight SMs busy, each walking the whole contraction. Here the same output is 32 tiles, times up to 8 ranks of a
// cluster that take a part of the contraction each. Every rank accumulates its part in TMEM, parks the fp32 tile in its
// shared memory, and after one cluster barrier finishes 128 / ranks rows of the tile: it reads that slice from all ranks
// over distributed shared memory, in rank order (the sum does not depend on timing), applies the epilogue and stores.
//
// One tile per CTA, 4 stages of 24 KiB and 64 TMEM columns, so two CTAs share an SM and one's epilogue runs under the
// other's loads. Warp 0 = TMA producer, warp 1 = MMA issuer + TMEM owner, warps 2..5 drain TMEM; all six finish the slice.
// 512 x 512 x 2048: 8.0 us (4 ranks) against 15.7 us with pair tiles; the rule and the sweep behind it are in gemm_kernels.cu.
// Waits are bounded as in gemm_kernels.cu; every thread reaches both cluster barriers whatever happened before.
#include "gemm_epilogue.cuh"
#include "dependent_launch.h"
#include "launch_count.h"
#include "per_device.h"

namespace coccl {
using namespace sm100;

namespace small {
constexpr int BM = 128, BN = 64, BK = 64;
constexpr int kStages = 4;
constexpr int kABytes = BM * BK * 2;            // 16 KiB
constexpr int kBBytes = BN * BK * 2;            // 8 KiB
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kThreads = 192;
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

struct __align__(8) Barriers {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t tmemFull;
  uint32_t tmemBase;
  int abortFlag;
};

// byte offset of 16-byte chunk c (four fp32 columns) of row r in the parked tile: swizzled, so that 32 rows write one chunk
// each without bank conflicts
__device__ __forceinline__ uint32_t parked(int r, int c) { return (uint32_t)(r * 256 + ((c ^ (r & 15)) << 4)); }

__device__ __forceinline__ float4 ldCluster(uint32_t clusterAddr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(clusterAddr) : "memory");
  return v;
}
}  // namespace small

__global__ void __launch_bounds__(small::kThreads, 2)
gemmSmallKernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g, const int ranks) {
  using namespace small;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + kStages * kStageBytes);
  volatile int* abortFlag = &bars->abortFlag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = ranks > 1 ? (int)clusterCtaRank() : 0;
  const int numM = (g.M + BM - 1) / BM;
  const int tile = blockIdx.x / ranks, m0 = tile % numM * BM, n0 = tile / numM * BN;
  const int kBlocks = (g.K + BK - 1) / BK, per = (kBlocks + ranks - 1) / ranks;
  const int kb0 = rank * per, steps = max(0, min(kBlocks, kb0 + per) - kb0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbarInit(&bars->full[s], 1); mbarInit(&bars->empty[s], 1); }
    mbarInit(&bars->tmemFull, 1);
    bars->abortFlag = 0;
    mbarFenceInit();
    prefetchTensorMap(&tmA);
    prefetchTensorMap(&tmB);
  }
  if (warp == 1) {
    tmemAlloc(&bars->tmemBase, BN);
    tmemRelinquish();
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint32_t tmem = bars->tmemBase;
  awaitPrevious();   // nothing above reads or writes what another kernel may

  if (warp == 0) {
    {
      bool ok = true;
      int i = 0;
      for (; i < steps; ++i) {
        const int s = i % kStages;
        ok = __all_sync(0xffffffffu, mbarWait(&bars->empty[s], ((i / kStages) & 1) ^ 1, abortFlag, kWaitLimitNs)) != 0;
        if (!ok) break;
        if (electOne()) {
          uint8_t* sa = smem + s * kStageBytes;
          uint8_t* sb = sa + kABytes;
          const int k = (kb0 + i) * BK;
          mbarArriveExpectTx(&bars->full[s], kStageBytes);
          if (!g.aMN) tmaLoad2d(sa, &tmA, &bars->full[s], k, m0);
          else for (int j = 0; j < BM / 64; ++j) tmaLoad2d(sa + j * 8192, &tmA, &bars->full[s], m0 + j * 64, k);
          if (!g.bMN) tmaLoad2d(sb, &tmB, &bars->full[s], k, n0);
          else tmaLoad2d(sb, &tmB, &bars->full[s], n0, k);
        }
        __syncwarp();
      }
      if (!ok) {   // drain: give the copies already issued a bounded time to land
        for (int back = 1; back <= kStages && back <= i; ++back) {
          const int j = i - back;
          const unsigned long long start = gtimer();
          while (!mbarTryWait(&bars->full[j % kStages], (j / kStages) & 1)) {
            if (gtimer() - start > 100000000ull) break;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = makeInstrDescBf16(BM, BN, g.aMN != 0, g.bMN != 0);
    const StageDescs ops(smemAddr(smem), kABytes, g.aMN != 0, g.bMN != 0);
    for (int i = 0; i < steps; ++i) {
      const int s = i % kStages;
      if (!__all_sync(0xffffffffu, mbarWait(&bars->full[s], (i / kStages) & 1, abortFlag, kWaitLimitNs))) break;
      tcFenceAfter();
      if (electOne()) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma(tmem, ops.a(s * kStageBytes, k), ops.b(s * kStageBytes, k), idesc, (i | k) != 0 ? 1u : 0u);
        ummaCommit(&bars->empty[s]);
        if (i == steps - 1) ummaCommit(&bars->tmemFull);
      }
      __syncwarp();
    }
    __syncwarp();
  } else {
    // all MMAs done: the stages are free and take the parked tile
    const int quad = warp & 3, row = quad * 32 + lane;
    bool ok = true;
    if (steps > 0) {
      ok = mbarWait(&bars->tmemFull, 0, abortFlag, kWaitLimitNs);
      ok = __all_sync(0xffffffffu, ok) != 0;  // tcgen05.ld below needs the whole warp
    }
    if (ok) {
      tcFenceAfter();
#pragma unroll
      for (int h = 0; h < BN / 32; ++h) {
        uint32_t r[32];
        if (steps > 0) {
          tmemLd32x32(tmem + h * 32 + ((uint32_t)(quad * 32) << 16), r);
          tmemLdWait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(smem + parked(row, h * 8 + j)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
      tcFenceBefore();
    }
    __syncwarp();
  }

  // Only now: CTAs of the next kernel that move in while the main loop runs share an SM with it (products in a graph of themselves,
  // released at the start and here, and launched in turn: 512 x 512 x 2048 9.1, 7.3 and 8.2 us, 256 x 1024 x 1024 7.9, 6.3 and 7.2).
  releaseNext();
  if (ranks > 1) clusterSync(); else __syncthreads();
  if (!bars->abortFlag) {
    const int rows = BM / ranks;                          // this rank's slice of the tile
    const uint32_t base = smemAddr(smem);
    for (int i = threadIdx.x; i < rows * (BN / 8); i += kThreads) {
      const int r = rank * rows + i / (BN / 8), c = i % (BN / 8) * 2;   // two chunks: eight columns
      const int row = m0 + r, col = n0 + c * 4;
      if (row >= g.M || col >= g.N) continue;             // N is a multiple of 8: eight columns are inside or outside as a whole
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
      for (int q = 0; q < ranks; ++q) {
        float4 a, b;
        if (ranks > 1) {
          const uint32_t at = mapToCta(base, (uint32_t)q);
          a = ldCluster(at + parked(r, c));
          b = ldCluster(at + parked(r, c + 1));
        } else {
          a = *reinterpret_cast<const float4*>(smem + parked(r, c));
          b = *reinterpret_cast<const float4*>(smem + parked(r, c + 1));
        }
        v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w; v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
      }
      const long at = (long)row * g.ldc + col;
      if (g.epi == GEMM_EPI_F32 || g.epi == GEMM_EPI_F32_ACC) {
        float4* cp = reinterpret_cast<float4*>(reinterpret_cast<float*>(g.C) + at);
        if (g.epi == GEMM_EPI_F32_ACC) {
          const float4 o0 = cp[0], o1 = cp[1];
          v[0] += o0.x; v[1] += o0.y; v[2] += o0.z; v[3] += o0.w; v[4] += o1.x; v[5] += o1.y; v[6] += o1.z; v[7] += o1.w;
        }
        cp[0] = make_float4(v[0], v[1], v[2], v[3]);
        cp[1] = make_float4(v[4], v[5], v[6], v[7]);
        continue;
      }
      auto put = [](void* p, const float (&x)[8]) {
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
          o[j] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(o[0], o[1], o[2], o[3]);
      };
      if (g.epi == GEMM_EPI_BIAS || g.epi == GEMM_EPI_BIAS_GELU) {
        const uint4 bw = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(g.bias) + col);
        const uint32_t w[4] = {bw.x, bw.y, bw.z, bw.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[2 * j] += __uint_as_float(w[j] << 16);
          v[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
        }
      }
      if (g.epi == GEMM_EPI_BIAS_GELU) {
        if (g.Z != nullptr) put(reinterpret_cast<__nv_bfloat16*>(g.Z) + at, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = geluTanh(v[j]);
      }
      put(reinterpret_cast<__nv_bfloat16*>(g.C) + at, v);
    }
  }
  // nobody leaves while another rank may still read its tile
  if (ranks > 1) clusterSync(); else __syncthreads();
  if (warp == 1) {
    tcFenceAfter();
    tmemDealloc(tmem, BN);
  }
  if (threadIdx.x == 0 && bars->abortFlag && g.err) atomicExch(g.err, 0x80000003u);
}

int makeBf16TensorMap(CUtensorMap* m, const void* base, long inner, long outer, long ld, int boxInner, int boxOuter);

}  // namespace coccl

using namespace coccl;

// ranks: CTAs that share a tile's contraction (1, 2, 4 or 8).
extern "C" int cocclkGemmBf16Small(const void* A, long lda, int aMN, const void* B, long ldb, int bMN, void* C, long ldc, int M, int N,
                                   int K, int epi, const void* bias, void* Z, unsigned int* err, int ranks, cudaStream_t stream) {
  using namespace small;
  if (M <= 0 || N <= 0 || K <= 0 || (N & 7) || ((!aMN || !bMN) && (K & 7))) return -1;
  if (ranks != 1 && ranks != 2 && ranks != 4 && ranks != 8) return -1;
  if ((epi == GEMM_EPI_BIAS || epi == GEMM_EPI_BIAS_GELU) && bias == nullptr) return -1;
  CUtensorMap ta, tb;
  int rc = aMN ? makeBf16TensorMap(&ta, A, M, K, lda, 64, 64) : makeBf16TensorMap(&ta, A, K, M, lda, BK, BM);
  if (rc) return rc;
  rc = bMN ? makeBf16TensorMap(&tb, B, N, K, ldb, 64, 64) : makeBf16TensorMap(&tb, B, K, N, ldb, BK, BN);
  if (rc) return rc;
  const int smemBytes = kStages * kStageBytes + (int)sizeof(Barriers) + 1024;
  static PerDevice<bool> allowed;
  const bool* unused;
  int dev = 0;
  cudaGetDevice(&dev);
  rc = allowed.get(dev, &unused, [&](bool&) {
    return (int)cudaFuncSetAttribute(gemmSmallKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes);
  });
  if (rc) return rc;
  GemmArgs g;
  g.C = C; g.Z = Z; g.bias = bias; g.M = M; g.N = N; g.K = K; g.ldc = ldc; g.epi = epi; g.aMN = aMN; g.bMN = bMN; g.err = err;
  g.stages = kStages;
  const long tiles = (long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  if (tiles * ranks > 0x7fffffffL) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * ranks), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)ranks;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ranks > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemmSmallKernel, ta, tb, g, ranks);
  cocclkCountLaunches(1);
  return (int)e;
}
