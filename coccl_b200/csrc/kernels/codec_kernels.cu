// Launchers for the standalone codec kernels (see collective_kernels.cuh).
#include "launch_count.h"
#include "collective_kernels.cuh"
#include "kernels_api.h"
#include <type_traits>

using namespace coccl;

static_assert(sizeof(cocclkCodec) == sizeof(CodecCfg), "codec POD mismatch");

static inline CodecCfg toCfg(const cocclkCodec* c) {
  CodecCfg r;
  r.kind = c->kind; r.bits = c->bits; r.group = c->group; r.asym = c->asym; r.hadamard = c->hadamard;
  r.stochastic = c->stochastic; r.paramBytes = c->paramBytes; r.seed = c->seed;
  r.aux = c->aux; r.f0 = c->f0; r.f1 = c->f1; r.f2 = c->f2;
  return r;
}

static int smCount() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// Persistent grid for `items` tiles when an SM holds `perSm` CTAs of the kernel: exactly the resident ones. (Four an SM for
// every codec left a quarter of them waiting behind kernels that hold three; 4 x 16 Mi bf16 block-scaled FP8 decode 42.8 ->
// 35.7 us. Fewer CTAs with equal numbers of tiles are worse again: SMs then hold two or three.)
static inline int gridFor(long items, int perSm) {
  const long cap = (long)smCount() * perSm;
  return (int)(items < cap ? (items > 0 ? items : 1) : cap);
}

template <class F>
static bool dispatchDtype(int dtype, F&& f) {
  switch (dtype) {
    case kF32: f(float{}); return true;
    case kF16: f(__half{}); return true;
    case kBF16: f(__nv_bfloat16{}); return true;
  }
  return false;
}

extern "C" long cocclkEncodedChunkBytes(const cocclkCodec* codec, long count) {
  return makeChunkLayout(toCfg(codec), count, 4).totalBytes;
}

extern "C" int cocclkTileCodecSupported(const cocclkCodec* codec) { return tileCodecSupported(toCfg(codec)) ? 1 : 0; }

extern "C" int cocclkEncode(const void* in, void* out, long count, long chunks, long rawPitch, long encStride,
                            int dtype, const cocclkCodec* codec, cudaStream_t stream) {
  CodecArgs a{};
  a.in = in; a.out = out; a.count = count; a.chunks = chunks; a.reduce = 1; a.rawPitch = rawPitch;
  a.encStrideOut = encStride; a.dtype = dtype; a.codec = toCfg(codec);
  if (!tileCodecSupported(a.codec) || count <= 0 || chunks <= 0) return -1;
  const long tiles = (count + kTileElems - 1) / kTileElems;
  bool ok = dispatchCodec(a.codec, [&](auto codecTag) {
    using C = decltype(codecTag);
    const int grid = gridFor(tiles * chunks, C::kEncodeBlocks);
    dispatchDtype(dtype, [&](auto t) {
      using T = decltype(t);
      encodeKernel<T, C><<<grid, kTileThreads, 0, stream>>>(a);
    });
  });
  if (!ok) return -1;
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

// Codecs whose sums take the registers of fewer CTAs only where the tiles are one round of them (cocclkDecodeReduce).
template <class C> constexpr bool kSumsOneRound = false;
template <bool ASYM, bool HAD> constexpr bool kSumsOneRound<SdpCodec<4, ASYM, HAD, false>> = true;

extern "C" int cocclkDecodeReduce(const void* in, void* out, long count, long chunks, long reduce, long rawPitch,
                                  long encStride, int dtype, const cocclkCodec* codec, cudaStream_t stream) {
  CodecArgs a{};
  a.in = in; a.out = out; a.count = count; a.chunks = chunks; a.reduce = reduce; a.rawPitch = rawPitch;
  a.encStrideIn = encStride; a.dtype = dtype; a.codec = toCfg(codec);
  if (!tileCodecSupported(a.codec) || count <= 0 || chunks <= 0 || reduce <= 0) return -1;
  const long tiles = (count + kTileElems - 1) / kTileElems;
  bool ok = dispatchCodec(a.codec, [&](auto codecTag) {
    using C = decltype(codecTag);
    // Sums hold the words of several copies in flight and are faster with the registers of one CTA an SM fewer (8 x 4 Mi bf16,
    // asymmetric groups of 16 18.7 -> 14.7 us), unless that means one more round of tiles (8 x 3,000,008 bf16, 367 tiles: 4 bits, groups
    // of 8 14.6 us on 296 places, 12.6 on 444; block-scaled FP8 10.5 and 9.4). Since sums settle their addresses once, the difference
    // is within 0.2 us for 4-bit digits in groups of 32 and more, and for TACO. ZFP, integer work throughout: always.
    const long items = tiles * chunks, few = (long)smCount() * C::kSumBlocks, many = (long)smCount() * C::kDecodeBlocks;
    const bool sum = reduce > 1 && (a.codec.kind == kCodecZfp || items <= few ||
                                    (!kSumsOneRound<C> && (items + few - 1) / few == (items + many - 1) / many));
    // One copy goes through a kernel that loads a tile ahead. Where it only waits for its stores, aligned fp32 of a codec whose lanes
    // exchange nothing, that gains nothing and costs the last per cent of the memory's rate (8 x 8 Mi, 4 bits, groups of 128: 57.1 us
    // ahead, 55.5 without; TACO with groups of 32 68.3 and 62.4, of 128 61.9 and 66.0, of 64 no difference; misaligned 8 x 3,000,003
    // 22.9 and 24.8).
    const bool aligned = ((reinterpret_cast<uintptr_t>(out) | (uintptr_t)(rawPitch * 4)) & 15u) == 0;
    dispatchDtype(dtype, [&](auto t) {
      using T = decltype(t);
      if constexpr (HasDirectSums<C>::value) {
        const bool plain = sizeof(T) == 4 && aligned && !(C::kExchanges && a.codec.group > 32);
        if (reduce == 1 && !plain) {
          decodeKernel<T, C><<<gridFor(items, C::kDecodeBlocks), kTileThreads, 0, stream>>>(a);
          return;
        }
      }
      if (sum) decodeReduceKernel<T, C, C::kSumBlocks><<<gridFor(items, C::kSumBlocks), kTileThreads, 0, stream>>>(a);
      else decodeReduceKernel<T, C, C::kDecodeBlocks><<<gridFor(items, C::kDecodeBlocks), kTileThreads, 0, stream>>>(a);
    });
  });
  if (!ok) return -1;
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

extern "C" int cocclkDecodeReduceEncode(const void* in, void* out, long count, long chunks, long reduce,
                                        long encStrideIn, long encStrideOut, const cocclkCodec* codec,
                                        cudaStream_t stream) {
  CodecArgs a{};
  a.in = in; a.out = out; a.count = count; a.chunks = chunks; a.reduce = reduce;
  a.encStrideIn = encStrideIn; a.encStrideOut = encStrideOut; a.codec = toCfg(codec);
  if (!tileCodecSupported(a.codec) || count <= 0 || chunks <= 0 || reduce <= 0) return -1;
  const long tiles = (count + kTileElems - 1) / kTileElems;
  bool ok = dispatchCodec(a.codec, [&](auto codecTag) {
    using C = decltype(codecTag);
    const int grid = gridFor(tiles * chunks, C::kMinBlocks);
    decodeReduceEncodeKernel<C><<<grid, kTileThreads, 0, stream>>>(a);
  });
  if (!ok) return -1;
  cocclkCountLaunches(1);
  return (int)cudaGetLastError();
}

// Bounds-checked build: the error word of this translation unit's codec kernels (see codecs.cuh).
extern "C" int cocclkBoundsWordCodec(unsigned int* out, int reset) {
#ifdef COCCL_BOUNDS_CHECK
  cudaError_t e = cudaMemcpyFromSymbol(out, coccl::gBoundsWord, 8 * sizeof(unsigned int));
  if (e == cudaSuccess && reset) {
    const unsigned int zero[8] = {};
    e = cudaMemcpyToSymbol(coccl::gBoundsWord, zero, sizeof(zero));
  }
  return (int)e;
#else
  for (int i = 0; i < 8; ++i) out[i] = 0;
  (void)reset;
  return 0;
#endif
}
