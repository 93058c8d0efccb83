// Tile-level codecs shared by the standalone codec kernels, the plugin adapters and the fused
// collective kernels.
//
// A CTA of 256 threads owns a tile of 8192 consecutive elements of one chunk; every thread owns one
// aligned run of 32 elements in registers (tile_io.cuh). A codec turns a run into an `Enc` (packed payload
// words + the parameters of the groups that start in the run) that can be stored to any number of
// destinations (local scratch or a peer's receive slot), and back. encode and finish get a 2 KiB window of shared memory for
// each warp, which TACO needs; the caller has not used it since the last __syncwarp().
//
// Numerics follow the reference codecs:
//  * SDP4Bit group quantisation: symmetric scale=(2^(b-1)-1)/absmax, stored parameter 1/scale, clamp to
//    [-2^(b-1), 2^(b-1)-1]; asymmetric scale=2^b/(max-min), offset=(max+min)/2
//    (sdp4bit/includes/quantization_utils.h:126-272), int4 pairs packed low nibble first
//    (sdp4bit/includes/quantization.h:18-21), optional unnormalised 32-point Walsh-Hadamard on every
//    aligned run of 32 elements, undone by a second transform and a 1/32 factor
//    (sdp4bit/includes/fast_hadamard_transform_common.h:248-264).
//  * Stochastic rounding uses a counter-based hash keyed by (seed, element) instead of the reference's
//    per-element curand_init(clock()) (quantization_utils.h:153-174); only the error statistics are
//    comparable.
//  * MX-FP8 (no counterpart in the reference; TACO, taco/taco.cu:89-295, is its behavioural model):
//    32-element blocks, UE8M0 power-of-two scale chosen so that the block maximum does not saturate, E4M3
//    payload.
//
// Float <-> integer conversions go through the mantissa ("magic number") instead of the conversion unit:
// adding 1.5 * 2^23 to y leaves round-to-nearest-even(y) in the low mantissa bits, and OR-ing an integer
// n < 2^23 into the bits of 2^23 gives the float 2^23 + n. Packing eight 4-bit values is then one
// multiply-add chain over the raw float bits: sum(bits_i * 16^i) = C + sum(q_i * 16^i), and adding
// 0x88888888 turns the signed digits into offset-binary nibbles, which differ from two's-complement nibbles
// by the XOR 0x88888888.
//
// Encoded chunk layout (all codecs): [payload bytes of every group][parameters of every group]; the chunk is
// padded to whole groups in the encoded stream only. Encoded sizes equal the reference's (544 B for 1024
// fp32 elements in 4 chunks at g128/q4, 576 B for 16-bit inputs;
// tests/coccl-tests/src/coccl_fixed_compressor_test.cc:97-105).
#pragma once
#include "common.cuh"
#include "oracle/zfp1d_planes.h"
#include <cuda_fp8.h>
#include <type_traits>

namespace coccl {

enum CodecKind : int { kCodecSdp4bit = 0, kCodecMxfp8 = 1, kCodecRaw = 2, kCodecTaco = 3, kCodecZfp = 4 };

struct CodecCfg {
  int kind;        // CodecKind
  int bits;        // 4 | 8 (sdp4bit); 8 (mxfp8)
  int group;       // elements per group; power of two in [8, 2048] for tile kernels
  int asym;        // sdp4bit: 1 = asymmetric
  int hadamard;    // sdp4bit: 1 = H32 rotation
  int stochastic;  // 1 = stochastic rounding, 0 = round to nearest even
  int paramBytes;  // bytes of parameters per group (4 | 8 sdp4bit, 1 mxfp8, 8 taco, 0 zfp)
  uint32_t seed;
  int aux;         // taco: bit 0 = E5M2 payload, bit 1 = saturating conversion
  float f0, f1, f2;  // taco: targetRange, lambda, fp8 maximum
};
// taco: bits = 8, group = 32..512. zfp: bits = rate (bits per value), group = 4 (one block).

struct ChunkLayout {
  long count;         // elements in the chunk
  long groups;        // ceil(count / group)
  long payloadBytes;  // groups * group * bits / 8
  long totalBytes;    // payload + parameters (exact)
  long stride;        // distance between consecutive chunks (>= totalBytes)
};

__host__ __device__ inline long alignUp(long x, long a) { return (x + a - 1) / a * a; }

__host__ __device__ inline ChunkLayout makeChunkLayout(const CodecCfg& c, long count, long strideAlign) {
  ChunkLayout L;
  L.count = count;
  L.groups = (count + c.group - 1) / c.group;
  L.payloadBytes = L.groups * (long)c.group * c.bits / 8;
  L.totalBytes = alignUp(L.payloadBytes + L.groups * c.paramBytes, 4);
  L.stride = alignUp(L.totalBytes, strideAlign);
  return L;
}

// ------------------------------------------------------------------ bounds-checked build
// With -DCOCCL_BOUNDS_CHECK (libcoccl_checked.so) every access of a codec to an encoded chunk is preceded by a check
// of the byte ranges it is about to touch against the chunk's layout: the payload part must end inside the payload,
// the parameter part inside the chunk. A violation records {site, element, offending end, limit} once in a device
// word that the host reads (cocclkBoundsWord) and the access is SKIPPED, so a wrong index shows up as an error word
// and wrong numbers, never as a fault. The normal build compiles the checks away.
#ifdef COCCL_BOUNDS_CHECK
static __device__ unsigned int gBoundsWord[8];   // one per translation unit; each checked unit exports a reader
__device__ __forceinline__ bool chunkRangeOk(const ChunkLayout& L, long elem, long payloadEnd, long totalEnd, int site) {
  if (elem >= 0 && payloadEnd <= L.payloadBytes && totalEnd <= L.totalBytes && L.totalBytes <= L.stride) return true;
  if (atomicCAS(&gBoundsWord[0], 0u, 0x80000000u | (unsigned)site) == 0u) {
    gBoundsWord[1] = (unsigned)elem; gBoundsWord[2] = (unsigned)((unsigned long long)elem >> 32);
    gBoundsWord[3] = (unsigned)payloadEnd; gBoundsWord[4] = (unsigned)L.payloadBytes;
    gBoundsWord[5] = (unsigned)totalEnd; gBoundsWord[6] = (unsigned)L.totalBytes;
  }
  return false;
}
#define COCCL_CHUNK_RANGE_OK(Codec, L, c, elem, site) \
  ([&] { long pe_, te_; Codec::touched(L, c, elem, &pe_, &te_); return chunkRangeOk(L, elem, pe_, te_, site); }())
#else
#define COCCL_CHUNK_RANGE_OK(Codec, L, c, elem, site) true
#endif

// ------------------------------------------------------------------ helpers
// Two fp32 operations in one instruction (sm_100 f32x2), each rounded like its scalar form: the codecs are bound by the
// number of instructions issued, not by the arithmetic units, so a packed add or multiply-add counts half.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t p, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Unnormalised 32-point Walsh-Hadamard transform of one run, entirely in registers: the first stage inside the pairs, the
// other four on pairs.
__device__ __forceinline__ void hadamardPairs(uint64_t (&p)[16]) {   // the four stages on pairs
#pragma unroll
  for (int s = 1; s < 16; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if ((i & s) == 0) {
        const uint64_t a = p[i], b = p[i | s];
        p[i] = add2(a, b);
        p[i | s] = sub2(a, b);
      }
    }
  }
}
__device__ __forceinline__ void hadamard32(float (&v)[32]) {
  uint64_t p[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) p[i] = pack2(v[2 * i] + v[2 * i + 1], v[2 * i] - v[2 * i + 1]);
  hadamardPairs(p);
#pragma unroll
  for (int i = 0; i < 16; ++i) unpack2(p[i], v[2 * i], v[2 * i + 1]);
}

// Reduce over the `lpg` consecutive threads that share a group (lpg = group/32, a power of two <= 64).
// For lpg > 32 the CTA cooperates through `sm` (8 floats) and every thread of the CTA must call this.
struct MaxOp { static __device__ __forceinline__ float f(float a, float b) { return fmaxf(a, b); } };
struct MinOp { static __device__ __forceinline__ float f(float a, float b) { return fminf(a, b); } };

// Maxima and minima of three in one instruction; NaN counts only where all are (as in fmaxf)
__device__ __forceinline__ float maxAbs3(float a, float b, float c) {
  float d;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// max |v| of a run: four chains, so that the maximum is not one chain of 16 steps
__device__ __forceinline__ float maxAbs(const float (&v)[32]) {
  float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = maxAbs3(m[j], v[i + 2 * j], v[i + 2 * j + 1]);
  }
  return maxAbs3(maxAbs3(m[0], m[1], m[2]), m[3], 0.f);
}

template <class Op>
__device__ __forceinline__ float groupReduce(float x, int lpg, float* sm) {
  const int w = lpg < 32 ? lpg : 32;
  for (int o = 1; o < w; o <<= 1) x = Op::f(x, __shfl_xor_sync(0xffffffffu, x, o));
  if (lpg > 32) {
    const int warp = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sm[warp] = x;
    __syncthreads();
    x = Op::f(sm[warp & ~1], sm[warp | 1]);
  }
  return x;
}

constexpr float kRoundMagic = 12582912.f;          // 1.5 * 2^23
constexpr uint32_t kRoundMagicBits = 0x4B400000u;  // its bit pattern
constexpr uint32_t kIntMagicBits = 0x4B000000u;    // 2^23: OR an integer < 2^23 into the mantissa

// Random bytes k and k + 1 of a word as (u - 0.5), u = (byte + 0.5) / 256: the byte goes into the middle of the mantissa of
// 1.0 with one byte permutation (1 + byte / 2^15), and 128 x - 128.498046875 is exact.
__device__ __forceinline__ uint64_t rngCentered2(uint32_t word, int k) {
  const uint32_t a = __byte_perm(word, 0x3F800000u, 0x7604 + (k << 4)), b = __byte_perm(word, 0x3F800000u, 0x7614 + (k << 4));
  return fma2(pack2(__uint_as_float(a), __uint_as_float(b)), pack2(128.f, 128.f), pack2(-128.498046875f, -128.498046875f));
}

// Payload words of a run: 16-byte vectors, 8-byte ones where only that much alignment is left (encoded chunks of an odd
// number of groups), else words.
template <int N>
__device__ __forceinline__ void storeWords(uint8_t* p, const uint32_t (&w)[N]) {
  if (N >= 4 && aligned16(p)) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) reinterpret_cast<uint4*>(p)[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  } else if ((reinterpret_cast<uintptr_t>(p) & 7u) == 0) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q) reinterpret_cast<uint2*>(p)[q] = make_uint2(w[2 * q], w[2 * q + 1]);
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) reinterpret_cast<uint32_t*>(p)[k] = w[k];
  }
}
// __ldcg: the bytes may have been written by a peer GPU during this launch
template <int N>
__device__ __forceinline__ void loadWords(const uint8_t* p, uint32_t (&w)[N]) {
  if (N >= 4 && aligned16(p)) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
      const uint4 t = __ldcg(reinterpret_cast<const uint4*>(p) + q);
      w[4 * q] = t.x; w[4 * q + 1] = t.y; w[4 * q + 2] = t.z; w[4 * q + 3] = t.w;
    }
  } else if ((reinterpret_cast<uintptr_t>(p) & 7u) == 0) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
      const uint2 t = __ldcg(reinterpret_cast<const uint2*>(p) + q);
      w[2 * q] = t.x; w[2 * q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) w[k] = __ldcg(reinterpret_cast<const uint32_t*>(p) + k);
  }
}

// The same where the alignment is known to be 16 or 8 bytes; 4: of whole words at least.
template <int ALIGN, int N>
__device__ __forceinline__ void loadWordsBy(const uint8_t* p, uint32_t (&w)[N]) {
  if constexpr (ALIGN == 16) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
      const uint4 t = __ldcg(reinterpret_cast<const uint4*>(p) + q);
      w[4 * q] = t.x; w[4 * q + 1] = t.y; w[4 * q + 2] = t.z; w[4 * q + 3] = t.w;
    }
  } else if constexpr (ALIGN == 8) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
      const uint2 t = __ldcg(reinterpret_cast<const uint2*>(p) + q);
      w[2 * q] = t.x; w[2 * q + 1] = t.y;
    }
  } else if constexpr (N > 4) {
    loadWords(p, w);   // copies at different distances: some are better aligned
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) w[k] = __ldcg(reinterpret_cast<const uint32_t*>(p) + k);
  }
}

// Where a thread's run lies in an encoded chunk: the tile's addresses, the same in all threads, and the thread's distances from them.
struct RunAddress {
  const uint8_t *tileWords, *tileParams;
  unsigned word, param;
  __device__ __forceinline__ const uint8_t* words() const { return tileWords + word; }
  __device__ __forceinline__ const uint8_t* params() const { return tileParams + param; }
  __device__ __forceinline__ void next(long stride) { tileWords += stride; tileParams += stride; }   // the next copy
};

// ------------------------------------------------------------------ SDP4Bit
// SMALLG: groups of 8 or 16 elements (several per run, no rotation); otherwise group >= 32.
template <int BITS, bool ASYM, bool HAD, bool SMALLG>
struct SdpCodec {
  static_assert(!(HAD && SMALLG), "the rotation needs groups of at least one run");
  static constexpr int kBits = BITS;
  static constexpr int kWords = BITS;          // payload words per run
  static constexpr int kPerWord = 32 / BITS;   // elements per payload word
  static constexpr int kParams = SMALLG ? 4 : 1;
  static constexpr bool kRotated = HAD;
  static constexpr int kMinBlocks = 3;  // resident CTAs per SM the fused kernels are compiled for
  // The same for the stand-alone kernels: encode, decode of one copy, sum of several (codec_kernels.cu says which sums). Eight
  // chunks of 4 Mi bf16, one CTA an SM fewer, these, one more: 4 bits, groups of 128: encode 20.8, 20.9, 20.9 us, decode 16.9, 16.7, 16.7
  // (four chunks of 16 Mi 37.6, 33.6, 33.1); 4 bits, groups of 8: 31.3, 29.9, 31.1 and 26.9, 24.8, 22.9 (3,000,008 values 16.7, 17.0, 17.2);
  // 8 bits, asymmetric groups of 8, whose parameters do not fit 80 registers beside a run: 36.5, 37.4, 40.8 and 39.3, 30.9, 34.3.
  static constexpr int kEncodeBlocks = SMALLG ? 3 : 4, kDecodeBlocks = BITS == 8 && SMALLG && ASYM ? 2 : 3, kSumBlocks = 2;
  static constexpr bool kExchanges = false;   // runs of neighbouring lanes through the window
  static constexpr bool kEncodeAhead = !SMALLG;   // collective_kernels.cuh: kEncodeStages
  static constexpr int kSmemFloats = 8; // shared scratch every kernel passes as `sm` (group reductions wider than a warp)
  static __device__ __forceinline__ void initShared(float*) {}
  static constexpr uint32_t kSignBits = BITS == 4 ? 0x88888888u : 0x80808080u;
  static constexpr uint32_t kPackFix = kSignBits - kRoundMagicBits * (BITS == 4 ? 0x11111111u : 0x01010101u);

  struct Enc {
    uint32_t w[kWords];
    float p0[kParams], p1[kParams];
  };

  template <bool ST>
  static __device__ __forceinline__ void quantise(const float (&v)[32], const float (&scale)[kParams],
                                                  const float (&offset)[kParams], const CodecCfg& c,
                                                  uint64_t rngElem, Enc& e) {
    constexpr float qlo = (float)(-(1 << (BITS - 1))), qhi = (float)((1 << (BITS - 1)) - 1);
    uint32_t rw[8];
    if (ST) {
      // the eight words of a run share the upper half of their counter: rngElem is a multiple of 32
      const uint32_t inner = hash32(c.seed + 0x9e3779b9u * ((uint32_t)(rngElem >> 34) + 1u)), q0 = (uint32_t)(rngElem >> 2);
#pragma unroll
      for (int k = 0; k < 8; ++k) rw[k] = hash32((q0 + k) ^ inner);
    }
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      uint32_t bits[kPerWord];
      const int pj = SMALLG ? k * kPerWord / 8 : 0;
      const uint64_t sc = pack2(scale[pj], scale[pj]);
#pragma unroll
      for (int i = 0; i < kPerWord; i += 2) {
        const int idx = k * kPerWord + i;
        uint64_t v2 = pack2(v[idx], v[idx + 1]);
        if (ASYM) v2 = sub2(v2, pack2(offset[pj], offset[pj]));
        // the product is rounded to fp32 before the rounding to an integer, as in the reference: written as a packed
        // multiply-add of +0, because the assembler contracts a packed multiply and the add behind it
        uint64_t y = fma2(v2, sc, 0ull);
        if (ST) y = add2(y, rngCentered2(rw[idx >> 2], idx & 3));
        // symmetric: |y| <= 2^(b-1)-1 by construction; asymmetric: the top of the range rounds to 2^(b-1)
        if (ASYM) {
          float lo, hi;
          unpack2(y, lo, hi);
          y = pack2(fminf(fmaxf(lo, qlo), qhi), fminf(fmaxf(hi, qlo), qhi));
        }
        float lo, hi;
        unpack2(add2(y, pack2(kRoundMagic, kRoundMagic)), lo, hi);
        bits[i] = __float_as_uint(lo);
        bits[i + 1] = __float_as_uint(hi);
      }
      uint32_t acc = bits[kPerWord - 1];
#pragma unroll
      for (int i = kPerWord - 2; i >= 0; --i) acc = acc * (1u << BITS) + bits[i];
      e.w[k] = (acc + kPackFix) ^ kSignBits;
    }
  }

  static __device__ __forceinline__ void params(float mx, float mn, float& scale, float& offset, float& p0, float& p1) {
    constexpr float qmax = (float)((1 << (BITS - 1)) - 1);
    if (!ASYM) {
      scale = (mx == 0.f) ? 1.f : qmax / mx;
      offset = 0.f;
    } else {
      const float range = mx - mn;
      scale = (range == 0.f) ? 1.f : (float)(1 << BITS) / range;
      offset = 0.5f * (mx + mn);
    }
    p0 = 1.f / scale;
    p1 = offset;
  }

  // v: the run of this thread (zero beyond the chunk). `rotate=false` when v is already in the rotated
  // domain. rngElem = message-wide element index of v[0] (keys the rounding RNG).
  static __device__ __forceinline__ Enc encode(float (&v)[32], const CodecCfg& c, bool rotate, float* sm,
                                               uint64_t rngElem, uint4* /*win*/ = nullptr) {
    if (HAD && rotate) hadamard32(v);
    Enc e;
    float scale[kParams], offset[kParams];
    if (!SMALLG) {
      float mx, mn = 0.f;
      if (!ASYM) {
        mx = groupReduce<MaxOp>(maxAbs(v), c.group >> 5, sm);
      } else {
        mx = v[0]; mn = v[0];
#pragma unroll
        for (int i = 0; i < 32; i += 2) { mx = max3(mx, v[i], v[i + 1]); mn = min3(mn, v[i], v[i + 1]); }
        mx = groupReduce<MaxOp>(mx, c.group >> 5, sm);
        mn = groupReduce<MinOp>(mn, c.group >> 5, sm);
      }
      params(mx, mn, scale[0], offset[0], e.p0[0], e.p1[0]);
    } else {
      float mx[4], mn[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!ASYM) {
          mx[j] = 0.f; mn[j] = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) mx[j] = fmaxf(mx[j], fabsf(v[8 * j + i]));
        } else {
          mx[j] = v[8 * j]; mn[j] = v[8 * j];
#pragma unroll
          for (int i = 1; i < 8; ++i) { mx[j] = fmaxf(mx[j], v[8 * j + i]); mn[j] = fminf(mn[j], v[8 * j + i]); }
        }
      }
      if (c.group == 16) {
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          mx[j] = mx[j + 1] = fmaxf(mx[j], mx[j + 1]);
          mn[j] = mn[j + 1] = fminf(mn[j], mn[j + 1]);
        }
      }
#pragma unroll
      for (int j = 0; j < kParams; ++j) params(mx[j], mn[j], scale[j], offset[j], e.p0[j], e.p1[j]);
    }
    if (c.stochastic) quantise<true>(v, scale, offset, c, rngElem, e);
    else quantise<false>(v, scale, offset, c, rngElem, e);
    return e;
  }

  // Exclusive ends of the payload bytes and of the parameter bytes that store / fetch touch for the run at `elem`
  // (0 when the run lies in the padding and nothing is touched); used by the bounds-checked build.
  static __device__ __forceinline__ void touched(const ChunkLayout& L, const CodecCfg& c, long elem, long* payloadEnd, long* totalEnd) {
    const int gs = 31 - __clz(c.group);
    const long padded = L.groups << gs;
    if (elem >= padded) { *payloadEnd = 0; *totalEnd = 0; return; }
    const long last = elem + 32 < padded ? elem + 32 : padded;
    *payloadEnd = last * BITS / 8;
    long g = (last - 1) >> gs;
    if (g >= L.groups) g = L.groups - 1;
    *totalEnd = L.payloadBytes + (g + 1) * c.paramBytes;
  }

  // elem = chunk-relative index of the run's first element
  static __device__ __forceinline__ void store(const Enc& e, uint8_t* chunk, const ChunkLayout& L,
                                               const CodecCfg& c, long elem) {
    const int gs = 31 - __clz(c.group);  // the group size is a power of two
    const long padded = L.groups << gs;
    if (elem >= padded) return;
    uint8_t* pw = chunk + elem * BITS / 8;
    if (elem + 32 <= padded) {
      storeWords(pw, e.w);
    } else {
#pragma unroll
      for (int k = 0; k < kWords; ++k)
        if (elem + k * kPerWord < padded) reinterpret_cast<uint32_t*>(pw)[k] = e.w[k];
    }
    uint8_t* pbase = chunk + L.payloadBytes;
    if (!SMALLG) {
      if ((elem & (c.group - 1)) == 0) {
        float* pp = reinterpret_cast<float*>(pbase + (elem >> gs) * c.paramBytes);
        pp[0] = e.p0[0];
        if (c.paramBytes == 8) pp[1] = e.p1[0];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long ge = elem + 8 * j;
        if ((ge & (c.group - 1)) == 0 && ge < padded) {
          float* pp = reinterpret_cast<float*>(pbase + (ge >> gs) * c.paramBytes);
          pp[0] = e.p0[j];
          if (c.paramBytes == 8) pp[1] = e.p1[j];
        }
      }
    }
  }

  // Encoded run as fetched from memory; `accumulate` dequantises it. Splitting the two lets a reduction
  // keep the loads of several sources in flight.
  struct Raw {
    uint32_t w[kWords];
    float inv[kParams], off[kParams];
    uint32_t magic;
    bool valid;
  };
  // The bits of 2^23 as a value that the compiler cannot see: a logical instruction takes one constant, the mask, and splits in
  // two where the other operand is a constant too (92 and 65 integer instructions a run and copy).
  static __device__ __forceinline__ uint32_t opaqueMagic(const CodecCfg& c) { return kIntMagicBits + ((uint32_t)c.bits >> 8); }
  static constexpr int kBatch = SMALLG || BITS == 8 ? 2 : 4;   // copies whose loads are in flight together

  // `mul` scales the dequantised values (a power of two: exact); decoders that leave the rotated domain
  // right afterwards pass 1/32 here instead of multiplying all 32 outputs.
  static __device__ __forceinline__ Raw fetch(const uint8_t* chunk, const ChunkLayout& L, const CodecCfg& c, long elem,
                                              float mul, const float* /*sm*/ = nullptr) {
    Raw r;
    const int gs = 31 - __clz(c.group);
    const long padded = L.groups << gs;
    r.magic = opaqueMagic(c);
    r.valid = elem < padded;
    if (!r.valid) return r;
    const uint8_t* pw = chunk + elem * BITS / 8;
    if (elem + 32 <= padded) {
      loadWords(pw, r.w);
    } else {
#pragma unroll
      for (int k = 0; k < kWords; ++k)
        r.w[k] = (elem + k * kPerWord < padded) ? __ldcg(reinterpret_cast<const uint32_t*>(pw) + k) : 0u;
    }
    const uint8_t* pbase = chunk + L.payloadBytes;
#pragma unroll
    for (int j = 0; j < kParams; ++j) {
      long g = (elem + 8 * j) >> gs;
      if (g >= L.groups) g = L.groups - 1;
      const float* pp = reinterpret_cast<const float*>(pbase + g * c.paramBytes);
      r.inv[j] = __ldcg(pp) * mul;
      r.off[j] = ASYM ? __ldcg(pp + 1) * mul : 0.f;
    }
    return r;
  }

  // Dequantise the run (still rotated when HAD) and ADD it into acc.
  //
  // A digit becomes a float by OR-ing it, where it stands in its half-word, into the mantissa of 2^23 and subtracting 2^23
  // plus the sign offset: exactly 16^i (q - 8) for nibble i < 4, and the power of 16 moves into the multiplier, so one
  // logical instruction per value and two packed ones per pair are all, and both half-words share two pairs of multipliers.
  // Moving the power is exact unless the scaled parameter leaves the normal range: such groups (|values| < 1e-32) shift
  // instead.
  static __device__ __forceinline__ void accumulate(const Raw& r, float (&acc)[32]) {
    if (!r.valid) return;
    addRun(r.w, r.inv, r.off, r.magic, acc);
  }
  static __device__ __forceinline__ void addRun(const uint32_t (&w)[kWords], const float (&inv)[kParams], const float (&off)[kParams],
                                                uint32_t magic, float (&acc)[32]) {
    if constexpr (BITS == 4) {
      bool tiny = false;
#pragma unroll
      for (int j = 0; j < kParams; ++j) tiny = tiny || !(inv[j] >= 7.8e-34f);   // 2^-110; NaN counts as tiny
      if (tiny) { accumulateShifted(w, inv, off, acc); return; }
      uint64_t m01 = 0, m23 = 0;
#pragma unroll
      for (int k = 0; k < kWords; ++k) {
        const int pj = SMALLG ? k * kPerWord / 8 : 0;   // the eight values of a word lie in one group
        if (SMALLG || k == 0) {
          m01 = pack2(inv[pj], inv[pj] * 0x1p-4f);
          m23 = pack2(inv[pj] * 0x1p-8f, inv[pj] * 0x1p-12f);
        }
        const uint32_t x = w[k] ^ kSignBits, y = x >> 16;   // offset-binary digits: q + 8
        const int b = k * kPerWord;
        add(digits2((x & 0xfu) | magic, (x & 0xf0u) | magic), offs2(0, 1), m01, off[pj], acc[b], acc[b + 1]);
        add(digits2((x & 0xf00u) | magic, (x & 0xf000u) | magic), offs2(2, 3), m23, off[pj], acc[b + 2], acc[b + 3]);
        add(digits2((y & 0xfu) | magic, (y & 0xf0u) | magic), offs2(0, 1), m01, off[pj], acc[b + 4], acc[b + 5]);
        add(digits2((y & 0xf00u) | magic, (y & 0xf000u) | magic), offs2(2, 3), m23, off[pj], acc[b + 6], acc[b + 7]);
      }
    } else {
      accumulateShifted(w, inv, off, acc);
    }
  }
  static __device__ __forceinline__ uint64_t digits2(uint32_t a, uint32_t b) {
    return pack2(__uint_as_float(a), __uint_as_float(b));
  }
  static __device__ __forceinline__ uint64_t offs2(int i, int j) {
    return pack2(8388608.f + (float)(8u << (4 * i)), 8388608.f + (float)(8u << (4 * j)));
  }
  static __device__ __forceinline__ void add(uint64_t digits, uint64_t offs, uint64_t mul, float off, float& lo, float& hi) {
    const uint64_t f = sub2(digits, offs), a = pack2(lo, hi);
    unpack2(ASYM ? add2(a, fma2(f, mul, pack2(off, off))) : fma2(f, mul, a), lo, hi);
  }
  static __device__ __forceinline__ void accumulateShifted(const uint32_t (&w)[kWords], const float (&inv)[kParams],
                                                           const float (&off)[kParams], float (&acc)[32]) {
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      const uint32_t x = w[k] ^ kSignBits;  // offset-binary digits: q + 2^(b-1)
      const int pj = SMALLG ? k * kPerWord / 8 : 0;
      const uint64_t mul = pack2(inv[pj], inv[pj]);
#pragma unroll
      for (int i = 0; i < kPerWord; i += 2) {
        const int idx = k * kPerWord + i;
        if (BITS == 4) add(digits2(((x >> (4 * i)) & 0xfu) | kIntMagicBits, ((x >> (4 * i + 4)) & 0xfu) | kIntMagicBits), offs2(0, 0), mul, off[pj],
                           acc[idx], acc[idx + 1]);
        else add(pack2(__uint_as_float(__byte_perm(x, kIntMagicBits, 0x7650 + i)), __uint_as_float(__byte_perm(x, kIntMagicBits, 0x7651 + i))),
                 pack2(8388736.f, 8388736.f), mul, off[pj], acc[idx], acc[idx + 1]);
      }
    }
  }

  // Sum of n copies whose runs and parameters start at pw and pp, `stride` bytes apart, all aligned to ALIGN bytes. Alignment
  // and addresses are settled once per run instead of once per copy. Sums of eight copies with groups of 128, 4 bits, rotated:
  // 224 -> 146 instructions a run and copy; 8 x 8 Mi fp32 24.6 -> 16.7 us, 8 x 5,000,003 bf16 16.2 -> 11.5 us.
  static constexpr bool kDirectSums = !SMALLG;
  template <int ALIGN, int B>
  static __device__ __forceinline__ void sumBatches(const uint8_t*& pw, const uint8_t*& pp, long stride, int& n, float mul, uint32_t magic,
                                                    float (&acc)[32]) {
#pragma unroll 1
    while (n >= B) {
      uint32_t w[B][kWords];
      float inv[B][1], off[B][1];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        loadWordsBy<ALIGN>(pw, w[j]);
        inv[j][0] = __ldcg(reinterpret_cast<const float*>(pp));
        off[j][0] = ASYM ? __ldcg(reinterpret_cast<const float*>(pp) + 1) : 0.f;
        pw += stride;
        pp += stride;
      }
#pragma unroll
      for (int j = 0; j < B; ++j) {
        inv[j][0] *= mul;
        off[j][0] *= mul;
        addRun(w[j], inv[j], off[j], magic, acc);
      }
      n -= B;
    }
  }
  template <int ALIGN>
  static __device__ __forceinline__ void sumAligned(const uint8_t* pw, const uint8_t* pp, long stride, int n, float mul, uint32_t magic,
                                                    float (&acc)[32]) {
    if constexpr (kBatch >= 4) sumBatches<ALIGN, 4>(pw, pp, stride, n, mul, magic, acc);
    sumBatches<ALIGN, 2>(pw, pp, stride, n, mul, magic, acc);
    sumBatches<ALIGN, 1>(pw, pp, stride, n, mul, magic, acc);
  }
  // A group has at least one run, so a run lies wholly in the chunk's groups or wholly behind them.
  static __device__ __forceinline__ bool runAt(const uint8_t* base, const ChunkLayout& L, const CodecCfg& c, long elem, const uint8_t*& pw,
                                               const uint8_t*& pp) {
    const int gs = 31 - __clz(c.group);
    const long e0 = elem - (long)threadIdx.x * kElemsPerThread;   // of the tile: uniform, so the addresses are base + lane offset
    pw = base + e0 * BITS / 8 + threadIdx.x * (kElemsPerThread * BITS / 8);
    pp = base + L.payloadBytes + (e0 >> gs) * c.paramBytes + ((threadIdx.x * kElemsPerThread) >> gs) * c.paramBytes;
    return elem < (L.groups << gs);
  }
  static __device__ __forceinline__ void sum(const uint8_t* base, long stride, int n, const ChunkLayout& L, const CodecCfg& c, long elem,
                                             float mul, bool aligned, bool /*spread*/, float (&acc)[32]) {
    const uint8_t *pw, *pp;
    if (!runAt(base, L, c, elem, pw, pp)) return;
    const uint32_t magic = opaqueMagic(c);
    if (aligned) sumAligned<16>(pw, pp, stride, n, mul, magic, acc);
    else if (((reinterpret_cast<uintptr_t>(base) | (uintptr_t)stride) & 7u) == 0) sumAligned<8>(pw, pp, stride, n, mul, magic, acc);
    else sumAligned<4>(pw, pp, stride, n, mul, magic, acc);
  }
  // One copy, its loads apart from its use, so that those of the next tile can be on their way (words behind the chunk: zero).
  struct Ahead {
    uint32_t w[kWords];
    float inv[1], off[1];
  };
  static __device__ __forceinline__ Ahead ahead(const uint8_t* base, const ChunkLayout& L, const CodecCfg& c, long elem) {
    Ahead r = {};
    const uint8_t *pw, *pp;
    if (!runAt(base, L, c, elem, pw, pp) || !COCCL_CHUNK_RANGE_OK(SdpCodec, L, c, elem, 2)) return r;
    loadWords(pw, r.w);
    r.inv[0] = __ldcg(reinterpret_cast<const float*>(pp));
    r.off[0] = ASYM ? __ldcg(reinterpret_cast<const float*>(pp) + 1) : 0.f;
    return r;
  }
  static __device__ __forceinline__ void addAhead(const Ahead& r, const CodecCfg& c, float mul, float (&acc)[32]) {
    const float inv[1] = {r.inv[0] * mul}, off[1] = {r.off[0] * mul};
    addRun(r.w, inv, off, opaqueMagic(c), acc);
  }

  // Leave the rotated domain (after any reduction: the transform is linear). The 1/32 of the inverse
  // transform was applied by fetch (kFinishScale).
  static __device__ __forceinline__ float finishScale(const CodecCfg&) { return HAD ? 1.f / 32.f : 1.f; }
  static __device__ __forceinline__ void finish(float (&v)[32], const CodecCfg&, uint4* /*win*/ = nullptr) {
    if (HAD) hadamard32(v);
  }
};

// ------------------------------------------------------------------ MX-FP8
// One 32-element block per run: the scale needs no cross-lane traffic at all.
struct MxFp8Codec {
  static constexpr int kBits = 8;
  static constexpr int kWords = 8;
  static constexpr bool kRotated = false;
  static constexpr int kMinBlocks = 3;
  // 4 x 16 Mi bf16: decode 39.2 us with two, 35.7 with three, 39.4 with four; encode 35.4 with three, 34.4 with four, 33.3 with five
  // (8 x 3,000,008 fp32 22.1, 21.2, 22.9)
  static constexpr int kEncodeBlocks = 4, kDecodeBlocks = 3, kSumBlocks = 2;
  static constexpr bool kExchanges = false;
  static constexpr bool kEncodeAhead = false;
  static constexpr int kSmemFloats = 8;
  static __device__ __forceinline__ void initShared(float*) {}

  struct Enc {
    uint32_t w[8];
    uint32_t scaleByte;
  };

  static __device__ __forceinline__ Enc encode(float (&v)[32], const CodecCfg& /*c*/, bool /*rotate*/, float* /*sm*/,
                                               uint64_t /*rngElem*/, uint4* /*win*/ = nullptr) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) m = fmaxf(m, fabsf(v[i]));
    // UE8M0: smallest power of two s with m / s <= 448.
    int biased = 0;
    if (m > 0.f && m < INFINITY) {
      const float r = m * (1.f / 448.f);
      const uint32_t rb = __float_as_uint(r);
      int ex = (int)((rb >> 23) & 0xff);
      if (rb & 0x7fffffu) ex += 1;
      biased = max(0, min(254, ex));
    }
    // 2^-(biased-127) as a float: exponent field 254 - biased (denormal-safe for biased in [1,253]).
    const int invExp = 254 - biased;
    const float inv = invExp > 0 ? __uint_as_float((uint32_t)invExp << 23) : __uint_as_float(0x00400000u);  // 2^-127
    Enc e;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * k] * inv, v[4 * k + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * k + 2] * inv, v[4 * k + 3] * inv), __NV_SATFINITE, __NV_E4M3);
      e.w[k] = lo | (hi << 16);
    }
    e.scaleByte = (uint32_t)biased;
    return e;
  }

  static __device__ __forceinline__ void touched(const ChunkLayout& L, const CodecCfg&, long elem, long* payloadEnd, long* totalEnd) {
    if (elem >= L.groups * 32) { *payloadEnd = 0; *totalEnd = 0; return; }
    *payloadEnd = elem + 32;
    *totalEnd = elem / 32 == L.groups - 1 ? L.totalBytes : L.payloadBytes + elem / 32 + 1;
  }

  static __device__ __forceinline__ void store(const Enc& e, uint8_t* chunk, const ChunkLayout& L, const CodecCfg& /*c*/,
                                               long elem) {
    if (elem >= L.groups * 32) return;
    uint8_t* pw = chunk + elem;
    storeWords(pw, e.w);
    chunk[L.payloadBytes + elem / 32] = (uint8_t)e.scaleByte;
    if (elem / 32 == L.groups - 1)   // up to three bytes that round the chunk up to whole words
      for (long i = L.payloadBytes + L.groups; i < L.totalBytes; ++i) chunk[i] = 0;
  }

  struct Raw {
    uint32_t w[8];
    uint32_t biased;
    bool valid;
  };
  static __device__ __forceinline__ void accumulate(const Raw& r, float (&acc)[32]) {
    if (!r.valid) return;
    addRun(r.w, r.biased, acc);
  }
  static __device__ __forceinline__ void addRun(const uint32_t (&w)[8], uint32_t biased, float (&acc)[32]) {
    const float scale = biased > 0 ? __uint_as_float(biased << 23) : __uint_as_float(0x00400000u);
    const uint64_t s2 = pack2(scale, scale);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[k >> 1] >> (16 * (k & 1))), __NV_E4M3);
      const float2 f = __half22float2(*reinterpret_cast<__half2*>(&hr));
      unpack2(fma2(pack2(f.x, f.y), s2, pack2(acc[2 * k], acc[2 * k + 1])), acc[2 * k], acc[2 * k + 1]);
    }
  }

  static constexpr bool kDirectSums = true;
  template <int ALIGN, int B>
  static __device__ __forceinline__ void sumBatches(RunAddress& r, long stride, int& n, float (&acc)[32]) {
#pragma unroll 1
    while (n >= B) {
      uint32_t w[B][8], biased[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        loadWordsBy<ALIGN>(r.words(), w[j]);
        biased[j] = __ldcg(r.params());
        r.next(stride);
      }
#pragma unroll
      for (int j = 0; j < B; ++j) addRun(w[j], biased[j], acc);
      n -= B;
    }
  }
  static __device__ __forceinline__ void sum(const uint8_t* base, long stride, int n, const ChunkLayout& L, const CodecCfg& /*c*/, long elem,
                                             float /*mul*/, bool aligned, bool /*spread*/, float (&acc)[32]) {
    if (elem >= L.groups * 32) return;
    const long e0 = elem - (long)threadIdx.x * kElemsPerThread;
    RunAddress r = {base + e0, base + L.payloadBytes + e0 / 32, threadIdx.x * 32u, threadIdx.x};
    if (aligned) {
      sumBatches<16, 2>(r, stride, n, acc);
      sumBatches<16, 1>(r, stride, n, acc);
    } else {
      sumBatches<4, 2>(r, stride, n, acc);
      sumBatches<4, 1>(r, stride, n, acc);
    }
  }
  // One copy, its loads apart from its use (behind the chunk: zeros).
  struct Ahead {
    uint32_t w[8], biased;
  };
  static __device__ __forceinline__ Ahead ahead(const uint8_t* base, const ChunkLayout& L, const CodecCfg& c, long elem) {
    Ahead r = {};
    if (elem >= L.groups * 32 || !COCCL_CHUNK_RANGE_OK(MxFp8Codec, L, c, elem, 2)) return r;
    loadWords(base + elem, r.w);
    r.biased = __ldcg(base + L.payloadBytes + elem / 32);
    return r;
  }
  static __device__ __forceinline__ void addAhead(const Ahead& r, const CodecCfg& /*c*/, float /*mul*/, float (&acc)[32]) { addRun(r.w, r.biased, acc); }

  static __device__ __forceinline__ float finishScale(const CodecCfg&) { return 1.f; }
  static __device__ __forceinline__ void finish(float (&)[32], const CodecCfg&, uint4* /*win*/ = nullptr) {}
};

// ------------------------------------------------------------------ TACO
// Adaptive FP8 with a Walsh-Hadamard transform over the whole group (reference numerics: taco/taco.cu:118-218):
//   ada = clamp(fp8max * rsqrt(mean(x^2) + lambda), 1e-3, 1e3);  y = H_G(x * ada) / sqrt(G);
//   qs = clamp(max|y| / targetRange, 1e-12, 1e6);  code = fp8(clamp(y / qs, +-448));  x^ = H_G(code * qs) / sqrt(G) / ada
// Chunk layout as the reference's: [one fp8 byte per value of every (padded) group][groups x f32 qs][groups x f32 ada].
// A group is G/32 consecutive runs, i.e. G/32 adjacent lanes of one warp: the first five butterfly stages are register work.
// For the next two, E = min(4, G/32) lanes exchange their runs through shared memory, so that each holds the same 32/E places
// of E runs (the "spread" ownership) and finds its partners in its own registers: 16 vector accesses instead of 64 shuffles
// and as many multiply-adds, and what follows (maxima, FP8, stores) is as easy there. Wider groups use shuffles for the rest.
// Groups of 128, 8 x 8 Mi fp16: encode 65.3 -> 53.7 us, sum 21.8 -> 20.8 us, re-encoding sum 24.3 -> 16.7 us; 8 x 3,000,008:
// encode 26.0 -> 22.9 us. (Groups of 64 with their one stage by shuffles: sum of 8 x 3,000,008 12.3 us, 9.2 with the exchange.)
// The group statistics are warp shuffles, so every lane of the warp must call encode() and finish() together. "Rotated domain"
// here is y / ada = H_G(x) / sqrt(G): independent of the sender's ada, so copies from different ranks add up there and one
// inverse transform serves the sum; the transform is orthonormal, so mean(x^2) for a re-encode is available without leaving the
// domain (in the order of the run ownership, in which a re-encoding sum is therefore formed).
struct TacoCodec {
  static constexpr int kBits = 8;
  static constexpr int kWords = 8;
  static constexpr bool kRotated = true;
  static constexpr int kEncodeBlocks = 4, kDecodeBlocks = 3, kSumBlocks = 2;
  static constexpr int kMinBlocks = 3;
  static constexpr bool kExchanges = true;
  static constexpr bool kEncodeAhead = true;
  static constexpr int kSmemFloats = 8;
  static __device__ __forceinline__ void initShared(float*) {}

  struct Enc {
    uint32_t w[8];
    float qs, ada;
    bool spread;
  };
  static __device__ __forceinline__ int groupShift(const CodecCfg& c) { return 31 - __clz(c.group); }  // a power of two
  template <class F>
  static __device__ __forceinline__ void byLanes(const CodecCfg& c, F&& f) {   // f(integral_constant<E>)
    if (c.group >= 128) f(std::integral_constant<int, 4>{});
    else if (c.group == 64) f(std::integral_constant<int, 2>{});
    else f(std::integral_constant<int, 1>{});
  }

  // Vector a (of four) of run r in the warp's 2 KiB window: neither the lanes that write their runs nor those that read one
  // place of several runs meet in a bank.
  static __device__ __forceinline__ int at(int r, int a) { return ((r ^ ((r >> 2) & 1)) << 2) + (a ^ ((r >> 1) & 3)); }
  // Run ownership -> spread (SPREAD) or back. Vector q of a run goes with pass q & 1; lane j of E owns the vectors j * 8 / E on.
  template <int E, bool SPREAD>
  static __device__ __forceinline__ void exchange(float (&v)[32], uint4* win) {
    const int lane = threadIdx.x & 31, j = lane & (E - 1);
    float o[32];
    auto own = [](int p, int i) { return 4 * (2 * i + p); };
    auto theirs = [](int p, int i) { return (i / (4 / E)) * (32 / E) + 4 * (2 * (i % (4 / E)) + p); };
    auto slotOf = [&](bool spread, int i) { return spread ? at(lane - j + i / (4 / E), j * (4 / E) + i % (4 / E)) : at(lane, i); };
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = SPREAD ? own(p, i) : theirs(p, i);
        win[slotOf(!SPREAD, i)] = make_uint4(__float_as_uint(v[k]), __float_as_uint(v[k + 1]), __float_as_uint(v[k + 2]), __float_as_uint(v[k + 3]));
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = SPREAD ? theirs(p, i) : own(p, i);
        const uint4 y = win[slotOf(SPREAD, i)];
        o[k] = __uint_as_float(y.x); o[k + 1] = __uint_as_float(y.y); o[k + 2] = __uint_as_float(y.z); o[k + 3] = __uint_as_float(y.w);
      }
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = o[i];
  }
  // The butterfly stages across lanes, in the spread ownership.
  template <int E>
  static __device__ __forceinline__ void lanes(float (&v)[32], int lpg) {
#pragma unroll
    for (int s = 1; s < E; s <<= 1) {
#pragma unroll
      for (int r = 0; r < E; ++r) {
        if (r & s) continue;
#pragma unroll
        for (int k = 0; k < 32 / E; k += 2) {
          const int lo = r * (32 / E) + k, hi = (r | s) * (32 / E) + k;
          const uint64_t a = pack2(v[lo], v[lo + 1]), b = pack2(v[hi], v[hi + 1]);
          unpack2(add2(a, b), v[lo], v[lo + 1]);
          unpack2(sub2(a, b), v[hi], v[hi + 1]);
        }
      }
    }
    for (int s = E; s < lpg; s <<= 1) {
      const float sign = (threadIdx.x & s) != 0 ? -1.f : 1.f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float o = __shfl_xor_sync(0xffffffffu, v[i], s);
        v[i] = fmaf(v[i], sign, o);   // upper lanes: o - v, lower lanes: o + v
      }
    }
  }
  static __device__ __forceinline__ void scaleAll(float (&v)[32], float f) {   // a packed multiply; -0 leaves the sign of zeros
    const uint64_t f2 = pack2(f, f), z2 = 0x8000000080000000ull;
#pragma unroll
    for (int i = 0; i < 32; i += 2) unpack2(fma2(pack2(v[i], v[i + 1]), f2, z2), v[i], v[i + 1]);
  }

  static __device__ __forceinline__ Enc encode(float (&v)[32], const CodecCfg& c, bool rotate, float* /*sm*/,
                                               uint64_t /*rngElem*/, uint4* win = nullptr) {
    const int lpg = c.group >> 5;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) ss = fmaf(v[i], v[i], ss);
    for (int o = 1; o < lpg; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    Enc e;
    e.ada = fminf(fmaxf(c.f2 * rsqrtf(ss / (float)c.group + c.f1), 1e-3f), 1e3f);
    e.spread = rotate;
    if (rotate) {
      // the first stage takes the product with ada along in a multiply-add
      uint64_t p[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float b = v[2 * i + 1] * e.ada;
        p[i] = pack2(fmaf(v[2 * i], e.ada, b), fmaf(v[2 * i], e.ada, -b));
      }
      hadamardPairs(p);
#pragma unroll
      for (int i = 0; i < 16; ++i) unpack2(p[i], v[2 * i], v[2 * i + 1]);
      byLanes(c, [&](auto n) {
        constexpr int E = decltype(n)::value;
        if constexpr (E > 1) exchange<E, true>(v, win);
        lanes<E>(v, lpg);
      });
      scaleAll(v, rsqrtf((float)c.group));
    } else {
      scaleAll(v, e.ada);
    }
    float m = maxAbs(v);
    for (int o = 1; o < lpg; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    e.qs = fminf(fmaxf(m / c.f0, 1e-12f), 1e6f);
    const float inv = 1.f / e.qs;
    scaleAll(v, inv);
    // Values within a rounding of +-448 are what the clamp and either conversion make 448 of; infinities, NaN (the sum of squares has
    // them too) and a range beyond +-448 take the clamp and the conversion that was asked for.
    auto convert = [&](__nv_saturation_t sat, __nv_fp8_interpretation_t fmt) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * k], v[4 * k + 1]), sat, fmt);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * k + 2], v[4 * k + 3]), sat, fmt);
        e.w[k] = lo | (hi << 16);
      }
    };
    const bool plain = m * inv <= 449.f && ss < INFINITY;
    if (!plain) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = fminf(fmaxf(v[i], -448.f), 448.f);
    }
    if (plain && (c.aux & 1) == 0) convert(__NV_SATFINITE, __NV_E4M3);
    else if (plain) convert(__NV_SATFINITE, __NV_E5M2);
    else convert((c.aux & 2) ? __NV_SATFINITE : __NV_NOSAT, (c.aux & 1) ? __NV_E5M2 : __NV_E4M3);
    return e;
  }

  static __device__ __forceinline__ void touched(const ChunkLayout& L, const CodecCfg& c, long elem, long* payloadEnd, long* totalEnd) {
    if (elem >= L.payloadBytes) { *payloadEnd = 0; *totalEnd = 0; return; }
    const int lpg = c.group >> 5, E = lpg < 4 ? lpg : 4;
    *payloadEnd = (elem | (32L * E - 1)) + 1;                                   // the runs of the lanes that exchange theirs
    *totalEnd = L.payloadBytes + (L.groups + (elem >> groupShift(c)) + 1) * 4;   // the group's scale, then its adaptive factor
  }

  // First byte of this lane's 32 / E places in the first of its E runs; the others follow 32 bytes apart.
  template <int E>
  static __device__ __forceinline__ long placesAt(long elem) {
    const int j = threadIdx.x & (E - 1);
    return elem - 32 * j + j * (32 / E);
  }

  static __device__ __forceinline__ void store(const Enc& e, uint8_t* chunk, const ChunkLayout& L, const CodecCfg& c,
                                               long elem) {
    if (elem >= L.payloadBytes) return;  // runs of the padded last group are part of the stream
    auto put = [&](auto n) {
      constexpr int E = decltype(n)::value, W = 8 / E;
      uint8_t* p = chunk + placesAt<E>(elem);
#pragma unroll
      for (int r = 0; r < E; ++r) {
        uint32_t part[W];
#pragma unroll
        for (int i = 0; i < W; ++i) part[i] = e.w[r * W + i];
        storeWords(p + 32 * r, part);
      }
    };
    if (e.spread) byLanes(c, put);
    else put(std::integral_constant<int, 1>{});
    if ((elem & (c.group - 1)) == 0) {
      float* ps = reinterpret_cast<float*>(chunk + L.payloadBytes);
      const long g = elem >> groupShift(c);
      ps[g] = e.qs;
      ps[L.groups + g] = e.ada;
    }
  }

  // acc += scale * values of the eight words
  static __device__ __forceinline__ void addRun(const uint32_t (&w)[8], float scale, bool e5m2, float (&acc)[32]) {
    const uint64_t s2 = pack2(scale, scale);
    auto add = [&](int i, __half2_raw hr) {
      const float2 f = __half22float2(*reinterpret_cast<__half2*>(&hr));
      unpack2(fma2(pack2(f.x, f.y), s2, pack2(acc[i], acc[i + 1])), acc[i], acc[i + 1]);
    };
    if (e5m2) {
#pragma unroll
      for (int k = 0; k < 16; ++k) add(2 * k, __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[k >> 1] >> (16 * (k & 1))), __NV_E5M2));
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k) add(2 * k, __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[k >> 1] >> (16 * (k & 1))), __NV_E4M3));
    }
  }
  template <int E, int ALIGN>
  static __device__ __forceinline__ void loadPlaces(const uint8_t* p, uint32_t (&w)[8]) {
    constexpr int W = 8 / E;
#pragma unroll
    for (int r = 0; r < E; ++r) {
      uint32_t part[W];
      loadWordsBy<(W >= 4 ? ALIGN : (ALIGN < 8 ? ALIGN : 8))>(p + 32 * r, part);
#pragma unroll
      for (int i = 0; i < W; ++i) w[r * W + i] = part[i];
    }
  }

  static constexpr bool kDirectSums = true;
  template <int E, int ALIGN, int B>
  static __device__ __forceinline__ void sumBatches(RunAddress& r, long groups, long stride, int& n, float mul, bool e5m2, float (&acc)[32]) {
#pragma unroll 1
    while (n >= B) {
      uint32_t w[B][8];
      float qs[B], ada[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        loadPlaces<E, ALIGN>(r.words(), w[j]);
        qs[j] = __ldcg(reinterpret_cast<const float*>(r.params()));
        ada[j] = __ldcg(reinterpret_cast<const float*>(r.params() + 4 * groups));
        r.next(stride);
      }
#pragma unroll
      for (int j = 0; j < B; ++j) addRun(w[j], qs[j] / ada[j] * mul, e5m2, acc);
      n -= B;
    }
  }
  static __device__ __forceinline__ void sum(const uint8_t* base, long stride, int n, const ChunkLayout& L, const CodecCfg& c, long elem,
                                             float mul, bool aligned, bool spread, float (&acc)[32]) {
    if (elem >= L.payloadBytes) return;
    const long e0 = elem - (long)threadIdx.x * kElemsPerThread;
    const int gs = groupShift(c);
    auto go = [&](auto lanesTag, auto alignTag) {
      constexpr int E = decltype(lanesTag)::value, ALIGN = decltype(alignTag)::value;
      RunAddress r = {base + e0, base + L.payloadBytes + (e0 >> gs) * 4, (unsigned)placesAt<E>((long)threadIdx.x * kElemsPerThread),
                      ((threadIdx.x * kElemsPerThread) >> gs) * 4u};
      sumBatches<E, ALIGN, 2>(r, L.groups, stride, n, mul, (c.aux & 1) != 0, acc);
      sumBatches<E, ALIGN, 1>(r, L.groups, stride, n, mul, (c.aux & 1) != 0, acc);
    };
    const uintptr_t address = reinterpret_cast<uintptr_t>(base) | (uintptr_t)stride;
    auto byAlign = [&](auto lanesTag) {   // four lanes' places are eight bytes, others' whole vectors
      constexpr int E = decltype(lanesTag)::value;
      if (E != 4 && aligned) go(lanesTag, std::integral_constant<int, 16>{});
      else if (E != 1 && (address & 7u) == 0) go(lanesTag, std::integral_constant<int, 8>{});
      else go(lanesTag, std::integral_constant<int, 4>{});   // of one lane: 32 bytes, as their address allows
    };
    if (spread) byLanes(c, byAlign);
    else byAlign(std::integral_constant<int, 1>{});
  }
  // One copy in the spread ownership, its loads apart from its use (behind the chunk: zeros).
  struct Ahead {
    uint32_t w[8];
    float qs, ada;
  };
  static __device__ __forceinline__ Ahead ahead(const uint8_t* base, const ChunkLayout& L, const CodecCfg& c, long elem) {
    Ahead r = {};
    r.ada = 1.f;
    if (elem >= L.payloadBytes || !COCCL_CHUNK_RANGE_OK(TacoCodec, L, c, elem, 2)) return r;
    byLanes(c, [&](auto n) {
      constexpr int E = decltype(n)::value;
      const uint8_t* p = base + placesAt<E>(elem);
      const uintptr_t address = reinterpret_cast<uintptr_t>(base);
      if (E != 4 && (address & 15u) == 0) loadPlaces<E, 16>(p, r.w);
      else if (E != 1 && (address & 7u) == 0) loadPlaces<E, 8>(p, r.w);
      else loadPlaces<E, 4>(p, r.w);
    });
    const float* ps = reinterpret_cast<const float*>(base + L.payloadBytes) + (elem >> groupShift(c));
    r.qs = __ldcg(ps);
    r.ada = __ldcg(ps + L.groups);
    return r;
  }
  static __device__ __forceinline__ void addAhead(const Ahead& r, const CodecCfg& c, float mul, float (&acc)[32]) {
    addRun(r.w, r.qs / r.ada * mul, (c.aux & 1) != 0, acc);
  }

  static __device__ __forceinline__ float finishScale(const CodecCfg& c) { return rsqrtf((float)c.group); }
  static __device__ __forceinline__ void finish(float (&v)[32], const CodecCfg& c, uint4* win = nullptr) {
    byLanes(c, [&](auto n) {
      constexpr int E = decltype(n)::value;
      lanes<E>(v, c.group >> 5);
      if constexpr (E > 1) exchange<E, false>(v, win);
    });
    hadamard32(v);
  }
};

// ------------------------------------------------------------------ ZFP fixed rate, 1-D
// A run of 32 values is eight ZFP blocks of four; at RATE bits per value a block takes 4 * RATE bits
// (zfp/src/zfp.c:773-803) and the run exactly RATE 32-bit words, so a thread writes whole words of the stream and
// nothing is assembled across threads (the reference's encoder ORs blocks into a zeroed stream with atomics,
// zfp/src/cuda_zfp/encode.cuh:224-231). Block i of a chunk sits at bit i * 4 * RATE, as in the reference stream;
// the block coder is oracle/zfp1d_planes.h, the CPU oracle's zfp1d.h arranged for the GPU. Lossy re-encoding (two-shot all-reduce) simply
// encodes the decoded sum again: there is no separate domain.
template <int RATE>
struct ZfpCodec {
  static_assert(RATE == 4 || RATE == 8 || RATE == 16, "fused rates: 4, 8, 16 bits per value");
  static constexpr int kBits = RATE;
  static constexpr int kWords = RATE;
  static constexpr bool kRotated = false;
  static constexpr int kMinBlocks = 2;
  // The coder is a chain of dependent integer work that neither warps nor registers shorten by much: eight chunks of 4 Mi fp32,
  // encode 71.5 us at rate 8 with four CTAs an SM and 70.0 with three (3,000,008 values 53.8 and 55.4), decode 90.4 and 89.8 (68.0 and
  // 70.0); rate 4 53.9 and 54.1, 65.3 and 63.8; rate 16 102.7 and 102.9, 139.8 and 138.4 (64 registers spill there: 8 x 262,147 values
  // 17.8 against 16.5 us). Sums, which hold a second run: 63.9 and 61.8 at rate 4, 92.5 and 86.4 at 8.
  static constexpr int kEncodeBlocks = 4, kDecodeBlocks = RATE == 16 ? 3 : 4, kSumBlocks = 3;
  static constexpr int kMaxBits = 4 * RATE;
  // the plane tables of oracle/zfp1d_planes.h live in the kernel's shared scratch, behind its first 8 floats
  static constexpr bool kExchanges = false;
  static constexpr bool kEncodeAhead = false;
  static constexpr int kSmemFloats = 8 + (int)sizeof(zfp1d::PlaneTables) / 4;
  static __device__ __forceinline__ const zfp1d::PlaneTables& tables(const float* sm) {
    return *reinterpret_cast<const zfp1d::PlaneTables*>(sm + 8);
  }
  // Every thread of the CTA calls this once, followed by a __syncthreads(), before any encode or fetch.
  static __device__ __forceinline__ void initShared(float* sm) {
    const uint4* t = reinterpret_cast<const uint4*>(&zfp1d::kPlaneTables);
    for (int i = threadIdx.x; i < (int)(sizeof(zfp1d::PlaneTables) / 16); i += blockDim.x) reinterpret_cast<uint4*>(sm + 8)[i] = __ldg(t + i);
  }

  struct Enc { uint32_t w[RATE]; };

  static __device__ __forceinline__ Enc encode(float (&v)[32], const CodecCfg& /*c*/, bool /*rotate*/, float* sm,
                                               uint64_t /*rngElem*/, uint4* /*win*/ = nullptr) {
    Enc e;
    const zfp1d::PlaneTables& tab = tables(sm);
    if (RATE == 4) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t lo = (uint32_t)zfp1d::encodePlanes<kMaxBits>(&v[8 * k], tab);
        const uint32_t hi = (uint32_t)zfp1d::encodePlanes<kMaxBits>(&v[8 * k + 4], tab);
        e.w[k] = lo | (hi << 16);
      }
    } else {
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const uint64_t s = zfp1d::encodePlanes<kMaxBits>(&v[4 * b], tab);
        if (RATE == 8) e.w[b] = (uint32_t)s;
        else { e.w[(2 * b) % RATE] = (uint32_t)s; e.w[(2 * b + 1) % RATE] = (uint32_t)(s >> 32); }
      }
    }
    return e;
  }

  static __device__ __forceinline__ void touched(const ChunkLayout& L, const CodecCfg&, long elem, long* payloadEnd, long* totalEnd) {
    const long off = (elem >> 5) * (4 * RATE);
    if (off >= L.totalBytes) { *payloadEnd = 0; *totalEnd = 0; return; }
    long end = off + 4 * RATE;
    if (end > L.totalBytes) end = L.totalBytes / 4 * 4;   // the tail is written word by word, whole words only
    *payloadEnd = end < L.payloadBytes ? end : L.payloadBytes;   // a ZFP chunk has no parameter part
    *totalEnd = end;
  }

  static __device__ __forceinline__ void store(const Enc& e, uint8_t* chunk, const ChunkLayout& L, const CodecCfg& /*c*/,
                                               long elem) {
    const long off = (elem >> 5) * (4 * RATE);
    if (off >= L.totalBytes) return;
    uint8_t* pw = chunk + off;
    if (off + 4 * RATE <= L.totalBytes && aligned16(pw)) {
#pragma unroll
      for (int q = 0; q < RATE / 4; ++q)
        reinterpret_cast<uint4*>(pw)[q] = make_uint4(e.w[4 * q], e.w[4 * q + 1], e.w[4 * q + 2], e.w[4 * q + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < RATE; ++k)
        if (off + 4 * k + 4 <= L.totalBytes) reinterpret_cast<uint32_t*>(pw)[k] = e.w[k];
    }
  }

  struct Raw {
    uint32_t w[RATE];
    const zfp1d::PlaneTables* tab;
    bool valid;
  };
  static constexpr int kBatch = 1;

  static __device__ __forceinline__ Raw fetch(const uint8_t* chunk, const ChunkLayout& L, const CodecCfg& /*c*/, long elem,
                                              float /*mul*/, const float* sm) {
    Raw r;
    r.tab = &tables(sm);
    const long off = (elem >> 5) * (4 * RATE);
    r.valid = off < L.totalBytes;
    if (!r.valid) return r;
    const uint8_t* pw = chunk + off;
    if (off + 4 * RATE <= L.totalBytes && aligned16(pw)) {
#pragma unroll
      for (int q = 0; q < RATE / 4; ++q) {
        const uint4 t = __ldcg(reinterpret_cast<const uint4*>(pw) + q);
        r.w[4 * q] = t.x; r.w[4 * q + 1] = t.y; r.w[4 * q + 2] = t.z; r.w[4 * q + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < RATE; ++k)
        r.w[k] = (off + 4 * k + 4 <= L.totalBytes) ? __ldcg(reinterpret_cast<const uint32_t*>(pw) + k) : 0u;
    }
    return r;
  }

  static __device__ __forceinline__ void accumulate(const Raw& r, float (&acc)[32]) {
    if (!r.valid) return;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      uint64_t s;
      if (RATE == 4) s = (r.w[b >> 1] >> (16 * (b & 1))) & 0xffffu;
      else if (RATE == 8) s = r.w[b % RATE];
      else s = (uint64_t)r.w[(2 * b) % RATE] | ((uint64_t)r.w[(2 * b + 1) % RATE] << 32);
      float x[4];
      zfp1d::decodePlanes<kMaxBits>(s, *r.tab, x);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[4 * b + i] += x[i];
    }
  }

  static __device__ __forceinline__ float finishScale(const CodecCfg&) { return 1.f; }
  static __device__ __forceinline__ void finish(float (&)[32], const CodecCfg&, uint4* /*win*/ = nullptr) {}
};

template <class Codec, class = void> struct HasDirectSums : std::false_type {};
template <class Codec> struct HasDirectSums<Codec, std::enable_if_t<Codec::kDirectSums>> : std::true_type {};

// acc += mul * sum over n encoded copies of the run at `elem`, copy i at base + i * stride, in order. The loads of B copies
// are issued before any of them is unpacked; what is left over after whole batches goes through the smaller batch sizes, so
// that a single copy (all-gather, all-to-all) carries no code for absent ones.
// `sm`: the kernel's shared scratch (Codec::kSmemFloats floats, Codec::initShared called); `aligned`: base and stride are
// multiples of 16 bytes; `spread`: finish() follows (a re-encoding sum stays in the run ownership, see TacoCodec).
template <class Codec, int B>
__device__ __forceinline__ void decodeBatches(const uint8_t*& src, long stride, int& n, const ChunkLayout& L, const CodecCfg& c,
                                              long elem, float mul, float (&acc)[32], const float* sm) {
#pragma unroll 1
  while (n >= B) {
    typename Codec::Raw r[B];
#pragma unroll
    for (int j = 0; j < B; ++j) r[j] = Codec::fetch(src + (long)j * stride, L, c, elem, mul, sm);
#pragma unroll
    for (int j = 0; j < B; ++j) Codec::accumulate(r[j], acc);
    src += (long)B * stride;
    n -= B;
  }
}
template <class Codec>
__device__ __forceinline__ void decodeSum(const uint8_t* base, long stride, int n, const ChunkLayout& L,
                                          const CodecCfg& c, long elem, float mul, float (&acc)[32], const float* sm, bool aligned,
                                          bool spread) {
  if (!COCCL_CHUNK_RANGE_OK(Codec, L, c, elem, 2)) return;   // the same range of every copy
  if constexpr (HasDirectSums<Codec>::value) {
    Codec::sum(base, stride, n, L, c, elem, mul, aligned, spread, acc);
  } else {
    if constexpr (Codec::kBatch >= 2) decodeBatches<Codec, 2>(base, stride, n, L, c, elem, mul, acc, sm);
    decodeBatches<Codec, 1>(base, stride, n, L, c, elem, mul, acc, sm);
  }
}

// Dispatch a generic lambda on the runtime codec configuration. The functor receives a codec type tag;
// unsupported configurations return false.
template <class F>
inline bool dispatchCodec(const CodecCfg& c, F&& f) {
  if (c.kind == kCodecMxfp8) { f(MxFp8Codec{}); return true; }
  if (c.kind == kCodecTaco) { f(TacoCodec{}); return true; }
  if (c.kind == kCodecZfp) {
    if (c.bits == 4) { f(ZfpCodec<4>{}); return true; }
    if (c.bits == 8) { f(ZfpCodec<8>{}); return true; }
    if (c.bits == 16) { f(ZfpCodec<16>{}); return true; }
    return false;
  }
  if (c.kind != kCodecSdp4bit) return false;
  const bool small = c.group < 32;
#define COCCL_SDP_CASE(B, A, H, S) \
  if (c.bits == B && (c.asym != 0) == A && (c.hadamard != 0) == H && small == S) { f(SdpCodec<B, A, H, S>{}); return true; }
  COCCL_SDP_CASE(4, false, true, false)
  COCCL_SDP_CASE(4, false, false, false)
  COCCL_SDP_CASE(8, false, true, false)
  COCCL_SDP_CASE(8, false, false, false)
  COCCL_SDP_CASE(4, true, true, false)
  COCCL_SDP_CASE(4, true, false, false)
  COCCL_SDP_CASE(8, true, true, false)
  COCCL_SDP_CASE(8, true, false, false)
  COCCL_SDP_CASE(4, false, false, true)
  COCCL_SDP_CASE(8, false, false, true)
  COCCL_SDP_CASE(4, true, false, true)
  COCCL_SDP_CASE(8, true, false, true)
#undef COCCL_SDP_CASE
  return false;
}

inline bool tileCodecSupported(const CodecCfg& c) {
  if (c.kind == kCodecMxfp8) return c.group == 32;
  if (c.kind == kCodecTaco)
    return c.bits == 8 && c.paramBytes == 8 && (c.group == 32 || c.group == 64 || c.group == 128 || c.group == 256 || c.group == 512);
  if (c.kind == kCodecZfp) return c.group == 4 && c.paramBytes == 0 && (c.bits == 4 || c.bits == 8 || c.bits == 16);
  if (c.kind != kCodecSdp4bit) return false;
  if (c.group < 8 || c.group > 2048 || (c.group & (c.group - 1))) return false;
  if (c.hadamard && c.group < 32) return false;
  return c.bits == 4 || c.bits == 8;
}

}  // namespace coccl
