// The ZFP block coder of zfp1d.h (same stream, same values) for blocks of 16, 32 or 64 bits, arranged for the GPU: the four
// values' bit planes are transposed once into a string of nibbles, first plane first, and the coder then works on the
// string instead of gathering four bits per plane:
//  * leading zero planes cost one stream bit each and are skipped by a count of leading zeros;
//  * while some value is not yet significant the encoder takes two planes per table look-up, the decoder as many whole planes as
//    eight stream bits hold (one to four); what is left when the budget cuts a look-up short, at most seven bits with the plane
//    that they end in, is one look-up more;
//  * from the plane on in which all four values are significant a plane's code is its four bits, so the rest of the string
//    IS the rest of the stream and is appended (or taken off) with one shift.
// The arithmetic and logic units bound it (half rate; 60 % of what the decoder issued with one plane a look-up and 64-bit words
// at every rate): 16 Mi fp32 at 8 bits each (84 MB each way, 13 us to copy): 40.7 -> 35.9 us to encode, 66.5 -> 46.9 us to decode.
#pragma once
#include "oracle/zfp1d.h"

namespace coccl {
namespace zfp1d {

struct alignas(16) PlaneTables {
  uint32_t enc[4 * 256];   // [n][two planes]: bits 0-15 code, 16-23 length, 24-31 n after them
  uint32_t dec[4 * 256];   // [n][next 8 bits]: bits 0-15 the whole planes in them, 16-19 their length, 20-24 four bits for each, 25-27 n after
  uint16_t tail[4 * 256];  // [n][1 << r | r bits], r < 8: the planes of a block's last r bits, the last of them cut by the budget
};

// One plane by the serial rules of decodeBlock, from `budget` bits: plane | bits used << 4 | n after it << 8.
COCCL_HD constexpr uint32_t serialPlane(int n, uint32_t s, int budget) {
  int bits = budget;
  const int m = n < bits ? n : bits;
  bits -= m;
  uint32_t plane = s & ((1u << m) - 1u);
  s >>= m;
  while (n < kBlock && bits) {
    --bits;
    const uint32_t any = s & 1u;
    s >>= 1;
    if (!any) break;
    while (n < kBlock - 1 && bits) {
      --bits;
      const uint32_t bit = s & 1u;
      s >>= 1;
      if (bit) break;
      ++n;
    }
    plane |= 1u << n;
    ++n;
  }
  return plane | ((uint32_t)(budget - bits) << 4) | ((uint32_t)n << 8);
}

constexpr int kPlaneTableWork = 4 * 256;
COCCL_HD constexpr void fillPlaneTables(PlaneTables& t, int k) {   // entry k of each table
  const uint32_t v = (uint32_t)(k & 255);
  const uint32_t a = planeCode(k >> 8, v & 15u);
  const uint32_t b = planeCode((int)(a >> 12), v >> 4);
  const uint32_t la = (a >> 8) & 15u, lb = (b >> 8) & 15u;
  t.enc[k] = (a & 0xffu) | ((b & 0xffu) << la) | ((la + lb) << 16) | ((b >> 12) << 24);

  int n = k >> 8, len = 0, at = 0;
  uint32_t planes = 0;
  while (n < kBlock && at < 16) {
    const uint32_t e = serialPlane(n, v >> len, 7);
    const int l = (int)((e >> 4) & 15u);
    if (len + l > 8) break;   // a code is at most seven bits long: the first always fits
    planes |= (e & 15u) << at;
    at += 4;
    len += l;
    n = (int)(e >> 8);
  }
  t.dec[k] = planes | ((uint32_t)len << 16) | ((uint32_t)at << 20) | ((uint32_t)n << 25);

  int r = 0;
  while ((v >> (r + 1)) != 0) ++r;
  uint32_t rest = v & ((1u << r) - 1u);
  planes = 0;
  n = k >> 8;
  at = 0;
  while (r > 0 && at < 16) {   // seven bits hold at most four planes that are not zero: the first has a value's first bit
    const uint32_t e = serialPlane(n, rest, r);
    const int l = (int)((e >> 4) & 15u);
    planes |= (e & 15u) << at;
    at += 4;
    r -= l;
    rest >>= l;
    n = (int)(e >> 8);
  }
  t.tail[k] = (uint16_t)planes;
}
constexpr PlaneTables makePlaneTables() {
  PlaneTables t = {};
  for (int k = 0; k < kPlaneTableWork; ++k) fillPlaneTables(t, k);
  return t;
}
// Worked out by the compiler: filling them takes a CTA longer than a few tiles do.
#ifdef __CUDACC__
static __device__ const PlaneTables kPlaneTables = makePlaneTables();
#endif

COCCL_HD int leadingZeros(uint32_t x) {   // x != 0
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return __builtin_clz(x);
#endif
}
COCCL_HD int trailingZeros(uint64_t x) {   // x != 0
#ifdef __CUDA_ARCH__
  return __ffsll((long long)x) - 1;
#else
  return __builtin_ctzll(x);
#endif
}
COCCL_HD int trailingZeros(uint32_t x) {   // x != 0
#ifdef __CUDA_ARCH__
  return __ffs((int)x) - 1;
#else
  return __builtin_ctz(x);
#endif
}
COCCL_HD uint32_t reverseBits(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __brev(x);
#else
  x = ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
  x = ((x >> 2) & 0x33333333u) | ((x & 0x33333333u) << 2);
  x = ((x >> 4) & 0x0f0f0f0fu) | ((x & 0x0f0f0f0fu) << 4);
  return __builtin_bswap32(x);
#endif
}
COCCL_HD uint32_t swapBits(uint32_t x, int s, uint32_t m) {
  const uint32_t t = ((x >> s) ^ x) & m;
  return x ^ t ^ (t << s);
}
COCCL_HD uint32_t floatBits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  union { float f; uint32_t u; } c;
  c.f = f;
  return c.u;
#endif
}
COCCL_HD float bitsFloat(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  union { float f; uint32_t u; } c;
  c.u = u;
  return c.f;
#endif
}

// Byte 3 - W of each of the four words: eight planes of four values -> eight nibbles, first plane lowest. A 4 x 8 bit
// transposition is a permutation of the five bits of a position and takes four exchanges of two of them.
template <int W>
COCCL_HD uint32_t planesToNibbles(const uint32_t (&u)[4]) {
#ifdef __CUDA_ARCH__
  constexpr uint32_t b = 3 - W, lo = b | ((b + 4) << 4);
  uint32_t x = __byte_perm(__byte_perm(u[3], u[2], lo), __byte_perm(u[1], u[0], lo << 8), 0x7610);
#else
  constexpr int sh = 24 - 8 * W;
  uint32_t x = ((u[3] >> sh) & 255u) | (((u[2] >> sh) & 255u) << 8) | (((u[1] >> sh) & 255u) << 16) | (((u[0] >> sh) & 255u) << 24);
#endif
  x = reverseBits(x);                     // value r in byte r, first plane in bit 0
  x = swapBits(x, 14, 0x0000CCCCu);
  x = swapBits(x, 7, 0x00AA00AAu);
  x = swapBits(x, 12, 0x0000F0F0u);
  return swapBits(x, 4, 0x00F000F0u);
}
// The way back: value r's byte (first plane in bit 7) ends up in byte 3 - r.
COCCL_HD uint32_t nibblesToPlanes(uint32_t x) {
  x = swapBits(x, 4, 0x00F000F0u);
  x = swapBits(x, 12, 0x0000F0F0u);
  x = swapBits(x, 7, 0x00AA00AAu);
  x = swapBits(x, 14, 0x0000CCCCu);
  return reverseBits(x);
}

// Byte k of each word, the first word's highest.
COCCL_HD uint32_t planeBytes(const uint32_t (&b)[1], int k) { return (b[0] >> (8 * k)) << 24; }
#ifdef __CUDA_ARCH__
COCCL_HD uint32_t planeBytes(const uint32_t (&b)[2], int k) { return __byte_perm(__byte_perm(b[0], b[1], (k << 4) | (k + 4)), 0u, 0x1044); }
COCCL_HD uint32_t planeBytes(const uint32_t (&b)[4], int k) {
  const uint32_t sel = (uint32_t)((k << 4) | (k + 4));
  return __byte_perm(__byte_perm(b[2], b[3], sel), __byte_perm(b[0], b[1], sel), 0x5410);
}
#else
COCCL_HD uint32_t planeBytes(const uint32_t (&b)[2], int k) { return (((b[0] >> (8 * k)) & 255u) << 24) | (((b[1] >> (8 * k)) & 255u) << 16); }
COCCL_HD uint32_t planeBytes(const uint32_t (&b)[4], int k) {
  return (((b[0] >> (8 * k)) & 255u) << 24) | (((b[1] >> (8 * k)) & 255u) << 16) | (((b[2] >> (8 * k)) & 255u) << 8) | ((b[3] >> (8 * k)) & 255u);
}
#endif

// A string of planes as it takes part in a block of MAXBITS bits: after the leading zeros a plane costs at least two stream
// bits, so MAXBITS - 9 bits hold (MAXBITS - 9) / 2 planes at most: 8, 16 and 32 nibbles.
template <int MAXBITS>
struct PlaneShape {
  static_assert(MAXBITS == 16 || MAXBITS == 32 || MAXBITS == 64, "rates 4, 8 and 16");
  static constexpr int kWords = MAXBITS / 16;   // words of eight nibbles
};
// Integers that hold a block's bits, and up to 16 nibbles of its string of planes.
template <int MAXBITS> struct PlaneInts { using Bits = uint32_t; using Planes = uint64_t; };
template <> struct PlaneInts<16> { using Bits = uint32_t; using Planes = uint32_t; };
template <> struct PlaneInts<64> { using Bits = uint64_t; using Planes = uint64_t; };

template <int MAXBITS>
COCCL_HD uint64_t encodePlanes(const float* x, const PlaneTables& t) {
  float m = 0.f;
  for (int i = 0; i < kBlock; ++i) m = fmaxf(m, fabsf(x[i]));
  if (!(m > 0.f) || !(m < INFINITY)) return 0;
  const int biased = (int)(floatBits(m) >> 23);          // common exponent = biased - 126; a subnormal maximum counts as the
  const int emax = biased - 126;                         // smallest normal exponent (biased 0)
  const int sc = 30 - emax + 127;                        // 2^(30 - emax), infinite beyond the range as ldexpf gives it
  const float scale = bitsFloat((uint32_t)(sc < 255 ? sc : 255) << 23);
  int32_t q[kBlock];
  for (int i = 0; i < kBlock; ++i) q[i] = (int32_t)(x[i] * scale);
  forwardLift(q);
  uint32_t u[kBlock];
  for (int i = 0; i < kBlock; ++i) u[i] = toNegabinary(q[i]);
  using Bits = typename PlaneInts<MAXBITS>::Bits;
  using Planes = typename PlaneInts<MAXBITS>::Planes;
  Bits acc = (Bits)(2 * (emax + kEbias) + 1);
  const uint32_t all = u[0] | u[1] | u[2] | u[3];
  if (all == 0) return acc;
  const int z = leadingZeros(all);
  int pos = 9 + z;
  if (pos >= MAXBITS) return acc;
  for (int i = 0; i < kBlock; ++i) u[i] <<= z;
  constexpr int W = PlaneShape<MAXBITS>::kWords;
  Planes p = planesToNibbles<0>(u);
  uint64_t ph = 0;
  if constexpr (W >= 2) p |= (Planes)planesToNibbles<1>(u) << 32;
  if constexpr (W >= 4) ph = (uint64_t)planesToNibbles<2>(u) | ((uint64_t)planesToNibbles<3>(u) << 32);
  uint32_t n = 0;
  while (n < (uint32_t)kBlock && pos < MAXBITS) {
    const uint32_t e = t.enc[n * 256u + (uint32_t)(p & 255u)];
    acc |= (Bits)(e & 0xffffu) << pos;   // bits beyond the block fall off
    pos += (int)((e >> 16) & 0xffu);
    n = e >> 24;
    p >>= 8;
    if (W >= 4) { p |= (Planes)(ph << 56); ph >>= 8; }
  }
  if (pos < MAXBITS) acc |= (Bits)p << pos;
  return MAXBITS == 16 ? (acc & 0xffffu) : acc;
}

// `s` must be zero above bit MAXBITS - 1.
template <int MAXBITS>
COCCL_HD void decodePlanes(uint64_t stream, const PlaneTables& t, float* x) {
  using Bits = typename PlaneInts<MAXBITS>::Bits;
  using Planes = typename PlaneInts<MAXBITS>::Planes;
  Bits s = (Bits)stream;
  const int field = (int)((s >> 1) & 0xffu);
  const uint32_t nonzero = (uint32_t)s & 1u;
  s >>= 9;
  const int z = s != 0 ? trailingZeros(s) : 32;
  if (nonzero == 0 || z >= 32) {   // no plane at all, or more zero planes than a value has bits
    for (int i = 0; i < kBlock; ++i) x[i] = 0.f;
    return;
  }
  s >>= z;
  int rem = MAXBITS - 9 - z, at = 0;   // stream bits left; bit position in the string of planes
  constexpr int W = PlaneShape<MAXBITS>::kWords;
  Planes p = 0;
  uint64_t ph = 0;
  auto put = [&](Bits planes) {   // from bit `at` of the string on
    if (W >= 4 && at >= 64) { ph |= (uint64_t)planes << (at - 64); return; }
    p |= (Planes)planes << at;
    if (W >= 4 && at > 0) ph |= (uint64_t)planes >> (64 - at);
  };
  uint32_t n = 0;
  while (n < (uint32_t)kBlock) {
    const uint32_t e = t.dec[n * 256u + ((uint32_t)s & 255u)];
    const int len = (int)((e >> 16) & 15u);
    if (len > rem) break;
    put((Bits)(e & 0xffffu));
    n = e >> 25;
    at += (int)((e >> 20) & 31u);
    s >>= len;
    rem -= len;
  }
  put(n < (uint32_t)kBlock ? (Bits)t.tail[n * 256u + ((1u << rem) | (uint32_t)s)] : s);
  uint32_t b[W];
  b[0] = nibblesToPlanes((uint32_t)p);
  if constexpr (W >= 2) b[1] = nibblesToPlanes((uint32_t)(p >> 32));
  if constexpr (W >= 4) { b[2] = nibblesToPlanes((uint32_t)ph); b[3] = nibblesToPlanes((uint32_t)(ph >> 32)); }
  int32_t q[kBlock];
  for (int i = 0; i < kBlock; ++i) q[i] = fromNegabinary(planeBytes(b, 3 - i) >> z);
  inverseLift(q);
  const int e = field - kEbias - 30;   // 2^e, which may be subnormal or vanish
  const float scale = bitsFloat(e >= -126 ? (uint32_t)(e + 127) << 23 : (e >= -149 ? 1u << (e + 149) : 0u));
  for (int i = 0; i < kBlock; ++i) x[i] = (float)q[i] * scale;
}

}  // namespace zfp1d
}  // namespace coccl
