// Entry points of the fused compressed collectives (see collective_kernels.cuh); the kernels are in collective_<type>.cu.
#include "collective_launch.h"
#include "kernels_api.h"
#include <string.h>

using namespace coccl;

static_assert(sizeof(cocclkCollArgs) == sizeof(CollArgs), "collective POD mismatch");
static_assert(COCCLK_MAX_SLICES == kMaxSlices && COCCLK_MAX_RANKS == kMaxRanks, "constant mismatch");

extern "C" long cocclkFlagBytes(void) { return 2L * kMaxRanks * kMaxSlices * (long)sizeof(unsigned int); }

extern "C" int cocclkTileElems(void) { return kTileElems; }

extern "C" long cocclkSlotBytes(const cocclkCodec* codec, long count) {
  CodecCfg c;
  memcpy(&c, codec, sizeof(c));
  return makeChunkLayout(c, count, 16).stride;
}

extern "C" int cocclkFusedCollective(const cocclkCollArgs* args, int emulatedRanks, int maxCtas,
                                     cudaStream_t stream) {
  CollArgs a;
  memcpy(&a, args, sizeof(a));
  if (a.nRanks < 1 || a.nRanks > kMaxRanks || a.count <= 0 || a.sliceTiles <= 0) return -1;
  if (emulatedRanks != 1 && emulatedRanks != a.nRanks) return -1;
  // what the kernel follows without looking: every rank's workspace and flags, and the tensors of the ranks played here
  if (a.rankBase < 0 || a.rankBase + emulatedRanks > a.nRanks) return -1;
  for (int r = 0; r < a.nRanks; ++r) {
    const bool here = r >= a.rankBase && r < a.rankBase + emulatedRanks;
    if (!a.ws[r] || !a.flags[r] || (here && (!a.in[r] || !a.out[r]))) return -1;
  }
  if (!tileCodecSupported(a.codec)) return -1;
  switch (a.dtype) {
    case kF32: return launchFusedF32(a, emulatedRanks, maxCtas, stream);
    case kF16: return launchFusedF16(a, emulatedRanks, maxCtas, stream);
    case kBF16: return launchFusedBf16(a, emulatedRanks, maxCtas, stream);
    default: return -1;
  }
}

// ---------------------------------------------------------------------------------------------
// Bounds-checked build (libcoccl_checked.so, -DCOCCL_BOUNDS_CHECK): 1 when the codec accesses of the fused collectives
// and the stand-alone codec kernels are range-checked, and the first violation they recorded:
// out[0] = 0x80000000 | site (1 encode store, 2 decode fetch, 3 re-encode store of the two-shot all-reduce) or 0,
// out[1..2] = element index, out[3] / out[4] = payload end touched / payload bytes, out[5] / out[6] = chunk end touched /
// chunk bytes. Synchronises the device.
extern "C" int cocclkBoundsWordCodec(unsigned int* out, int reset);
extern "C" int cocclkBoundsChecked(void) {
#ifdef COCCL_BOUNDS_CHECK
  return 1;
#else
  return 0;
#endif
}
extern "C" int cocclkBoundsWord(unsigned int* out, int reset) {
  if (out == nullptr) return -1;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return (int)e;
  for (int i = 0; i < 8; ++i) out[i] = 0;
  int (*const readers[])(unsigned int*, int) = {boundsWordF32, boundsWordF16, boundsWordBf16, cocclkBoundsWordCodec};
  for (auto read : readers) {
    unsigned int w[8];
    const int rc = read(w, reset);
    if (rc != 0) return rc;
    if (out[0] == 0) for (int i = 0; i < 8; ++i) out[i] = w[i];
  }
  return 0;
}
