// Launch of the fused collectives for one element type (collective_<type>.cu).
#pragma once
#include "collective_launch.h"
#include "launch_count.h"
#include "per_device.h"

namespace coccl {

template <typename T, class C, int FORM>
static int launchForm(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream) {
  auto kern = fusedCollectiveKernel<T, C, FORM>;
  struct Places { int perSm, sms; };
  static PerDevice<Places> places;
  const Places* at;
  int dev = 0;
  cudaGetDevice(&dev);
  const int rc = places.get(dev, &at, [&](Places& v) {
    cudaDeviceGetAttribute(&v.sms, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v.perSm, kern, kTileThreads, 0);
    return e != cudaSuccess ? (int)e : (v.perSm <= 0 ? -1 : 0);
  });
  if (rc != 0) return rc;
  const long tiles = (a.count + kTileElems - 1) / kTileElems;
  const long slices = (tiles + a.sliceTiles - 1) / a.sliceTiles;
  if (slices > kMaxSlices) return -1;
  long items = slices * a.nRanks;
  long cap = (long)at->perSm * at->sms / emulatedRanks;
  if (maxCtas > 0 && maxCtas < cap) cap = maxCtas;
  if (cap < 1) cap = 1;
  int gx = (int)(items < cap ? items : cap);
  dim3 grid(gx, emulatedRanks, 1);
  CollArgs copy = a;
  cocclkCountLaunches(1);
  void* params[] = {&copy};
  if (emulatedRanks > 1) {
    // the emulated ranks wait on one another: co-residency must be guaranteed
    return (int)cudaLaunchCooperativeKernel((const void*)kern, grid, dim3(kTileThreads), params, 0, stream);
  }
  return (int)cudaLaunchKernel((const void*)kern, grid, dim3(kTileThreads), params, 0, stream);
}

template <typename T, class C>
static int launchOne(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream) {
  switch (collForm(a.op)) {
    case kFormReduce: return launchForm<T, C, kFormReduce>(a, emulatedRanks, maxCtas, stream);
    case kFormTwoShot: return launchForm<T, C, kFormTwoShot>(a, emulatedRanks, maxCtas, stream);
    case kFormGatherDelta: return launchForm<T, C, kFormGatherDelta>(a, emulatedRanks, maxCtas, stream);
    default: return launchForm<T, C, kFormGather>(a, emulatedRanks, maxCtas, stream);
  }
}

template <typename T>
static int launchFused(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream) {
  int rc = -1;
  const bool ok = dispatchCodec(a.codec, [&](auto codecTag) { rc = launchOne<T, decltype(codecTag)>(a, emulatedRanks, maxCtas, stream); });
  return ok ? rc : -1;
}

static inline int readBoundsWord(unsigned int* out, int reset) {
#ifdef COCCL_BOUNDS_CHECK
  cudaError_t e = cudaMemcpyFromSymbol(out, gBoundsWord, 8 * sizeof(unsigned int));
  if (e == cudaSuccess && reset) {
    const unsigned int zero[8] = {};
    e = cudaMemcpyToSymbol(gBoundsWord, zero, sizeof(zero));
  }
  return (int)e;
#else
  for (int i = 0; i < 8; ++i) out[i] = 0;
  (void)reset;
  return 0;
#endif
}

}  // namespace coccl
