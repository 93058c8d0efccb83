// Fused collectives of __nv_bfloat16 tensors.
#include "collective_launch.cuh"

namespace coccl {
int launchFusedBf16(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream) {
  return launchFused<__nv_bfloat16>(a, emulatedRanks, maxCtas, stream);
}
int boundsWordBf16(unsigned int* out, int reset) { return readBoundsWord(out, reset); }
}  // namespace coccl
