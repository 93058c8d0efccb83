// Fused collectives of float tensors.
#include "collective_launch.cuh"

namespace coccl {
int launchFusedF32(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream) {
  return launchFused<float>(a, emulatedRanks, maxCtas, stream);
}
int boundsWordF32(unsigned int* out, int reset) { return readBoundsWord(out, reset); }
}  // namespace coccl
