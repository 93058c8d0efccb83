// Fused collectives of __half tensors.
#include "collective_launch.cuh"

namespace coccl {
int launchFusedF16(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream) {
  return launchFused<__half>(a, emulatedRanks, maxCtas, stream);
}
int boundsWordF16(unsigned int* out, int reset) { return readBoundsWord(out, reset); }
}  // namespace coccl
