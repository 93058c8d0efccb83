// The fused collectives, one translation unit for each element type: each holds 4 forms x 16 codecs of the kernel.
#pragma once
#include "collective_kernels.cuh"

namespace coccl {
int launchFusedF32(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream);
int launchFusedF16(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream);
int launchFusedBf16(const CollArgs& a, int emulatedRanks, int maxCtas, cudaStream_t stream);
// The bounds-checked build's error word of each (see codecs.cuh); zeros in the normal build.
int boundsWordF32(unsigned int* out, int reset);
int boundsWordF16(unsigned int* out, int reset);
int boundsWordBf16(unsigned int* out, int reset);
}  // namespace coccl
