// Launches that overlap the end of the kernel before them (programmatic dependent launch).
//
// A kernel calls releaseNext() at its start (the small GEMM behind its main loop) and awaitPrevious() before it touches anything
// that an earlier kernel of the stream may read or write. Its CTAs then take the places that the CTAs of the kernel before it
// leave, and set themselves up while the last of those run. awaitPrevious() returns when that kernel has completed and its memory
// is visible; since that one waited in the same way, everything before it has completed too. Every thread of every kernel that is
// launched like this must therefore call it. All CTAs of a kernel have started before any of the next one does, so nothing can be
// held up. Launched in the ordinary way both calls do nothing.
//
// What an earlier kernel of the stream may have written is read with loadOrdered (common.cuh) or plain dereferences, behind
// awaitPrevious(). Loads that take memory to be read-only for the kernel's whole life (__ldg, ld.global.nc, const pointers with
// __restrict__) are not ordered by the wait: the compiler may move them ahead of it, and that life begins while earlier kernels write.
//
// The trainers' short kernels and small GEMMs are launched like this: a chain of them is bound by launch latency, and a replayed
// training step of two layers, 512 wide, takes 666 us instead of 750 (steps 4096 wide: 17.4 against 17.5 ms and 18.39 against 18.37, no
// difference). The codec kernels are not. They fill the chip for tens of microseconds with a fixed share of the tiles for
// each CTA, and CTAs that move in early share an SM with the last ones of the kernel before: a stochastic 4-bit encode + sum of
// 8 x 8 Mi fp32 took 84.7 us instead of 77.3, although the shorter codec chains gained (49.9 -> 45.5 us for 8 x 5,000,003 bf16). For
// the same reason launchIfEarly leaves out norm backwards and rotations of several rows a CTA, and norms of wide rows alone.
#pragma once
#include <cuda_runtime.h>

namespace coccl {

#ifdef __CUDACC__
__device__ __forceinline__ void releaseNext() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void awaitPrevious() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... Params, class... Args>
static inline cudaError_t launchIfEarly(bool early, void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                        Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}
template <class... Params, class... Args>
static inline cudaError_t launchAfter(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  return launchIfEarly(true, kern, grid, block, smem, stream, args...);
}
#endif

}  // namespace coccl
