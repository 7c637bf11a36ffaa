// Programmatic dependent launch: a kernel that starts while the kernel before
// it in the stream drains.
//
// A kernel launched by launch_after has its launch and its blocks' start
// overlap the last blocks of its predecessor; its first statement,
// after_previous(), holds every thread until that predecessor has ended and its
// writes are visible, so the order of memory is the stream's. Kernels in a row
// may all be launched so: each waits before it does anything, so the end of
// one implies the end of all before it. Used where the predecessor is a
// kernel of this library in the same stream.
//
// Only where one chain of kernels has the device to itself: see follow() in
// render.cu. No kernel lets its successor start before its own blocks have ended
// (griddepcontrol.launch_dependents): waiting blocks hold the slots that the
// other lanes' kernels would run in (1080p terrain, 64 spp: 57.0 -> 59.5 ms;
// ten renders in a batch 12.1 -> 12.8).
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

namespace rmn {

template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t shared, cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = shared;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace rmn
