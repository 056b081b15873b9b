// Launches of the pass kernels, overlapping each one's start with the end of
// the kernel before it on the stream (programmatic dependent launch).
//
// A plan is a chain of 1 to 14 kernels of a few microseconds in a small box,
// and the gaps between them were a third of a round trip.  A kernel launched
// here may start once every block of the one before it has exited; each
// thread's first statement (pass_enter) then waits until the kernels before it
// are complete and their writes visible, so nothing is read or written early.
// Kernels without pass_enter are launched the usual way and see the usual order.
// No block lets the next kernel in before it exits: with that at the start,
// blocks of the next kernel crowded onto the SMs that fell idle first (100^3
// Float32 round trip 52.0 us against 37.7).
// Round trips without and with the overlap: 50x40x60 Float32 49.2 -> 32.6 us,
// 100^3 Float32 52.3 -> 37.7, 16x32x64 Float64 43.1 -> 36.4, 101x97x103 Float32
// 73.8 -> 57.5, 512^3 Float32 1255 -> 1232.
#pragma once

#include <cuda_runtime.h>

namespace pfgb {

#if defined(__CUDACC__)
__device__ __forceinline__ void pass_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

template <typename A>
static cudaError_t launch_pass_kernel(void (*kernel)(A), int64_t grid, int threads, size_t smem, cudaStream_t s, const A& args) {
  cudaLaunchAttribute overlap;
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &overlap;
  c.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&c, kernel, args);
  if (e != cudaSuccess) cudaGetLastError();  // reported here, and not by the caller's next check
  return e;
}

}  // namespace pfgb
