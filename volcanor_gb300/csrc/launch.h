// Launches that follow one another on a stream.
//
// A step is a chain of 35 to 45 kernels, most of them a few microseconds
// long; launched one after the other, each waited 2.7 us more for its
// predecessor than the arithmetic needs.  launch_next lets a kernel be set up
// while the kernel before it on the stream still runs (programmatic stream
// serialization): 60 small kernels in a chain take 1.4 us each instead of 4.1.
// In a captured graph a launch costs 1.3 to 1.7 us anyway (1.1 to 1.4 this way),
// and there the blocks set up early hold registers that the kernels of other
// branches want: with it 8 steps of a 6-revolution hover rotor take 6.1 to 6.3 ms
// instead of 5.95 and 4 steps of 8 uneven rotors 10.8 instead of 10.0, so a
// stream under capture gets plain launches.
//
// Every kernel launched this way begins with after_previous(), in every
// thread and before any memory access: it returns when the kernel before has
// finished and its writes are visible.  A kernel finishes only after its own
// after_previous(), so the whole chain before it has finished too, and events,
// copies, memsets and plain launches after it order as after any kernel.
// Such kernels take no const __restrict__ pointers: what they read is written
// by the kernel before, perhaps after they were set up, so nothing may be
// loaded as read-only data.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace vlm {

#ifdef __CUDACC__
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// kernel<<<grid, block, smem, st>>>(args...), set up early; errors are left
// for cudaGetLastError like that form's
template <class... P, class... A>
inline void launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(st, &capture);
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
#endif

}  // namespace vlm
