// Launches whose start-up overlaps the end of the kernel before them in the stream (programmatic dependent launch).
//
// A step is a chain of dozens of kernels of a few microseconds.  Launched plainly, each waits until the one before has drained and its
// writes are flushed, and only then are its blocks scheduled.  With this attribute a kernel's blocks are scheduled as soon as every block of
// the kernel before has passed `after_previous` and there is room; they set up what needs no memory and wait inside `after_previous`.
//
// Every kernel that is launched through `launch_after` runs `after_previous` in all of its threads, before any return and before it reads or
// writes global memory or allocates tensor memory.  So the bodies of two kernels of a stream never overlap, and as a kernel ends only after its
// own wait did, the wait of the next one covers all that came before.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#ifdef __CUDACC__
// Waits until the kernels before this one in the stream have ended and their writes are visible, then lets the next one be scheduled.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// kernel<<<grid, block, smem, s>>>(args...); a failure is left for cudaGetLastError.
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}
#endif
