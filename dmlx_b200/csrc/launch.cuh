// Launches whose start-up overlaps the end of the kernel before them in the stream (programmatic dependent launch).
//
// A step is a chain of dozens of kernels of a few microseconds.  Launched plainly, each waits until the one before has drained and its
// writes are flushed, and only then are its blocks scheduled.  With this attribute a kernel's blocks are scheduled as soon as every block of
// the kernel before has passed `let_next_start` and there is room; they set up what needs no memory and wait.
//
// In every kernel that is launched through `launch_after`, each thread that reads or writes global memory (weights apart, which nothing writes
// after their creation) or allocates tensor memory runs `wait_previous` before it does, and so does some thread of every block before it ends.
// So the bodies of two kernels of a stream never overlap, and as a kernel ends only after its own wait did, the wait of the next one covers all
// that came before.
//
// No kernel's input is `const T* __restrict__`: a kernel runs from its early start on, so what the one ahead writes changes within its lifetime, and
// the qualifier would let the compiler load it ahead of the wait (no other pointer reaches the object, so the wait's "memory" clobber would not
// stand in the way) or through the read-only path.  Memory that is only written may be `__restrict__`, so that loads are not held back by stores,
// and so may the parameters of a function that is called after the wait.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#ifdef __CUDACC__
// Waits until the kernels before this one in the stream have ended and their writes are visible.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel be scheduled once every block has come here (one thread of a block is enough) or ended.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Both.  For kernels of a few microseconds, or of many blocks per SM.  Blocks that wait take issue slots from those that work, so one long wave
// waits alone and lets the next kernel start when its main loop is done (the block-scaled matmul of 24576 expert rows: 372 us with 54 waiting
// warps on every SM, 334 without).
__device__ __forceinline__ void after_previous() {
  wait_previous();
  let_next_start();
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

// The same without the overlap, for two kinds of kernels:
//   * long ones of about as many blocks as there are SMs: scheduled while the one ahead still fills most of them, its blocks would come to lie two
//     and three on the SMs that have room, and the others stay idle;
//   * many blocks of next to no work, kManyBlocks and more: each waits for the kernels ahead by itself, 0.4 ns a block of the whole chip's time.
//     These neither wait nor let the next kernel start.
constexpr int kManyBlocks = 2048;
template <class... P, class... A>
inline void launch_apart(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  kernel<<<grid, block, smem, s>>>(static_cast<P>(std::forward<A>(args))...);
}

// CTAs of `kernel` that run at the same time in clusters of `size`, no more than `per_sm` on an SM of `sms`: a cluster's CTAs stay within a GPC, so
// some SMs are left over (33 clusters of eight, 71 of four and 148 of two at two CTAs on each of 148 SMs).
template <class... P>
inline int ctas_in_clusters(void (*kernel)(P...), int size, int per_sm, int sms, int threads, size_t smem) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = size;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(size * sms));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int clusters = 0, fit = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, smem) != cudaSuccess ||
      fit == 0) {
    cudaGetLastError();
    return 0;
  }
  return (int)((long long)clusters * size * std::min(per_sm, fit) / fit);
}
#endif
