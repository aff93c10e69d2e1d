// Launches whose prologue overlaps the end of the kernel before them on the stream (programmatic dependent launch).
//
// A chain of dependent kernels pays, between any two, for the first one's completion to be seen and the second one's blocks
// to be started: 2 - 3 us, as long as some of the kernels themselves.  A kernel launched with launch_overlapped may start
// while its predecessor still runs; it sets up its barriers and tensor memory and then calls wait_previous, which returns
// once the predecessor has completed and its writes are visible.  Every such kernel calls it in all threads before its
// first access to global memory, so completion is transitive along the stream.
//
// Used where a transformer block's kernels follow each other (linear, layer norm, attention, bias gradient): forward and
// backward of a block of 8 x 1024 x 1024 in bf16 take 926 us, 950 without it; attention forward and backward at
// 8 x 16 x 1024 x 64 take 170 us, 173 without; a prefill of 1 x 16 x 2048 x 64 with a team per item 31.1 us, 32.8 without.  A launch whose
// blocks do not all fit beside the one before it starts them as SMs become free: a grid of one block per SM has to take up an SM
// alone to be spread over all of them (see layernorm.cu).  Not for the
// batch-norm, convolution and pooling kernels, which fill the chip for longer than a launch takes: with it a bottleneck of
// 256 x 28 x 28 took 1154 us instead of 1166 (runs differ by 1.9 %), the stem with its pooling stage 1037 instead of 850.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace tmpi {

// The pointers given to it get an offset of zero that the compiler only knows after the wait, so that no load through them
// (a const __restrict__ one may be taken for invariant) can be moved in front of it.
template <typename... T>
__device__ __forceinline__ void wait_previous(T&... pointers) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the next kernel may start; it waits for this one in turn
  int zero;
  asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(zero)::"memory");
  ((pointers += zero), ...);
}

template <typename... P, typename... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream; cfg.attrs = at; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace tmpi
