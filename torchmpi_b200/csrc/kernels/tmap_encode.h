// The driver's tensor-map encoders want a current context.  A thread that has made no CUDA runtime call yet has none: PyTorch's
// backward thread where the first operation of a process's first backward is one of these kernels and its outputs come out of
// the allocator's cache.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace tmpi {

// encode(), once more with the thread's device context made current if it was missing
template <typename F>
inline CUresult encode_in_context(F encode) {
  CUresult r = encode();
  int dev = 0;
  if (r == CUDA_ERROR_INVALID_CONTEXT && cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
  return r;
}

}  // namespace tmpi
