// Lists in device memory that depend on a launch's shape alone (task queues,
// tile lists): made on first use, kept by a handle.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace bta {

// New device memory with a copy of `bytes` bytes at src, complete on return
// whichever stream reads it next.  The copy has a stream of its own: a plain
// cudaMemcpy from pageable memory may return before its bytes have arrived,
// which orders it before a kernel of the legacy stream and of streams that
// wait for that one, but not of a non-blocking stream; and the launch's own
// stream may be under capture.
inline cudaError_t upload_list(void** out, const void* src, size_t bytes) {
  *out = nullptr;
  void* d = nullptr;
  cudaError_t e = cudaMalloc(&d, bytes);
  if (e != cudaSuccess) return e;
  cudaStream_t s = nullptr;
  e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) {
    e = cudaMemcpyAsync(d, src, bytes, cudaMemcpyHostToDevice, s);
    const cudaError_t w = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = w;
    cudaStreamDestroy(s);
  }
  if (e != cudaSuccess) {
    cudaFree(d);
    return e;
  }
  *out = d;
  return cudaSuccess;
}

}  // namespace bta
