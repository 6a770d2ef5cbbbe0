// Lists in device memory that depend on a launch's shape alone (task queues,
// tile lists): made on first use, kept by a handle.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdlib.h>

#include <map>
#include <utility>
#include <vector>

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

inline bool is_capturing(cudaStream_t s) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &c) == cudaSuccess) return c != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;
}

// A handle's lists by launch shape.  They take at most LISTS_BYTES (or one list,
// where that is larger; DALIA_B200_LIST_BYTES sets another limit): a new shape
// beyond it first frees the others, once the launches that read them have
// ended -- all of them precede the given stream's end, since a handle's calls
// share their workspace in any case.  A list that a stream capture has taken is
// part of a graph that may run later and stays until the handle's end.
class ShapeLists {
 public:
  struct List {
    void* d = nullptr;
    int n = 0;
    size_t bytes = 0;
    bool captured = false;
  };
  // nullptr: a new shape
  const List* find(const std::vector<int>& key, cudaStream_t s) {
    auto it = by_shape_.find(key);
    if (it == by_shape_.end()) return nullptr;
    if (!it->second.captured) it->second.captured = is_capturing(s);
    return &it->second;
  }
  cudaError_t add(std::vector<int> key, const void* src, int n, size_t bytes, cudaStream_t s, const List** out) {
    List l;
    l.n = n;
    l.bytes = bytes;
    l.captured = is_capturing(s);
    if (!l.captured && held_ + bytes > limit()) {
      const cudaError_t e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return e;
      for (auto it = by_shape_.begin(); it != by_shape_.end();) {
        if (it->second.captured) {
          ++it;
          continue;
        }
        held_ -= it->second.bytes;
        cudaFree(it->second.d);
        it = by_shape_.erase(it);
      }
    }
    if (bytes > 0) {
      const cudaError_t e = upload_list(&l.d, src, bytes);
      if (e != cudaSuccess) return e;
    }
    held_ += bytes;
    *out = &by_shape_.emplace(std::move(key), l).first->second;
    return cudaSuccess;
  }
  ~ShapeLists() {
    for (auto& kv : by_shape_) cudaFree(kv.second.d);
  }

 private:
  static constexpr size_t LISTS_BYTES = size_t(256) << 20;
  static size_t limit() {
    const char* e = getenv("DALIA_B200_LIST_BYTES");
    return e && *e ? (size_t)strtoull(e, nullptr, 10) : LISTS_BYTES;
  }
  std::map<std::vector<int>, List> by_shape_;
  size_t held_ = 0;
};

}  // namespace bta
