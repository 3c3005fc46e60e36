// Scratch memory from the stream-ordered pool, given back on its stream when it goes
// out of scope: also when a later allocation, kernel load or launch throws.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>

namespace mapb {

class StreamMemory {
 public:
  explicit StreamMemory(cudaStream_t st) : st_(st) {}
  StreamMemory(const StreamMemory &) = delete;
  StreamMemory &operator=(const StreamMemory &) = delete;
  ~StreamMemory() {
    if (p_) cudaFreeAsync(p_, st_);
  }
  // cudaSuccess, or the error (no memory is held then, and the error is not left behind
  // for the next check of an asynchronous one)
  cudaError_t alloc(size_t bytes) {
    const cudaError_t e = cudaMallocAsync(&p_, bytes, st_);
    if (e != cudaSuccess) {
      p_ = nullptr;
      cudaGetLastError();
    }
    return e;
  }
  void *ptr() const { return p_; }
  // the memory, no longer given back by this object
  void *release() {
    void *p = p_;
    p_ = nullptr;
    return p;
  }

 private:
  cudaStream_t st_;
  void *p_ = nullptr;
};

}  // namespace mapb
