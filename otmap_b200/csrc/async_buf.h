// Device memory in stream order, and the error that a failed CUDA call throws. Host code only.
#pragma once

#include <cuda_runtime_api.h>

#include <string>

namespace otm {

struct CudaError {
  cudaError_t code;
  std::string where;
};

#define OTM_CUDA(call)                                                                  \
  do {                                                                                  \
    cudaError_t _e = (call);                                                            \
    if (_e != cudaSuccess)                                                              \
      throw ::otm::CudaError{_e, std::string(#call) + " at " + __FILE__ + ":" +         \
                                     std::to_string(__LINE__)};                         \
  } while (0)

// Device buffer from the stream-ordered allocator (cudaMallocFromPoolAsync / cudaFreeAsync
// from one of the context's memory pools): freeing it does not synchronise the device, and the pool
// hands the memory to the next allocation. It is freed on its home stream, after the work
// queued there: the stream of its last users, which need not be the one it is reserved on. Used for
// the per-map buffers, which live and die with each TransportMap, and for the temporaries of
// a call (a cudaMalloc and cudaFree of 25 MB cost a 512^2 barycenter image 0.4 ms).
struct AsyncBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaStream_t home = nullptr;
  AsyncBuf() = default;
  AsyncBuf(const AsyncBuf&) = delete;
  AsyncBuf& operator=(const AsyncBuf&) = delete;
  ~AsyncBuf() { release(); }
  void release() {
    if (p) cudaFreeAsync(p, home);
    p = nullptr;
    bytes = 0;
  }
  // Grows (never shrinks) to at least `b` bytes on stream s from `pool`; contents are not
  // preserved.
  void reserve(size_t b, cudaStream_t s, cudaMemPool_t pool) { reserve(b, s, pool, s); }
  void reserve(size_t b, cudaStream_t s, cudaMemPool_t pool, cudaStream_t home_stream) {
    if (b > bytes) {
      release();
      OTM_CUDA(cudaMallocFromPoolAsync(&p, b, pool, s));
      bytes = b;
    }
    home = home_stream;
  }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

}  // namespace otm
