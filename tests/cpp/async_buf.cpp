// AsyncBuf against a recording stand-in for the allocator: prints the stream of every allocation and
// free. Streams 1 and 2 are the context's and its side stream.
#include <cstdio>
#include <cstdlib>

#include "async_buf.h"

static int id(cudaStream_t s) { return (int)reinterpret_cast<size_t>(s); }
extern "C" cudaError_t CUDARTAPI cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t s) {
  std::printf("m%d ", id(s));
  *p = std::malloc(1);
  return cudaSuccess;
}
extern "C" cudaError_t CUDARTAPI cudaFreeAsync(void* p, cudaStream_t s) {
  std::printf("f%d ", id(s));
  std::free(p);
  return cudaSuccess;
}

int main() {
  const auto home = reinterpret_cast<cudaStream_t>(1), side = reinterpret_cast<cudaStream_t>(2);
  {
    otm::AsyncBuf plain, filled_beside;
    plain.reserve(100, home, nullptr);
    filled_beside.reserve(100, side, nullptr, home);
    filled_beside.reserve(50, side, nullptr, home);
    filled_beside.reserve(200, side, nullptr, home);
  }
  std::printf("\n");
}
