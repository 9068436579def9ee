// Shared device/host helpers for the otmap_b200 CUDA library.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <string>

#include "async_buf.h"

namespace otm {

// Thread-local message behind otm_last_error().
void set_error(const std::string& msg);

struct BadArg {
  std::string what;
};

// A bounded device-side wait gave up (reported as OTM_ERR_TIMEOUT).
struct DeviceTimeout {
  std::string what;
};

// True when p points into device (or managed) memory; host pointers, registered
// or not, report false.
inline bool is_device_ptr(const void* p) {
  if (!p) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// ---- device-side reductions (fixed order: results are run-to-run identical) ----

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sums of K values per thread; result valid in thread 0. `red` is
// shared scratch of K * 32 doubles. Blocks are multiples of 32 threads.
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = warp_sum(v[k]);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) red[k * 32 + warp] = v[k];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double x = lane < nw ? red[k * 32 + lane] : 0.0;
      v[k] = warp_sum(x);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ double block_max(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) v = warp_max(lane < nw ? red[lane] : -INFINITY);
  __syncthreads();
  return v;
}

// ---- programmatic dependent launch ----
//
// A kernel launched with ctx->overlap (context.h) may start while the one before it in the
// stream still runs. It reads or writes nothing that another kernel changes before
// overlap_wait, which returns when the kernel before it has completed with its writes visible;
// no block leaves before that wait, so a kernel's end implies the end of all before it. Tables
// and work lists may be read earlier, with loads that leave no copy in L1 of lines the wait
// should see fresh. overlap_begin lets the successor's blocks take the places that this
// kernel's have left: it stands behind the main loop, since blocks that only wait slow the ones
// at work -- but on entry in the register transforms of small batches, which leave most of the
// chip free (OVERLAP_EARLY_CELLS). In a kernel launched plainly both are no-ops.
__device__ __forceinline__ void overlap_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class T>
__device__ __forceinline__ const T* early_pointer(const T* const* p) {  // a pointer field, past L1
  return reinterpret_cast<const T*>(__ldcg(reinterpret_cast<const unsigned long long*>(p)));
}
__device__ __forceinline__ void overlap_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// "Last block" election for a reduction spread over `total` blocks that share
// `counter`: every block calls it once after thread 0 has written the block's
// partials; it returns true (in all threads) in exactly one block, the last to
// arrive, which may then read every block's partials. The counter is reset for
// the next kernel by the last block.
__device__ __forceinline__ bool last_block(unsigned int* counter, unsigned int total) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int prev = atomicAdd(counter, 1u);
    s_last = (prev == total - 1u);
    if (s_last) *counter = 0u;
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// std::max / std::min semantics (NaN in the second argument yields the first).
__host__ __device__ __forceinline__ double std_max(double a, double b) { return a < b ? b : a; }
__host__ __device__ __forceinline__ double std_min(double a, double b) { return b < a ? b : a; }

}  // namespace otm
