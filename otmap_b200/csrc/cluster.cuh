// The whole solve of a small instance by one thread-block cluster.
//
// At small sizes an iteration's five kernels (launch_iteration) are mostly their own beginnings and
// ends: launches, records and tables read again, code fetched again, last-block elections. Here one
// cluster of up to 16 blocks keeps an instance from its first iteration to its last: the kernels'
// line and strip functions on the same arrays (L2-resident), a hardware cluster barrier between
// the stages (0.6 us with its release and acquire), the size's tables and the instance's record in
// every block's shared memory: each block forms the totals and the step from the partial sums
// itself, all alike, so nothing is handed round. The sums are formed by the kernels' trees over
// the same strips.
//
// Bound by latency (64^2: an iteration is 30000 cycles, 6500 of them barriers, 5000 the step) up to
// the size at which the FP64 and shared-memory rates of 16 SMs bound it. Microseconds per
// iteration by the kernels and so: 20^2 32.7 and 23.2, 32^2 34.4 and 21.1, 50^2 34.5 and 28.3, 64^2
// 25.6 and 16.9, 100^2 35.8 and 30.8, 127^2 35.9 and 31.4; eight 50^2 38.9 and 30.0, eight 100^2 41.0
// and 38.5. With the register transforms 128^2 took 33.3 against 31.6 and 256^2 37.6 against 33.8:
// those keep the kernels, as do batches of more instances than clusters run at once.
#pragma once

#include <type_traits>

#include "sweep.cuh"

namespace otm {

constexpr int CL_T = 256, CL_WARPS = CL_T / 32;  // two sweep blocks of ST threads
constexpr int CL_WARP_BYTES = RD * Ring<3, 2>::STAGE_BYTES;  // a warp's ring, or its lines

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// All threads of the cluster; what each wrote before it is visible to all after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
struct HalfSync {  // the ST threads of a sweep block within the block
  int half;
  __device__ __forceinline__ void operator()() const {
    asm volatile("bar.sync %0, %1;" ::"r"(half + 1), "n"(ST) : "memory");
  }
};

// A thread's place in the cluster, the record and the warps' regions.
struct ClusterBlock {
  const int C = cluster_size(), rank = cluster_rank(), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = warp / SWARPS;
  Inst& I;
  double* partials;
  unsigned char* regions;
  __device__ __forceinline__ ClusterBlock(Inst& rec, double* part, unsigned char* reg)
      : I(rec), partials(part), regions(reg) {}
  __device__ __forceinline__ unsigned char* region() const { return regions + warp * CL_WARP_BYTES; }
  __device__ __forceinline__ unsigned char* ring() const { return regions + half * SWARPS * CL_WARP_BYTES; }
  // f(item) for this warp's share of the items; consecutive ones go to different blocks
  template <class F>
  __device__ __forceinline__ void items(int count, F f) const {
    for (int item = warp * C + rank; item < count; item += CL_WARPS * C) f(item);
  }
};

__device__ __forceinline__ void cluster_sums(const ClusterBlock& B, int it, double* red) {
  const int tid = threadIdx.x % ST;
  for (int b = B.half * B.C + B.rank; b < B.I.nstrip; b += 2 * B.C) {
    double acc[S_COUNT];
#pragma unroll
    for (int k = 0; k < S_COUNT; ++k) acc[k] = 0.0;
    sums_strip<Ring<3, 2>, false>(B.I, it, strip_coord(B.I, B.I.strip0 + b, B.warp % SWARPS), B.ring(), acc);
    const double part = block_totals<S_COUNT>(acc, red, tid, HalfSync{B.half});
    if (tid < S_COUNT) B.partials[(size_t)(B.I.strip0 + b) * KA + tid] = part;
  }
}
// The totals and the step, on the first half of the block.
__device__ __forceinline__ void cluster_step(const ClusterBlock& B, int n, int it, double* red, double* sums) {
  const HalfSync sync{0};
  double S[S_COUNT];
  sum_partials(B.I, B.partials, threadIdx.x, S);
  const double total = block_totals<S_COUNT>(S, red, threadIdx.x, sync);
  if (threadIdx.x < S_COUNT) sums[threadIdx.x] = total;
  sync();
  if (B.warp == 0) {
#pragma unroll
    for (int k = 0; k < S_COUNT; ++k) S[k] = sums[k];
    sums_step(B.I, S, n, it);
  }
}
static_assert(CL_T == 2 * ST && SWEEP_SLOTS - S_COUNT >= SWARPS, "two sweep blocks; slots for the maxima");
__device__ __forceinline__ void cluster_update(const ClusterBlock& B, int it) {
  for (int b = B.half * B.C + B.rank; b < B.I.nstrip; b += 2 * B.C) {
    const int w = B.warp % SWARPS;
    const double m = warp_max(update_strip<Ring<3, 1>, false>(B.I, it, strip_coord(B.I, B.I.strip0 + b, w), B.ring()));
    // slots that no block still reads sums from
    if (B.lane == 0) B.partials[(size_t)(B.I.strip0 + b) * KA + KA - SWARPS + w] = m;
  }
}

// Transform: the three passes of M^+ over the instance's lines, tables in shared memory:
// table_bytes(n) of it (n <= MAX_N), Transform(I, smem) (fills them), rows_fwd(B, it), cols(B), rows_inv(B).
template <class Transform>
__global__ __launch_bounds__(CL_T, 1) void k_cluster_loop(Inst* insts, double* partials, int table_bytes) {
  extern __shared__ __align__(16) unsigned char cluster_smem[];
  __shared__ __align__(16) Inst I;
  __shared__ double red[2][32 * SWARPS];
  const ClusterBlock B(I, partials, cluster_smem + table_bytes);
  Inst& G = insts[blockIdx.x / B.C];
  static_assert(sizeof(Inst) % 8 == 0, "the record is copied by words");
  for (int e = threadIdx.x; e < (int)(sizeof(Inst) / 8); e += CL_T)
    reinterpret_cast<unsigned long long*>(&I)[e] = reinterpret_cast<const unsigned long long*>(&G)[e];
  __syncthreads();
  if (!I.active) return;  // the whole cluster
  const int n = I.n;
  const Transform tr(I, cluster_smem);
  __syncthreads();
  while (true) {
    const int it = I.it;
    tr.rows_fwd(B, it);
    cluster_sync();
    tr.cols(B);
    cluster_sync();
    tr.rows_inv(B);
    cluster_sync();
    cluster_sums(B, it, red[B.half]);
    cluster_sync();
    if (B.half == 0) cluster_step(B, n, it, red[0], red[1]);
    __syncthreads();
    if (!I.active) break;
    cluster_update(B, it);
    cluster_sync();
    double m = -INFINITY;
    for (int e = threadIdx.x; e < I.nstrip * SWARPS; e += CL_T)
      m = fmax(m, __ldcg(&partials[(size_t)(I.strip0 + e / SWARPS) * KA + KA - SWARPS + e % SWARPS]));
    m = block_max(m, red[0]);
    if (threadIdx.x == 0) update_step(I, m, n, it);
    __syncthreads();
    if (!I.active) break;
  }
  // the host watches `active`: cleared when everything else is in place
  if (B.rank == 0 && threadIdx.x == 0) {
    G.it = I.it;
    G.outcome = I.outcome;
    G.use_beta = I.use_beta;
    G.residual = I.residual;
    G.alpha = I.alpha;
    G.beta = I.beta;
    G.linf = I.linf;
    G.dnorm = I.dnorm;
    __threadfence();
    *const_cast<volatile int*>(&G.active) = 0;
  }
}

template <class Transform>
cudaLaunchConfig_t cluster_config(otm_context* ctx, int n, int count, int blocks, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(count * blocks);
  cfg.blockDim = dim3(CL_T);
  cfg.dynamicSmemBytes = Transform::table_bytes(n) + (size_t)CL_WARPS * CL_WARP_BYTES;
  cfg.stream = ctx->stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim = {(unsigned)blocks, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// The kernel's limits, the same for every size it takes: another thread may be launching it.
template <class Transform>
void cluster_attrs() {
  const auto kernel = k_cluster_loop<Transform>;
  OTM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                Transform::table_bytes(Transform::MAX_N) + CL_WARPS * CL_WARP_BYTES));
  OTM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

// Blocks per cluster (16, else 8) with which `count` clusters run at once, or 0.
template <class Transform>
int cluster_blocks(otm_context* ctx, int n, int count) {
  cluster_attrs<Transform>();
  for (int c : {16, 8}) {
    cudaLaunchAttribute attr = {};
    const cudaLaunchConfig_t cfg = cluster_config<Transform>(ctx, n, count, c, &attr);
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, k_cluster_loop<Transform>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      fit = 0;
    }
    if (fit >= count) return c;
  }
  return 0;
}
template <class Transform>
void cluster_launch(otm_context* ctx, int n, int count, int blocks, Inst* d_insts, double* partials) {
  cudaLaunchAttribute attr = {};
  const cudaLaunchConfig_t cfg = cluster_config<Transform>(ctx, n, count, blocks, &attr);
  ctx->launches++;
  OTM_CUDA(cudaLaunchKernelEx(&cfg, k_cluster_loop<Transform>, d_insts, partials, Transform::table_bytes(n)));
}

}  // namespace otm
