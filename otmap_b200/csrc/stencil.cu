// The per-iteration stencil work of the solve in two passes over the grid
// (otlib/otsolver_2dgrid.cpp:179-220, 248-261, 467-606):
//
//   k_sweep_sums   reads psi, d_hat, d_prev, r_k, r_{k-1}; per cell the line
//                  coefficients of d_hat (b1, a11) and of d_prev (b2, a22) and their
//                  cross term a12, and 23 partial sums. The last block of an instance
//                  turns them into |d_hat| (early exit, :182), beta (:248-261, with
//                  r(psi - eps d_hat) - r_k = -eps b1 + eps^2 a11, exact for the
//                  quadratic area) and the quartic of the line search for
//                  d = d_hat + beta d_prev (its five sums are polynomials in beta of the
//                  cross sums), then solves the cubic for alpha (:556-595).
//   k_sweep_update reads psi, d_hat, d_prev, r_k; writes d = d_hat + beta d_prev,
//                  psi + alpha d and r_k + alpha b + alpha^2 a (:599-604); the last
//                  block advances the iteration and tests the loop condition (:160).
//
// Geometry: one warp owns a strip of 32 consecutive columns (j, contiguous in memory) and
// Inst::srows rows (32; 64 when the batch has strips to spare, 16, 8 or 4 when it has too few
// to fill the SMs) and walks down it. Grid rows are prefetched asynchronously (cp.async) into
// a per-warp ring of RD rows in shared memory, so RD-2 rows per warp are in flight while
// it computes; the previous vertex-gradient row is kept in registers. The strip's two halo
// columns are staged with the row; neighbours come from the ring. A block is SWARPS strips
// side by side.
// Per cell the arithmetic is the reference's, in FP64, without FMA contraction. The device code
// is in sweep.cuh: small instances run it from one kernel (cluster.cuh).

#include "sweep.cuh"

namespace otm {

template <class RT, bool SPLIT>
__global__ __launch_bounds__(ST) void k_sweep_sums_t(Inst* insts, const int* strip_inst, int base, double* partials) {
  extern __shared__ __align__(16) unsigned char ring_raw[];
  __shared__ double red[32 * SWARPS];
  const int blk = base + blockIdx.x;
  Inst& I = insts[strip_inst[blk]];
  overlap_wait();
  if (!I.active) return;
  const int n = I.n, it = I.it;
  const StripCoord sc = strip_coord(I, blk, threadIdx.x >> 5);
  double acc[S_COUNT];
#pragma unroll
  for (int k = 0; k < S_COUNT; ++k) acc[k] = 0.0;
  sums_strip<RT, SPLIT>(I, it, sc, ring_raw, acc);
  // no overlap_begin: the update's blocks, resident early, take the memory system from the
  // strips still running (1024^2 alone 75.8 us per iteration without, 80.6 with; plain 79.4)
  const double part = block_totals<S_COUNT>(acc, red, threadIdx.x, BlockSync());
  if (threadIdx.x < S_COUNT) partials[(size_t)blk * KA + threadIdx.x] = part;
  if (last_block(&I.counter, I.nstrip)) {
    double S[S_COUNT];
    sum_partials(I, partials, threadIdx.x, S);
    const double total = block_totals<S_COUNT>(S, red, threadIdx.x, BlockSync());
    if (threadIdx.x < S_COUNT) red[threadIdx.x] = total;
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
      for (int k = 0; k < S_COUNT; ++k) S[k] = red[k];
      sums_step(I, S, n, it);
    }
  }
}

template <class RT, bool SPLIT>
__global__ __launch_bounds__(ST) void k_sweep_update_t(Inst* insts, const int* strip_inst, int base,
                                                       double* partials) {
  extern __shared__ __align__(16) unsigned char ring_raw[];
  __shared__ double red[32];
  const int blk = base + blockIdx.x;
  Inst& I = insts[strip_inst[blk]];
  overlap_wait();
  if (!I.active) return;
  const int n = I.n, it = I.it;
  const StripCoord sc = strip_coord(I, blk, threadIdx.x >> 5);
  double mx = update_strip<RT, SPLIT>(I, it, sc, ring_raw);
  overlap_begin();
  mx = block_max(mx, red);
  if (threadIdx.x == 0) partials[(size_t)blk * KA] = mx;
  if (last_block(&I.counter, I.nstrip)) {
    double m = -INFINITY;
    for (int t = threadIdx.x; t < I.nstrip; t += blockDim.x)
      m = fmax(m, __ldcg(&partials[(size_t)(I.strip0 + t) * KA]));
    m = block_max(m, red);
    if (threadIdx.x == 0) update_step(I, m, n, it);
  }
}

int strip_blocks(int n, int srows) {
  const int strips = ((n + srows - 1) / srows) * ((n + SW - 1) / SW);
  return (strips + SWARPS - 1) / SWARPS;
}

using SumsF64 = Ring<3, 2>;
using UpdF64 = Ring<3, 1>;
using SumsSplit = RingS<2>;
using UpdSplit = RingS<1>;

void sweep_attrs(int device) {
  static bool done[64] = {};
  if (device < 64 && done[device]) return;
  OTM_CUDA(cudaFuncSetAttribute(k_sweep_sums_t<SumsF64, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                SWARPS * RD * SumsF64::STAGE_BYTES));
  OTM_CUDA(cudaFuncSetAttribute(k_sweep_update_t<UpdF64, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                SWARPS * RD * UpdF64::STAGE_BYTES));
  OTM_CUDA(cudaFuncSetAttribute(k_sweep_sums_t<SumsSplit, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                SWARPS * RD * SumsSplit::STAGE_BYTES));
  OTM_CUDA(cudaFuncSetAttribute(k_sweep_update_t<UpdSplit, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                SWARPS * RD * UpdSplit::STAGE_BYTES));
  if (device < 64) done[device] = true;
}

void sweep_sums(otm_context* ctx, Inst* d_insts, const int* strip_inst, int base, int nblocks, bool split,
                double* partials) {
  sweep_attrs(ctx->device);
  if (nblocks <= 0) return;
  if (split)
    launch_smem(ctx, "sweep32_sums", k_sweep_sums_t<SumsSplit, true>, nblocks, ST, SWARPS * RD * SumsSplit::STAGE_BYTES,
                d_insts, strip_inst, base, partials);
  else
    launch_smem(ctx, "sweep_sums", k_sweep_sums_t<SumsF64, false>, nblocks, ST, SWARPS * RD * SumsF64::STAGE_BYTES,
                d_insts, strip_inst, base, partials);
}

void sweep_update(otm_context* ctx, Inst* d_insts, const int* strip_inst, int base, int nblocks, bool split,
                  double* partials) {
  sweep_attrs(ctx->device);
  if (nblocks <= 0) return;
  if (split)
    launch_smem(ctx, "sweep32_update", k_sweep_update_t<UpdSplit, true>, nblocks, ST,
                SWARPS * RD * UpdSplit::STAGE_BYTES, d_insts, strip_inst, base, partials);
  else
    launch_smem(ctx, "sweep_update", k_sweep_update_t<UpdF64, false>, nblocks, ST, SWARPS * RD * UpdF64::STAGE_BYTES,
                d_insts, strip_inst, base, partials);
}

}  // namespace otm
