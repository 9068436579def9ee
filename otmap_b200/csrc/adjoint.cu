// Implicit adjoint of a converged transport map with respect to its input density.
//
// The reference has no derivative; this follows from its equations. The solve drives
// the area residual F(psi, rho~) = A(psi) - e^2 rho~ to zero (otsolver_2dgrid.cpp:449-465)
// where A(psi) is the area of each quad of the grid displaced by the vertex gradients
// g = G psi (otsolver_2dgrid.cpp:362-447) and rho~ = adjust(rho) (otsolver_2dgrid.cpp:47-63).
// For a loss L(fwd) of the forward mesh fwd = grid + g, with q = dL/dfwd (per vertex):
//   dL/dpsi   = G^T q
//   J^T lambda = G^T q,  J = dA/dpsi = (dA/dg) G      (mean-zero subspace: J 1 = 0, 1^T J = 0)
//   dL/drho~  = e^2 lambda
//   dL/drho   = (lambda - (lambda . rho) / S) / S,  S = sum(rho)   (ratio clamp inactive)
// J^T is applied matrix-free (jt_cell): h_v = sum_c lambda_c dA_c/dg_v over the four cells
// around each vertex (dA_c/dD1 = (D2y, -D2x)/2, dA_c/dD2 = (-D1y, D1x)/2 with the cell
// diagonals D1 = g11 - g00 + (e,e), D2 = g01 - g10 + (-e,e)), then (G^T h)_f over every vertex
// whose clamped gradient stencil touches cell f. Both are deterministic gathers. lambda solves J^T lambda = b by restarted GMRES right-
// preconditioned with the pseudo-inverse of M (the reference's pseudo-Laplacian; J = -M at
// psi = 0), using the same cosine-transform Poisson solve as the forward loop; the
// one-step mode stops at lambda = -M^+ b (one Poisson solve). For strongly deformed maps
// J departs far from -M (a plain preconditioned fixed-point iteration diverges there),
// hence the Krylov method.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "engine.cuh"

namespace otm {

__device__ __forceinline__ int clampv(int v, int n) { return v < 0 ? 0 : (v >= n ? n - 1 : v); }

// Device state of one restart cycle of the Krylov solve. The cycle's Arnoldi steps run on
// the device (a CUDA graph with a WHILE node, or the same kernels launched one step at a
// time): every step kernel reads the step index j here instead of taking it as a launch
// argument; the last kernel of a step advances it and decides whether the cycle goes on.
struct AdjCtl {
  int j;       // the step being taken: basis vectors 0..j are orthonormal
  int go;      // the cycle takes another step
  int live;    // the map takes part in the cycle
  int m;       // restart length
  int budget;  // steps allowed in this cycle (the call's cap on Poisson solves)
  double bnorm, tol;
  double rnorm;          // norm of the vector last formed by k_adj_resid
  unsigned int counter;  // block ticket of the running kernel
  int fault;             // the steps' transform gave up a bounded wait
};

// The adjoints of up to 8 maps of one size run together: block row y of every kernel works
// for map y, on the map's own control block and its own slice of the workspace (the
// pointers of map 0 plus y times the stride).
constexpr int ADJ_MAPS = 8;
struct AdjArgs {  // the call's buffers per map
  const double* fwd[ADJ_MAPS];
  const double* q[ADJ_MAPS];
  const double* rho[ADJ_MAPS];
  double* out[ADJ_MAPS];
};
struct AdjCycle {  // a restart cycle's parameters per map
  double bnorm[ADJ_MAPS];
  int budget[ADJ_MAPS], live[ADJ_MAPS];
};

// Displacements g of the vertices from the forward mesh.
__global__ void k_adj_disp(int n, AdjArgs args, double2* g, long stride) {
  const double* fwd = args.fwd[blockIdx.y];
  g += blockIdx.y * (stride / 2);
  const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (long)(n + 1) * (n + 1)) return;
  const double dx = 1.0 / (double)n;
  g[v] = make_double2(fwd[2 * v] - (double)(v / (n + 1)) * dx, fwd[2 * v + 1] - (double)(v % (n + 1)) * dx);
}

// (G^T h)_f: vertex (vi, vj) reads cells (clamp(vi-1+a), clamp(vj-1+b)), a, b in {0, 1},
// with gx coefficient (2a-1) n/2 and gy coefficient (2b-1) n/2
// (otsolver_2dgrid.cpp:379-422 with clamped indices). Cell (i, j) collects every
// (vertex, a, b) whose clamped position is (i, j).
__global__ void k_adj_cells(int n, AdjArgs args, double* out, long stride) {
  const double* h = args.q[blockIdx.y];
  out += blockIdx.y * stride;
  const long f = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= (long)n * n) return;
  const int i = (int)(f / n), j = (int)(f % n);
  // row choices: (vi, a) with clamp(vi - 1 + a) == i
  int ri[3], ra[3], nr = 0;
  ri[nr] = i + 1; ra[nr++] = 0;
  ri[nr] = i; ra[nr++] = 1;
  if (i == 0) { ri[nr] = 0; ra[nr++] = 0; }
  if (i == n - 1) { ri[nr] = n; ra[nr++] = 1; }
  int cj[3], cb[3], nc = 0;
  cj[nc] = j + 1; cb[nc++] = 0;
  cj[nc] = j; cb[nc++] = 1;
  if (j == 0) { cj[nc] = 0; cb[nc++] = 0; }
  if (j == n - 1) { cj[nc] = n; cb[nc++] = 1; }
  const double hw = 0.5 * (double)n;
  double acc = 0.0;
  for (int p = 0; p < nr; ++p)
    for (int q = 0; q < nc; ++q) {
      const size_t v = (size_t)cj[q] + (size_t)ri[p] * (n + 1);
      acc += hw * ((2 * ra[p] - 1) * h[2 * v] + (2 * cb[q] - 1) * h[2 * v + 1]);
    }
  out[f] = acc;
}

// ---- the Arnoldi step ----
//
// After z = M^+ v_j a step is four kernels: w = J^T z with its products with v_0..v_j
// (k_adj_apply), the first Gram-Schmidt update with the products of the second
// (k_adj_orth), the second update with the norm, the Givens rotation and the loop test
// (k_adj_norm), and the normalisation (k_adj_scale_by). At 256^2 a step is bound by the
// latency of launches and grid-wide reductions, not by the basis it reads from L2 (10 MB a
// pass on average), so every reduction ends in the last block of the kernel that forms its
// terms. Against one kernel per operation (source, vertices, cells, 3 x products, 3 x
// one-block sums, 2 x update, scale, rotation) a step with its transform went from 96 to
// 51 us at 256^2 (four maps: 147 to 80), from 159 to 85 us at 512^2.
//
// Cell f belongs to block (f / 256) mod 256 and thread f mod 256; a thread's cells (one for
// N <= 65536) follow each other 65536 apart. A product is an FMA chain over a thread's cells,
// a fixed tree over the block's threads and a sum over the blocks in block order: the order
// is that of a grid of 256 blocks whatever the grid launched, so results do not depend on
// the device.

constexpr int AT = 256;         // threads per block
constexpr int ANB = 256;        // blocks (fewer when the cells run out)
constexpr int ADJ_MAX_M = 200;  // largest restart length
constexpr int DOT_CHUNK = 8;    // products formed per pass over a thread's cells

// (J^T lambda)_f of cell (i, j), gathered from the 3 x 3 cells and 4 x 4 vertices around it
// (g: vertex displacements). h_v = sum over the cells c around vertex v of
// lambda_c dA_c / dg_v: v00 of the cell at (vi, vj) takes -dA/dD1, v10 of (vi-1, vj) -dA/dD2,
// v01 of (vi, vj-1) dA/dD2, v11 of (vi-1, vj-1) dA/dD1.
__device__ __forceinline__ double jt_cell(int n, const double2* g, const double* lambda, int i, int j) {
  const double e = 1.0 / (double)n, hw = 0.5 * (double)n;
  double2 d1[3][3], d2[3][3];  // lambda/2 D1 and lambda/2 D2 of the cells around (i, j)
  double2 p[2][4];             // vertex rows i-1+r, i+r
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int vi = i - 1, vj = j - 1 + c;
    p[0][c] = vi >= 0 && vj >= 0 && vj <= n ? g[(size_t)vi * (n + 1) + vj] : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int vi = i + r, vj = j - 1 + c;
      p[(r + 1) & 1][c] = vi <= n && vj >= 0 && vj <= n ? g[(size_t)vi * (n + 1) + vj] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int ci = i - 1 + r, cj = j - 1 + c;
      const double l = ci >= 0 && cj >= 0 && ci < n && cj < n ? 0.5 * lambda[(size_t)ci * n + cj] : 0.0;
      const double2 g00 = p[r & 1][c], g01 = p[r & 1][c + 1], g10 = p[(r + 1) & 1][c], g11 = p[(r + 1) & 1][c + 1];
      d1[r][c] = make_double2(l * (g11.x - g00.x + e), l * (g11.y - g00.y + e));
      d2[r][c] = make_double2(l * (g01.x - g10.x - e), l * (g01.y - g10.y + e));
    }
  }
  double2 h[2][2];  // vertices (i, j) .. (i+1, j+1)
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
      h[a][b] = make_double2(((d1[a][b + 1].y - d2[a + 1][b + 1].y) - d1[a + 1][b].y) + d2[a][b].y,
                             ((d2[a + 1][b + 1].x - d1[a][b + 1].x) + d1[a + 1][b].x) - d2[a][b].x);
  // k_adj_cells' gather: vertex rows (i+1, a = 0), (i, a = 1) and, at the border, the clamped ones
  double acc = 0.0;
  auto add = [&](const double2& v, int a, int b) { acc += hw * ((a ? v.x : -v.x) + (b ? v.y : -v.y)); };
  auto row = [&](const double2 (&v)[2], int a) {
    add(v[1], a, 0);
    add(v[0], a, 1);
    if (j == 0) add(v[0], a, 0);
    if (j == n - 1) add(v[1], a, 1);
  };
  row(h[1], 0);
  row(h[0], 1);
  if (i == 0) row(h[0], 0);
  if (i == n - 1) row(h[1], 1);
  return acc;
}

// Warp totals of s[0..7], each by the tree of warp_sum; afterwards s[0] on lane l is the
// total of value 4 (l>>4 & 1) + 2 (l>>3 & 1) + (l>>2 & 1). Nine shuffles instead of the 40
// of eight separate trees.
__device__ __forceinline__ void warp_sum8(double (&s)[8], int lane) {
#pragma unroll
  for (int o = 16, h = 4; h >= 1; o >>= 1, h >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const double send = up ? s[q] : s[q + h], keep = up ? s[q + h] : s[q];
      s[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
  s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
}

// block_sum's tree over the eight warps' values.
__device__ __forceinline__ double sum_warps(const double* r, int stride) {
  static_assert(AT / 32 == 8, "eight warps");
  return ((r[0] + r[4 * stride]) + (r[2 * stride] + r[6 * stride])) +
         ((r[stride] + r[5 * stride]) + (r[3 * stride] + r[7 * stride]));
}

// partial[i * ANB + block] = this block's part of w . V_i, i < P. The loads of a thread's
// next chunk of vectors are issued before the current chunk is reduced.
constexpr int RED_LD = ADJ_MAX_M + 8;
__device__ __forceinline__ void block_dots(long N, const double* w, const double* V, long ld, int P, double* red,
                                           double* partial) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long f0 = (long)blockIdx.x * AT + threadIdx.x;
  if (N <= (long)ANB * AT) {  // one cell per thread
    const bool in = f0 < N;
    const double wf = in ? w[f0] : 0.0;
    double v[DOT_CHUNK];
    auto fetch = [&](int i0) {
#pragma unroll
      for (int c = 0; c < DOT_CHUNK; ++c) v[c] = in && i0 + c < P ? V[(size_t)(i0 + c) * ld + f0] : 0.0;
    };
    fetch(0);
    for (int i0 = 0; i0 < P; i0 += DOT_CHUNK) {
      double s[DOT_CHUNK];
#pragma unroll
      for (int c = 0; c < DOT_CHUNK; ++c) s[c] = fma(wf, v[c], 0.0);
      fetch(i0 + DOT_CHUNK);
      warp_sum8(s, lane);
      const int i = i0 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
      if ((lane & 3) == 0 && i < P) red[warp * RED_LD + i] = s[0];
    }
  } else {
    for (int i0 = 0; i0 < P; i0 += DOT_CHUNK) {
      double s[DOT_CHUNK];
#pragma unroll
      for (int c = 0; c < DOT_CHUNK; ++c) s[c] = 0.0;
#pragma unroll 2
      for (long f = f0; f < N; f += (long)ANB * AT) {
        const double wf = w[f];
#pragma unroll
        for (int c = 0; c < DOT_CHUNK; ++c)
          if (i0 + c < P) s[c] = fma(wf, V[(size_t)(i0 + c) * ld + f], s[c]);
      }
      warp_sum8(s, lane);
      const int i = i0 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
      if ((lane & 3) == 0 && i < P) red[warp * RED_LD + i] = s[0];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < P; i += AT) partial[(size_t)i * ANB + blockIdx.x] = sum_warps(red + i, RED_LD);
}

// Last block: out(i, total) for the P totals of the blocks' partials. Each is a chain of adds
// in block order on one thread (the order that fixes the result), so all values' chains run
// at once and the partials come through shared memory in tiles, the next tile's loads in
// flight during a tile's adds.
constexpr int TOT_V = 48, TOT_B = 64;  // values and blocks per tile
constexpr int TOT_STAGE = TOT_V * (TOT_B + 1);
template <class F>
__device__ __forceinline__ void totals(const double* partial, int P, double* stage, F out) {
  constexpr int PER = TOT_V * TOT_B / AT;
  const int nb = gridDim.x, b = threadIdx.x % TOT_B, v0 = threadIdx.x / TOT_B;
  for (int i0 = 0; i0 < P; i0 += TOT_V) {
    const int cnt = min(TOT_V, P - i0);
    double next[PER], t = 0.0;
    auto fetch = [&](int b0) {
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int i = v0 + k * (AT / TOT_B);
        next[k] = i < cnt && b0 + b < nb ? __ldcg(&partial[(size_t)(i0 + i) * ANB + b0 + b]) : 0.0;
      }
    };
    fetch(0);
    for (int b0 = 0; b0 < nb; b0 += TOT_B) {
      __syncthreads();
#pragma unroll
      for (int k = 0; k < PER; ++k) stage[(v0 + k * (AT / TOT_B)) * (TOT_B + 1) + b] = next[k];
      __syncthreads();
      fetch(b0 + TOT_B);
      if (threadIdx.x < cnt) {
        const double* s = stage + threadIdx.x * (TOT_B + 1);
        if (b0 + TOT_B <= nb) {
#pragma unroll 16
          for (int k = 0; k < TOT_B; ++k) t += s[k];
        } else {
          for (int k = 0; k < nb - b0; ++k) t += s[k];
        }
      }
    }
    if (threadIdx.x < cnt) out(i0 + threadIdx.x, t);
  }
}

// w = V_{j+1} = J^T z (z = M^+ v_j); Hessenberg column and combine coefficients c_i of the
// first Gram-Schmidt pass.
__global__ __launch_bounds__(AT) void k_adj_apply(int n, const double2* g, const double* z, double* V, long ld,
                                                  AdjCtl* ctl, double* partial, double* hcol, double* c, long stride) {
  __shared__ double red[AT / 32 * RED_LD], stage[TOT_STAGE];
  const long off = blockIdx.y * stride;
  overlap_wait();
  ctl += blockIdx.y;
  if (!ctl->go) return;
  g += off / 2;
  z += off;
  V += off;
  partial += off;
  hcol += off;
  c += off;
  const int j = ctl->j, P = j + 1;
  const long N = (long)n * n;
  double* w = V + (size_t)(j + 1) * ld;
  for (long f = (long)blockIdx.x * AT + threadIdx.x; f < N; f += (long)ANB * AT)
    w[f] = jt_cell(n, g, z, (int)(f / n), (int)(f % n));
  block_dots(N, w, V, ld, P, red, partial);
  overlap_begin();
  if (!last_block(&ctl->counter, gridDim.x)) return;
  totals(partial, P, stage, [&](int i, double d) {
    c[i] = d;
    hcol[i] = 0.0 + d;
  });
}

// w -= sum_i c_i V_i at this thread's cells; returns the chain of the new w^2 there.
__device__ __forceinline__ double combine(long N, double* w, const double* V, long ld, int P, const double* c,
                                          double* sc) {
  for (int i = threadIdx.x; i < P; i += AT) sc[i] = c[i];
  __syncthreads();
  double ss = 0.0;
  for (long f = (long)blockIdx.x * AT + threadIdx.x; f < N; f += (long)ANB * AT) {
    double x = w[f];
#pragma unroll 16
    for (int i = 0; i < P; ++i) x = fma(-sc[i], V[(size_t)i * ld + f], x);
    w[f] = x;
    ss = fma(x, x, ss);
  }
  return ss;
}

// First Gram-Schmidt update and the products of the second pass. With one cell per thread and
// a basis of at most ORTH_V vectors (a default cycle) the thread's basis values stay in
// registers between the two, all their loads in flight together.
constexpr int ORTH_V = 40;
__global__ __launch_bounds__(AT) void k_adj_orth(int n, double* V, long ld, AdjCtl* ctl, double* partial, double* hcol,
                                                 double* c, long stride) {
  __shared__ double sc[ADJ_MAX_M + 8], red[AT / 32 * RED_LD], stage[TOT_STAGE];
  const long off = blockIdx.y * stride;
  overlap_wait();
  ctl += blockIdx.y;
  if (!ctl->go) return;
  V += off;
  partial += off;
  hcol += off;
  c += off;
  const int j = ctl->j, P = j + 1;
  const long N = (long)n * n;
  double* w = V + (size_t)(j + 1) * ld;
  if (N <= (long)ANB * AT && P <= ORTH_V) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long f = (long)blockIdx.x * AT + threadIdx.x;
    const bool in = f < N;
    double v[ORTH_V], x = in ? w[f] : 0.0;
#pragma unroll
    for (int i0 = 0; i0 < ORTH_V; i0 += DOT_CHUNK)
      if (i0 < P) {
#pragma unroll
        for (int k = i0; k < i0 + DOT_CHUNK; ++k) v[k] = in && k < P ? V[(size_t)k * ld + f] : 0.0;
      }
    for (int i = threadIdx.x; i < P; i += AT) sc[i] = c[i];
    __syncthreads();
#pragma unroll
    for (int i0 = 0; i0 < ORTH_V; i0 += DOT_CHUNK)
      if (i0 < P) {
#pragma unroll
        for (int k = i0; k < i0 + DOT_CHUNK; ++k)
          if (k < P) x = fma(-sc[k], v[k], x);
      }
    if (in) w[f] = x;
#pragma unroll
    for (int i0 = 0; i0 < ORTH_V; i0 += DOT_CHUNK)
      if (i0 < P) {
        double s[DOT_CHUNK];
#pragma unroll
        for (int k = 0; k < DOT_CHUNK; ++k) s[k] = fma(x, v[i0 + k], 0.0);
        warp_sum8(s, lane);
        const int i = i0 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
        if ((lane & 3) == 0 && i < P) red[warp * RED_LD + i] = s[0];
      }
    __syncthreads();
    for (int i = threadIdx.x; i < P; i += AT) partial[(size_t)i * ANB + blockIdx.x] = sum_warps(red + i, RED_LD);
  } else {
    combine(N, w, V, ld, P, c, sc);
    block_dots(N, w, V, ld, P, red, partial);
  }
  overlap_begin();
  if (!last_block(&ctl->counter, gridDim.x)) return;
  totals(partial, P, stage, [&](int i, double d) {
    c[i] = d;
    hcol[i] = hcol[i] + d;
  });
}

// Second Gram-Schmidt update and H_{j+1,j} = |w|; then, on one thread, the end of step j: the
// previous Givens rotations applied to the new Hessenberg column, the rotation that zeroes
// H_{j+1,j}, the updated residual estimate |g_{j+1}|, and the loop test: go on while it is
// above tol * |b|, the new basis vector is non-zero, the cycle has room, the call's budget
// is not spent and the transform has not given up a wait. H is (m+1) x m, row-major. The
// Poisson record of the next step gets its source.
__global__ __launch_bounds__(AT) void k_adj_norm(int n, double* V, long ld, AdjCtl* ctl, double* inv, double* partial,
                                                 const double* hcol, const double* c, double* H, double* cs, double* sn,
                                                 double* gv, Inst* rec, long stride) {
  __shared__ double sc[ADJ_MAX_M + 8], sh[ADJ_MAX_M + 8], ss[ADJ_MAX_M + 8], red[64], stage[TOT_STAGE];
  const long off = blockIdx.y * stride;
  overlap_wait();
  ctl += blockIdx.y;
  if (!ctl->go) return;
  V += off;
  inv += off;
  partial += off;
  hcol += off;
  c += off;
  H += off;
  cs += off;
  sn += off;
  gv += off;
  rec += blockIdx.y;
  const int j = ctl->j, P = j + 1;
  const long N = (long)n * n;
  double v[1] = {combine(N, V + (size_t)(j + 1) * ld, V, ld, P, c, sc)};
  overlap_begin();
  block_sum<1>(v, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = v[0];
  if (!last_block(&ctl->counter, gridDim.x)) return;
  for (int i = threadIdx.x; i < j; i += AT) {
    sc[i] = cs[i];
    ss[i] = sn[i];
  }
  for (int i = threadIdx.x; i <= j; i += AT) sh[i] = hcol[i];
  const int m = ctl->m;
  totals(partial, 1, stage, [&](int, double w2) {
    const double hn = sqrt(w2);
    double x = sh[0];
    for (int i = 0; i < j; ++i) {
      const double y = sh[i + 1];
      sh[i] = sc[i] * x + ss[i] * y;
      x = -ss[i] * x + sc[i] * y;
    }
    const double den = hypot(x, hn);
    const double cj = den > 0 ? x / den : 1.0, sj = den > 0 ? hn / den : 0.0;
    sh[j] = den;
    cs[j] = cj;
    sn[j] = sj;
    const double gj = gv[j], gk = -sj * gj;
    gv[j + 1] = gk;
    gv[j] = cj * gj;
    *inv = hn > 0 ? 1.0 / hn : 1.0;
    const int k = j + 1;
    const int go = (fabs(gk) / ctl->bnorm > ctl->tol) && hn != 0 && k < m && k < ctl->budget && !rec->fault;
    ctl->j = k;
    ctl->go = go;
    rec->r[0] = V + (size_t)k * ld;
    rec->active = go;
    ctl->fault = rec->fault;
  });
  __syncthreads();
  for (int i = threadIdx.x; i <= j; i += AT) H[(size_t)i * m + j] = sh[i];
}

// v_j = w / |w|, the vector k_adj_norm has just moved the cycle on to (the last one of a
// cycle is not used). The step's last kernel: in the graph it keeps the WHILE node going
// while any map's cycle goes on.
__global__ void k_adj_scale_by(long N, double* V, long ld, const double* a, const AdjCtl* ctl, long stride,
                               cudaGraphConditionalHandle handle, int in_graph) {
  overlap_wait();
  if (in_graph && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    int any = 0;
    for (int y = 0; y < (int)gridDim.y; ++y) any |= ctl[y].go;
    cudaGraphSetConditional(handle, any ? 1u : 0u);
  }
  ctl += blockIdx.y;
  if (!ctl->go) return;
  const long f = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f < N) V[blockIdx.y * stride + (size_t)ctl->j * ld + f] *= a[blockIdx.y * stride];
}

// Every Poisson record of the workspace ready for a new call: a bounded wait that gave up in
// an earlier call stopped its record and flagged it.
__global__ void k_adj_reset_recs(Inst* recs, int count) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) {
    recs[k].active = 1;
    recs[k].fault = 0;
  }
}

// Start of a restart cycle from the vector in V_0, whose norm k_adj_resid left in the state:
// v_0, g, the cycle's state and the Poisson records of its steps (rec) and of its end (rec_h).
__global__ void k_adj_cycle_init(long N, AdjCtl* ctl, double* gv, int m, AdjCycle cyc, double tol, Inst* rec,
                                 Inst* rec_h, double* V, long stride) {
  const int y = blockIdx.y;
  ctl += y;
  const int live = cyc.live[y];
  const double rnorm = ctl->rnorm, a = 1.0 / rnorm;
  const long f = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f < N && live) V[y * stride + f] *= a;
  if (f <= m) gv[y * stride + f] = f ? 0.0 : rnorm;
  if (f != 0) return;
  ctl->live = live;
  ctl->j = 0;
  ctl->go = live && cyc.budget[y] > 0 ? 1 : 0;
  ctl->m = m;
  ctl->budget = cyc.budget[y];
  ctl->bnorm = cyc.bnorm[y];
  ctl->tol = tol;
  ctl->fault = rec[y].fault;
  rec[y].r[0] = V + y * stride;
  rec[y].active = live && !rec[y].fault;
  rec_h[y].active = live && !rec_h[y].fault;
}

// H y = g for the k = j steps of the cycle: y into c (row-oriented back substitution by one
// thread, on a shared copy of the triangle: read where it lies, each of its k^2 / 2 elements
// was a wait on L2, 51 us at k = 40).
__global__ __launch_bounds__(256) void k_adj_trisolve(const AdjCtl* ctl, const double* H, const double* gv, double* c,
                                                      long stride) {
  constexpr int KS = 64;  // triangles up to this order are staged; larger ones are read where they lie
  __shared__ double sH[KS * KS], y[ADJ_MAX_M + 8];
  ctl += blockIdx.y;
  if (!ctl->live) return;
  H += blockIdx.y * stride;
  gv += blockIdx.y * stride;
  c += blockIdx.y * stride;
  const int k = ctl->j, m = ctl->m;
  const bool staged = k <= KS;
  if (staged)
    for (int q = threadIdx.x; q < k * k; q += blockDim.x) sH[q] = H[(size_t)(q / k) * m + q % k];
  for (int i = threadIdx.x; i < k; i += blockDim.x) y[i] = gv[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    const double* R = staged ? sH : H;
    const int ldr = staged ? k : m;
    for (int i = k - 1; i >= 0; --i) {
      double t = y[i];
#pragma unroll 8
      for (int l = i + 1; l < k; ++l) t -= R[(size_t)i * ldr + l] * y[l];
      y[i] = t / R[(size_t)i * ldr + i];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < k; i += blockDim.x) c[i] = y[i];
}

// out = sum_i c_i v_i over the cycle's steps
__global__ void k_adj_span(long N, double* out, const double* V, long ld, const double* c, const AdjCtl* ctl,
                           long stride) {
  ctl += blockIdx.y;
  if (!ctl->live) return;
  out += blockIdx.y * stride;
  V += blockIdx.y * stride;
  c += blockIdx.y * stride;
  const int m = ctl->j;
  const long f = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= N) return;
  double x = 0.0;
#pragma unroll 8
  for (int i = 0; i < m; ++i) x = fma(c[i], V[(size_t)i * ld + f], x);
  out[f] = x;
}

// v = b - J^T lambda for the maps of the last cycle (lambda null: v = b, every map) and its
// norm into the state.
__global__ __launch_bounds__(AT) void k_adj_resid(int n, const double2* g, const double* lambda, const double* b,
                                                  double* v, AdjCtl* ctl, double* partial, long stride) {
  __shared__ double red[64], stage[TOT_STAGE];
  ctl += blockIdx.y;
  if (lambda) {
    if (!ctl->live) return;
    lambda += blockIdx.y * stride;
  }
  g += blockIdx.y * (stride / 2);
  b += blockIdx.y * stride;
  v += blockIdx.y * stride;
  partial += blockIdx.y * stride;
  const long N = (long)n * n;
  double s[1] = {0.0};
  for (long f = (long)blockIdx.x * AT + threadIdx.x; f < N; f += (long)ANB * AT) {
    double r = b[f];
    if (lambda) r = r - jt_cell(n, g, lambda, (int)(f / n), (int)(f % n));
    v[f] = r;
    s[0] = fma(r, r, s[0]);
  }
  block_sum<1>(s, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
  if (!last_block(&ctl->counter, gridDim.x)) return;
  totals(partial, 1, stage, [&](int, double t) { ctl->rnorm = sqrt(t); });
}

__global__ void k_adj_neg(long N, const double* z, double* lambda, long stride) {
  z += blockIdx.y * stride;
  lambda += blockIdx.y * stride;
  const long f = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f < N) lambda[f] = -z[f];
}

__global__ void k_adj_add(long N, const double* z, double* lambda, const AdjCtl* ctl, long stride) {
  if (!ctl[blockIdx.y].live) return;
  z += blockIdx.y * stride;
  lambda += blockIdx.y * stride;
  const long f = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f < N) lambda[f] += z[f];
}

// sums[0] = lambda . rho, sums[1] = sum rho in the order of one block of 1024 threads (a chain
// per thread, trees over its lanes and warps), each of its warps on an SM of its own: one SM
// draws 4 MB at about 90 GB/s, 41 us at 512^2 where 32 take 8.
constexpr int RHO_BLOCKS = 32;
__global__ __launch_bounds__(32) void k_adj_rho_sums(long N, const double* lambda, AdjArgs args, AdjCtl* ctl,
                                                     double* partial, double* sums, long stride) {
  const double* rho = args.rho[blockIdx.y];
  lambda += blockIdx.y * stride;
  ctl += blockIdx.y;
  partial += blockIdx.y * stride;
  sums += blockIdx.y * stride;
  constexpr int B = 8, T = 32 * RHO_BLOCKS;
  double v[2] = {0.0, 0.0};
  for (long f0 = (long)blockIdx.x * 32 + threadIdx.x; f0 < N; f0 += (long)B * T) {
    double l[B], r[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
      const long f = f0 + (long)k * T;
      l[k] = f < N ? lambda[f] : 0.0;
      r[k] = f < N ? rho[f] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < B; ++k) {
      v[0] = fma(l[k], r[k], v[0]);
      v[1] += r[k];
    }
  }
  v[0] = warp_sum(v[0]);
  v[1] = warp_sum(v[1]);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = v[0];
    partial[RHO_BLOCKS + blockIdx.x] = v[1];
  }
  if (!last_block(&ctl->counter, RHO_BLOCKS)) return;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double t = warp_sum(__ldcg(&partial[k * RHO_BLOCKS + threadIdx.x]));
    if (threadIdx.x == 0) sums[k] = t;
  }
}

__global__ void k_adj_finish(long N, const double* lambda, const double* sums, AdjArgs args, long stride) {
  double* out = args.out[blockIdx.y];
  lambda += blockIdx.y * stride;
  sums += blockIdx.y * stride;
  const long f = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f < N) out[f] = (lambda[f] - sums[0] / sums[1]) / sums[1];
}

}  // namespace otm

using namespace otm;

namespace otm {
void dense_poisson(otm_context* ctx, Inst* d_inst, const int* gemm_inst, int G);

// Adjoint workspace of one grid size, number of maps and kind of transform, kept by the context:
// the layout of its device vectors and Krylov bases and its Poisson records, so a call
// allocates nothing and uploads nothing but its inputs' pointers. The vectors hold nothing from
// one call to the next: all workspaces lie in one allocation of the context, as large as the
// largest needs (a slice per map: 1.6 GB at 2048^2, so losses of 8 maps, then 7, 6, ... would
// keep 36 of them if each had its own).
struct AdjointWs : otm_context::Erased {
  int n = 0, m = 0, maps = 0;
  size_t N = 0, V = 0, ld = 0;
  long stride = 0;  // doubles from one map's slice to the next one's
  DevBuf recs;  // the Poisson records, then ctl and the work lists
  int* lists = nullptr;
  double *b, *lam, *z, *h, *t1, *t2, *Vb, *c, *part, *sums, *hcol, *inv;  // of map 0
  double2* g;                // the call's vertex displacements
  double *H, *cs, *sn, *gv;  // the cycle's Hessenberg state
  AdjCtl* ctl = nullptr;     // one per map
  int nb = 0;                // blocks of the step kernels per map
  int G = 0, rows = 0, cols = 0, reg = 0, fft = 0, col_warps = 0;  // transform items over all maps
  // the Arnoldi step as a graph with a WHILE node (built on first use) and its kernel count
  cudaGraphExec_t step_graph = nullptr;
  long step_kernels = 0;
  void drop_graph() override {
    if (step_graph) cudaGraphExecDestroy(step_graph);
    step_graph = nullptr;
  }
  ~AdjointWs() override { drop_graph(); }
  // Poisson records, one per map of each kind; destination z. Kind 0: source b; 1: source h;
  // 2: source the basis vector of the current step (set on the device, as is the active flag)
  Inst* rec(int kind) { return recs.as<Inst>() + kind * maps; }
};

static AdjointWs* adjoint_ws(otm_context* ctx, int n, int m, int maps) {
  const int fft = (ctx->poisson_mode != OTM_POISSON_DENSE && fft_eligible(n)) ? 1 : 0;
  const int key = (n * ADJ_MAPS + maps - 1) * 2 + fft;
  if (const auto it = ctx->adjoint.find(key); it != ctx->adjoint.end()) {
    auto* W = static_cast<AdjointWs*>(it->second.get());
    if (W->m >= m) return W;
    ctx->adjoint.erase(it);
  }
  auto own = std::make_unique<AdjointWs>();
  AdjointWs* W = own.get();
  W->n = n;
  W->m = m;
  W->maps = maps;
  W->N = (size_t)n * n;
  W->V = (size_t)(n + 1) * (n + 1);
  W->ld = (W->N + 31) / 32 * 32;
  W->nb = (int)std::min<size_t>(ANB, (W->N + AT - 1) / AT);
  auto up = [](size_t w) { return (w + 31) / 32 * 32; };  // every array starts on 256 bytes
  W->stride = (long)(W->ld * 6 + up(2 * W->V) + (size_t)(m + 1) * W->ld + 3 * up(m + 2) + up((size_t)ANB * (m + 2)) +
                     2 * up(8) + up((size_t)(m + 1) * m) + 2 * up(m));
  const size_t bytes = sizeof(double) * (size_t)W->stride * maps;
  if (bytes > ctx->adjoint_buf.bytes) {
    ctx->adjoint.clear();  // their pointers and graphs go with the allocation
    ctx->adjoint_buf.reserve(bytes);
  }
  double* q = ctx->adjoint_buf.as<double>();
  auto take = [&](size_t w) {
    double* r = q;
    q += up(w);
    return r;
  };
  W->b = take(W->ld);
  W->lam = take(W->ld);
  W->z = take(W->ld);
  W->t1 = take(W->ld);
  W->t2 = take(W->ld);
  W->h = take(W->ld);
  W->g = reinterpret_cast<double2*>(take(2 * W->V));
  W->Vb = take((size_t)(m + 1) * W->ld);
  W->c = take(m + 2);
  W->hcol = take(m + 2);
  W->gv = take(m + 2);
  W->part = take((size_t)ANB * (m + 2));
  W->inv = take(8);
  W->sums = take(8);
  W->H = take((size_t)(m + 1) * m);
  W->cs = take(m);
  W->sn = take(m);
  SizeTables* T = ctx->tables.at(n).get();
  Inst base;
  std::memset(&base, 0, sizeof(base));
  base.n = n;
  base.active = 1;
  base.C = T->C.as<double>();
  base.cosk = T->cosk.as<double>();
  base.tw = T->tw.as<double2>();
  base.pt = T->pt.as<double2>();
  base.fft = W->fft = fft;
  if (base.fft) {
    W->reg = dct_reg_supported(n) ? 1 : 0;
    const int per = W->reg ? dct_reg_lines_per_block(n) : fft_lines(n, false);
    W->col_warps = W->reg ? dct_reg_col_warps(n, maps, ctx->num_sms) : 0;
    const int cper = W->reg ? dct_reg_cols_per_block(n, W->col_warps) : fft_lines(n, true);
    base.nrow = (n + per - 1) / per;
    base.ncol = (n + cper - 1) / cper;
  } else {
    int t = (n + 63) / 64;
    base.ngemm = t * t;
  }
  W->rows = base.nrow * maps;
  W->cols = base.ncol * maps;
  W->G = base.ngemm * maps;
  std::vector<Inst> recs((size_t)3 * maps, base);
  for (int y = 0; y < maps; ++y) {
    const double* src[3] = {W->b, W->h, W->Vb};
    for (int kind = 0; kind < 3; ++kind) {
      Inst& r = recs[(size_t)kind * maps + y];
      r.r[0] = const_cast<double*>(src[kind]) + y * W->stride;
      r.dhat = W->z + y * W->stride;
      r.t1 = W->t1 + y * W->stride;
      r.t2 = W->t2 + y * W->stride;
      r.row0 = y * base.nrow;
      r.col0 = y * base.ncol;
      r.gemm0 = y * base.ngemm;
    }
  }
  // work list: item -> map, for the rows, the columns and the product tiles
  std::vector<int> items;
  for (int per : {base.nrow, base.ncol, base.ngemm})
    for (int y = 0; y < maps; ++y) items.insert(items.end(), per, y);
  static_assert(sizeof(Inst) % alignof(AdjCtl) == 0 && sizeof(AdjCtl) % alignof(int) == 0, "one buffer for the three");
  W->recs.reserve(sizeof(Inst) * recs.size() + sizeof(AdjCtl) * maps + sizeof(int) * items.size());
  W->ctl = reinterpret_cast<AdjCtl*>(W->recs.as<Inst>() + recs.size());
  W->lists = reinterpret_cast<int*>(W->ctl + maps);
  OTM_CUDA(cudaMemsetAsync(W->ctl, 0, sizeof(AdjCtl) * maps, ctx->stream));
  OTM_CUDA(cudaMemcpyAsync(W->recs.p, recs.data(), sizeof(Inst) * recs.size(), cudaMemcpyHostToDevice, ctx->stream));
  OTM_CUDA(cudaMemcpyAsync(W->lists, items.data(), sizeof(int) * items.size(), cudaMemcpyHostToDevice, ctx->stream));
  OTM_CUDA(cudaStreamSynchronize(ctx->stream));
  ctx->adjoint[key] = std::move(own);
  return W;
}

// z = M^+ (source of the records of a kind), every map whose record is active
static void poisson_rec(otm_context* ctx, AdjointWs* W, int kind) {
  Inst* d = W->rec(kind);
  const int *L = W->lists, *LC = L + W->rows, *LG = LC + W->cols;
  if (W->fft) {
    if (W->reg)
      dct_reg_run(ctx, W->n, false, d, L, 0, W->rows, LC, 0, W->cols, W->col_warps);
    else
      poisson_fft(ctx, W->n, d, L, 0, W->rows, LC, 0, W->cols);
  } else {
    dense_poisson(ctx, d, LG, W->G);
  }
}

// One Arnoldi step j of every map's cycle (j read on the device): z = M^+ v_j and the four
// step kernels, which do nothing for a map whose cycle has ended. They overlap their
// predecessor's end (common.cuh) except beside the product kernels, which do not wait for it:
// the gradient at 512^2 takes 1.17 ms so, 1.21 launched plainly.
static void arnoldi_step(otm_context* ctx, AdjointWs* W, int n, cudaGraphConditionalHandle handle, int in_graph) {
  const long ld = (long)W->ld, sd = W->stride;
  const dim3 grid(W->nb, W->maps);
  Inst* rec = W->rec(2);
  const Overlap overlap(ctx, W->fft, (long)W->N * W->maps);
  poisson_rec(ctx, W, 2);
  launch(ctx, "adj_apply", k_adj_apply, grid, AT, n, (const double2*)W->g, (const double*)W->z, W->Vb, ld, W->ctl,
         W->part, W->hcol, W->c, sd);
  launch(ctx, "adj_orth", k_adj_orth, grid, AT, n, W->Vb, ld, W->ctl, W->part, W->hcol, W->c, sd);
  launch(ctx, "adj_norm", k_adj_norm, grid, AT, n, W->Vb, ld, W->ctl, W->inv, W->part, (const double*)W->hcol,
         (const double*)W->c, W->H, W->cs, W->sn, W->gv, rec, sd);
  launch(ctx, "adj_scale", k_adj_scale_by, dim3((unsigned)((W->N + 255) / 256), W->maps), 256, (long)W->N, W->Vb, ld,
         (const double*)W->inv, (const AdjCtl*)W->ctl, sd, handle, in_graph);
}

// Steps per body of the cycles' WHILE node: a body costs 2.8 us beside its kernels (measured
// with empty ones), a step after the last cycle's end 7 launches that return at once (about 7 us).
constexpr int STEPS_PER_BODY = 4;

// The cycles' steps as a graph: a WHILE node whose body is STEPS_PER_BODY Arnoldi steps, its
// condition set by the last kernel of a step (at most m steps per launch).
static void build_step_graph(otm_context* ctx, AdjointWs* W, int n) {
  cudaStream_t st = ctx->stream;
  dct_reg_attrs(ctx->device);
  poisson_fft_attrs(ctx->device);
  cudaGraph_t g = nullptr;
  OTM_CUDA(cudaGraphCreate(&g, 0));
  try {
    cudaGraphConditionalHandle handle;
    OTM_CUDA(cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams params = {};
    params.type = cudaGraphNodeTypeConditional;
    params.conditional.handle = handle;
    params.conditional.type = cudaGraphCondTypeWhile;
    params.conditional.size = 1;
    cudaGraphNode_t node;
    OTM_CUDA(cudaGraphAddNode(&node, g, nullptr, 0, &params));
    cudaGraph_t body = params.conditional.phGraph_out[0];
    const long before = ctx->launches;
    OTM_CUDA(cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    try {
      for (int u = 0; u < STEPS_PER_BODY; ++u) arnoldi_step(ctx, W, n, handle, 1);
    } catch (...) {
      cudaGraph_t dummy;
      cudaStreamEndCapture(st, &dummy);
      throw;
    }
    OTM_CUDA(cudaStreamEndCapture(st, &body));
    W->step_kernels = ctx->launches - before;
    ctx->launches = before;  // captured, not executed
    OTM_CUDA(cudaGraphInstantiate(&W->step_graph, g, 0));
  } catch (...) {
    cudaGraphDestroy(g);
    throw;
  }
  cudaGraphDestroy(g);
}

// The adjoints of `count` (<= ADJ_MAPS) maps of size n side by side. One map's step is too
// small to fill the GPU and bound by latency; run from a host thread and stream of its own each,
// four took 83 us a step at 256^2 where one takes 51, and the time varied with the host. In
// common launches four take 80 us, falling as maps finish (63 us a step over a call whose
// longest map needs twice the steps of the others). Each map's arithmetic is that of a call
// of its own.
void adjoint_maps(otm_context* ctx, int n, int count, const double* const* density, const double* const* fwd_xy,
                  const double* const* grad_fwd, const otm_adjoint_options& o, double* const* grad_density,
                  otm_adjoint_stats* stats) {
  cudaStream_t st = ctx->stream;
  const int m = o.mode == OTM_ADJOINT_KRYLOV ? std::max(1, std::min(o.restart, ADJ_MAX_M)) : 1;
  AdjointWs* W = adjoint_ws(ctx, n, m, count);
  launch(ctx, "adj_reset", k_adj_reset_recs, 1, 32, W->rec(0), 3 * count);
  const size_t N = W->N, V = W->V;
  const long sd = W->stride;
  const unsigned RB = 256;
  const dim3 gN((unsigned)((N + RB - 1) / RB), count), gV((unsigned)((V + RB - 1) / RB), count), gT(W->nb, count);
  // inputs: used in place when they are device memory, else staged
  AdjArgs args = {};
  {
    size_t words = 0;
    for (int y = 0; y < count; ++y)
      words += (is_device_ptr(fwd_xy[y]) ? 0 : 2 * V) + (is_device_ptr(grad_fwd[y]) ? 0 : 2 * V) +
               (is_device_ptr(density[y]) ? 0 : N);
    if (words) ctx->staging.reserve(sizeof(double) * words);
    double* next = ctx->staging.as<double>();
    auto stage = [&](const double* src, size_t w) -> const double* {
      if (is_device_ptr(src)) return src;
      double* d = next;
      next += w;
      copy_in(ctx, d, src, sizeof(double) * w);
      return d;
    };
    for (int y = 0; y < count; ++y) {
      args.fwd[y] = stage(fwd_xy[y], 2 * V);
      args.q[y] = stage(grad_fwd[y], 2 * V);
      args.rho[y] = stage(density[y], N);
      args.out[y] = is_device_ptr(grad_density[y]) ? grad_density[y] : W->z + y * sd;
    }
  }
  // b = G^T q
  launch(ctx, "adj_cells", k_adj_cells, gN, RB, n, args, W->b, sd);
  std::vector<int> solves(count, 0);
  std::vector<double> rel(count, -1.0);
  if (o.mode == OTM_ADJOINT_ONE_STEP) {
    // lambda = -M^+ b: the solve writes z, lambda = -z
    poisson_rec(ctx, W, 0);
    std::fill(solves.begin(), solves.end(), 1);
    launch(ctx, "adj_scale", k_adj_neg, gN, RB, (long)N, (const double*)W->z, W->lam, sd);
  } else {
    for (int y = 0; y < count; ++y) OTM_CUDA(cudaMemsetAsync(W->lam + y * sd, 0, sizeof(double) * N, st));
    // Restarted GMRES(m) on J^T lambda = b, right-preconditioned: J^T M^+ y = b, lambda = M^+ y.
    // The cycles' Arnoldi steps run on the device (classical Gram-Schmidt applied twice,
    // Givens rotations and the loop test) as one graph launch with a WHILE node -- or, in
    // the host-driven loop mode and under the profiler, the same kernels one step at a
    // time; the host reads the cycles' step counts and the true residuals' norms once per
    // restart and decides which maps go on.
    launch(ctx, "adj_disp", k_adj_disp, gV, RB, n, args, W->g, sd);
    const bool graph = ctx->loop_mode == OTM_LOOP_GRAPH && !ctx->prof.on;
    AdjCtl hc[ADJ_MAPS];
    auto read = [&] {
      OTM_CUDA(cudaMemcpyAsync(hc, W->ctl, sizeof(AdjCtl) * count, cudaMemcpyDeviceToHost, st));
      OTM_CUDA(cudaStreamSynchronize(st));
    };
    auto residual = [&](const double* lambda) {
      launch(ctx, "adj_resid", k_adj_resid, gT, AT, n, (const double2*)W->g, lambda, (const double*)W->b, W->Vb, W->ctl,
             W->part, sd);
      read();
    };
    residual(nullptr);
    AdjCycle cyc = {};
    std::vector<char> done(count, 0);
    for (int y = 0; y < count; ++y) {
      cyc.bnorm[y] = hc[y].rnorm;
      if (!(cyc.bnorm[y] > 0)) {
        rel[y] = 0.0;
        done[y] = 1;
      }
    }
    while (true) {
      bool any = false;
      for (int y = 0; y < count; ++y) {
        if (!done[y]) {
          rel[y] = hc[y].rnorm / cyc.bnorm[y];
          if (!(rel[y] > o.tol) || solves[y] >= o.max_iter) done[y] = 1;
        }
        cyc.live[y] = !done[y];
        cyc.budget[y] = o.max_iter - solves[y];
        any |= !done[y];
      }
      if (!any) break;
      launch(ctx, "adj_cycle", k_adj_cycle_init, gN, RB, (long)N, W->ctl, W->gv, m, cyc, o.tol, W->rec(2), W->rec(1),
             W->Vb, sd);
      if (graph) {
        if (!W->step_graph) build_step_graph(ctx, W, n);
        OTM_CUDA(cudaGraphLaunch(W->step_graph, st));
      } else {
        bool go = true;
        while (go) {
          arnoldi_step(ctx, W, n, (cudaGraphConditionalHandle)0, 0);
          read();
          ctx->prof.flush();
          go = false;
          for (int y = 0; y < count; ++y) go |= hc[y].go != 0;
        }
      }
      // lambda += M^+ (V y), H y = g solved on the device
      launch(ctx, "adj_trisolve", k_adj_trisolve, dim3(1, count), 256, (const AdjCtl*)W->ctl, (const double*)W->H,
             (const double*)W->gv, W->c, sd);
      launch(ctx, "adj_span", k_adj_span, gN, RB, (long)N, W->h, (const double*)W->Vb, (long)W->ld,
             (const double*)W->c, (const AdjCtl*)W->ctl, sd);
      poisson_rec(ctx, W, 1);  // z = M^+ h
      launch(ctx, "adj_add", k_adj_add, gN, RB, (long)N, (const double*)W->z, W->lam, (const AdjCtl*)W->ctl, sd);
      residual(W->lam);
      int longest = 0;
      bool fault = false;
      for (int y = 0; y < count; ++y) {
        if (!cyc.live[y]) continue;
        longest = std::max(longest, hc[y].j);
        solves[y] += hc[y].j + 1;
        if (hc[y].j == 0) done[y] = 1;  // no step was possible: nothing changes by restarting
        fault |= hc[y].fault != 0;
      }
      if (graph) ctx->launches += W->step_kernels * (long)((longest + STEPS_PER_BODY - 1) / STEPS_PER_BODY);
      if (fault) break;  // reported below
    }
  }
  // chain through the density normalisation, reduced and applied on the device
  launch(ctx, "adj_rho_sums", k_adj_rho_sums, dim3(RHO_BLOCKS, count), 32, (long)N, (const double*)W->lam, args, W->ctl,
         W->part, W->sums, sd);
  launch(ctx, "adj_finish", k_adj_finish, gN, RB, (long)N, (const double*)W->lam, (const double*)W->sums, args, sd);
  OTM_CUDA(cudaGetLastError());
  for (int y = 0; y < count; ++y)
    if (args.out[y] != grad_density[y]) copy_out(ctx, grad_density[y], args.out[y], sizeof(double) * N);
  // a bounded wait inside a transform that gave up flags its record
  std::vector<Inst> recs_h((size_t)3 * count);
  OTM_CUDA(cudaMemcpyAsync(recs_h.data(), W->rec(0), sizeof(Inst) * recs_h.size(), cudaMemcpyDeviceToHost, st));
  OTM_CUDA(cudaStreamSynchronize(st));
  ctx->prof.flush();
  for (const Inst& r : recs_h)
    if (r.fault) throw DeviceTimeout{"otm_adjoint: a bounded device-side wait gave up"};
  if (stats)
    for (int y = 0; y < count; ++y) {
      stats[y].iterations = solves[y];
      stats[y].relative_residual = rel[y];
    }
}

void check_adjoint_options(const otm_adjoint_options& o) {
  if (o.mode != OTM_ADJOINT_ONE_STEP && o.mode != OTM_ADJOINT_KRYLOV) throw BadArg{"otm_adjoint: unknown mode"};
}

}  // namespace otm

extern "C" void otm_default_adjoint_options(otm_adjoint_options* o) {
  if (!o) return;
  o->mode = OTM_ADJOINT_KRYLOV;
  o->tol = 1e-10;
  o->max_iter = 2000;
  o->restart = 40;
}

extern "C" int otm_adjoint(otm_context* ctx, int n, const double* density, const double* fwd_xy,
                           const double* grad_fwd, const otm_adjoint_options* opt, double* grad_density,
                           otm_adjoint_stats* stats) {
  return guarded([&] {
    if (!ctx || !density || !fwd_xy || !grad_fwd || !grad_density) throw BadArg{"otm_adjoint: null argument"};
    if (n < 1 || n > 16384) throw BadArg{"otm_adjoint: grid size out of range"};
    otm_adjoint_options o;
    otm_default_adjoint_options(&o);
    if (opt) o = *opt;
    check_adjoint_options(o);
    make_current(ctx);
    if (otm_init(ctx, n) != OTM_OK) throw BadArg{std::string("otm_adjoint: ") + otm_last_error()};
    adjoint_maps(ctx, n, 1, &density, &fwd_xy, &grad_fwd, o, &grad_density, stats);
    return (int)OTM_OK;
  });
}
