// Fast cosine-transform Poisson solve, FP64, for the grid sizes that the register transforms
// (dct_reg.cu) do not cover: any n in 8 .. 4096.
//
// d_hat = M^+ r with M the reference's pseudo-Laplacian (otlib/otsolver_2dgrid.cpp:284-311):
// with C the orthonormal DCT-II, M^+ r = C^T ((C R C^T) / lambda) C where
// lambda_kl = 2 - 2 cos(pi k/n) cos(pi l/n) and the (0,0) mode is dropped (the
// mean-zero projection of :179). Three passes over the n x n array:
//   k_fft_rows_fwd   T[i][l] = DCT-II of r[i][.]                  (rows, contiguous)
//   k_fft_cols       for columns l: DCT-II along i, divide by lambda, DCT-III back along k
//                    (in place)
//   k_fft_rows_inv   d_hat[i][j] = DCT-III of T[i][.]
// Each length-n cosine transform is an n-point complex DFT with Makhoul's even/odd
// reordering and a quarter-wave twiddle; one DFT carries two real lines as its real and
// imaginary parts:
//   DCT-II : v_m = x_2m, v_{n-1-m} = x_{2m+1}; Z = DFT(v^a + i v^b);
//            A_k = (Z_k + conj Z_{n-k}) / 2, B_k = (Z_k - conj Z_{n-k}) / 2i;
//            X_k = s_k Re(e^{-i pi k/2n} A_k)
//   DCT-III: W_0 = Y_0, W_k = e^{i pi k/2n} (Y_k - i Y_{n-k}) / 2, Y = s X; v = IDFT(W) (no 1/n);
//            x_2m = Re v_m, x_{2m+1} = Re v_{n-1-m}
// with s_0 = sqrt(1/n), s_k = sqrt(2/n).
//
// The DFT. A power of two is transformed directly. Any other n uses Bluestein's chirp
// convolution ("A linear filtering approach to the computation of discrete Fourier
// transform", IEEE Trans. Audio Electroacoust. 18, 1970): with w_j = e^{-i pi j^2/n},
// X_k = w_k sum_j (x_j w_j) conj(w_{k-j}), a circular convolution of length M, the power of
// two >= 2n - 1, whose kernel's transform is a table. A line pair's M points are held in
// registers, 8 per thread on M/8 threads, as radix-8 passes (decimation in frequency; the
// last radix is 2, 4 or 8) that trade elements through shared memory; the inverse runs
// the passes backwards, so the digit-reversed order between the two is never undone.
// The passes' and the chirp's tables come from the host in extended precision, rounded once; the
// quarter-wave twiddles and the cosines (pt, cosk) are formed in double, as for the other sizes.
//
// What it replaces: n not a power of two took four dense products with the cosine basis
// (8 n^3 flops; 4 x 145 us at n = 500, 4 x 404 at 1000), 2048 and 4096 radix-4 passes over
// shared memory with one real line per transform (120 + 250 + 126 us at 2048). Here a solve
// takes 8 + 12 + 8 us at 500, 20 + 42 + 21 at 1000 and 38 + 82 + 36 at 2048 (event times less an
// empty kernel's). It is bound by the barriers between passes at 8 to 16 warps per SM
// (2048^2: 201 MB in and out, 31 us of copy time). Its error against extended precision is
// 3 to 20 times below the dense products' for n = 12 .. 401.

#include <algorithm>
#include <cmath>
#include <vector>

#include "cluster.cuh"

namespace otm {
namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 w) {
  return make_double2(fma(a.x, w.x, -a.y * w.y), fma(a.x, w.y, a.y * w.x));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 w) {  // a conj(w)
  return make_double2(fma(a.x, w.x, a.y * w.y), fma(a.y, w.x, -a.x * w.y));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
template <bool INV>
__device__ __forceinline__ double2 rot(double2 a) {  // times -i (forward), i (inverse)
  return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// DFTs in registers, natural order in and out; stride-S elements v[B], v[B + S], ...
template <bool INV>
__device__ __forceinline__ void dft4(double2& a, double2& b, double2& c, double2& d) {
  const double2 s0 = cadd(a, c), d0 = csub(a, c), s1 = cadd(b, d), d1 = rot<INV>(csub(b, d));
  a = cadd(s0, s1);
  c = csub(s0, s1);
  b = cadd(d0, d1);
  d = csub(d0, d1);
}
template <bool INV>
__device__ __forceinline__ void dft8(double2 (&v)[8]) {
  constexpr double h = 0.70710678118654752440;
  double2 e[4], o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    e[k] = cadd(v[k], v[k + 4]);
    o[k] = csub(v[k], v[k + 4]);
  }
  // o_k times W_8^k (its conjugate for the inverse)
  const double2 r1 = rot<INV>(o[1]), r3 = rot<INV>(o[3]);
  o[1] = make_double2(h * (o[1].x + r1.x), h * (o[1].y + r1.y));
  o[2] = rot<INV>(o[2]);
  o[3] = make_double2(h * (r3.x - o[3].x), h * (r3.y - o[3].y));
  dft4<INV>(e[0], e[1], e[2], e[3]);
  dft4<INV>(o[0], o[1], o[2], o[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] = e[k];
    v[2 * k + 1] = o[k];
  }
}

// Geometry of the M-point block transform: T threads per line pair, slots of 16 bytes with one
// of padding per 8 (radix-8 strides and the last pass's contiguous eights are then free of
// bank conflicts; the odd four keep two lines' slots apart). A block of the row passes holds
// one line pair from T = 128 on, a block of the column pass two up to T = 256, so that it
// reads whole 32-byte sectors: at n = 2048 the rows took 43 / 36 us with one pair per block against
// 48 / 49 with two, the columns 97 with one against 87 with two. M = 2048 is held to 128
// registers per thread, 16 warps per SM (n = 1000: rows 24.6 us against 28.7 with 178 registers
// and 8 warps); below, an instance has too few lines for a second block per SM, and the cap
// only spills (n = 500 columns: 16.8 us without, 18.6 with).
template <int M, bool COLS>
struct Geom {
  static constexpr int T = M / 8;
  static constexpr int LB = T < 16 ? 32 / T : T <= (COLS ? 256 : 64) ? 2 : 1;
  static constexpr int THREADS = LB * T;
  static constexpr int MIN_BLOCKS = T == 256 ? 512 / THREADS : 1;
  static constexpr int SLOTS = M + M / 8 + 4;
  static constexpr size_t SMEM = sizeof(double2) * LB * SLOTS;
};
template <int M>
struct Passes {
  // length of the last pass: 8, 4 or 2
  static constexpr int last() {
    int l = M;
    while (l > 8) l /= 8;
    return l;
  }
  // twiddles W_L^(t r), r = 1..7, t < L/8, of the passes L = M, M/8, ... > 8, [r-1][t]
  static constexpr int twiddles() {
    int c = 0;
    for (int l = M; l > 8; l /= 8) c += 7 * (l / 8);
    return c;
  }
};
__device__ __forceinline__ int slot(int p) { return p + (p >> 3); }

// The last pass: 8 / R DFTs of R contiguous elements.
template <int R, bool INV>
__device__ __forceinline__ void last_pass(double2 (&v)[8]) {
  if (R == 8) {
    dft8<INV>(v);
  } else if (R == 4) {
    dft4<INV>(v[0], v[1], v[2], v[3]);
    dft4<INV>(v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const double2 a = v[k], b = v[k + 1];
      v[k] = cadd(a, b);
      v[k + 1] = csub(a, b);
    }
  }
}

// Position of element q of thread t in the pass of length L.
template <int L>
__device__ __forceinline__ int place(int t, int q) {
  constexpr int S = L > 8 ? L / 8 : 1;
  return L > 8 ? (t / S) * L + t % S + q * S : 8 * t + q;
}
// Where a line's threads live and its tables lie.
struct BlockLine {  // in the block of one of the kernels below; tables in global memory
  static __device__ __forceinline__ void sync() { __syncthreads(); }
  static __device__ __forceinline__ double2 table(const double2* p) { return __ldg(p); }
  static __device__ __forceinline__ void computed() { overlap_begin(); }
};
struct WarpLine {  // in a warp of the one-cluster solve; tables in shared memory
  static __device__ __forceinline__ void sync() { __syncwarp(); }
  static __device__ __forceinline__ double2 table(const double2* p) { return *p; }
  static __device__ __forceinline__ void computed() {}
};

// Moves the elements from the places of pass A to those of pass B.
template <int A, int B, class Line>
__device__ __forceinline__ void exchange(double2 (&v)[8], int t, double2* sm) {
  Line::sync();
#pragma unroll
  for (int q = 0; q < 8; ++q) sm[slot(place<A>(t, q))] = v[q];
  Line::sync();
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = sm[slot(place<B>(t, q))];
}

// Forward transform: element q of thread t is x[t + q M/8] on entry and at position 8 t + q
// of the digit-reversed order on return.
template <int L, class Line>
__device__ __forceinline__ void fft_fwd(double2 (&v)[8], int t, double2* sm, const double2* __restrict__ tw) {
  if constexpr (L > 8) {
    constexpr int S = L / 8;
    double2 w[7];
#pragma unroll
    for (int r = 1; r < 8; ++r) w[r - 1] = Line::table(&tw[(r - 1) * S + t % S]);
    dft8<false>(v);
#pragma unroll
    for (int r = 1; r < 8; ++r) v[r] = cmul(v[r], w[r - 1]);
    exchange<L, S, Line>(v, t, sm);
    fft_fwd<S, Line>(v, t, sm, tw + 7 * S);
  } else {
    last_pass<L, false>(v);
  }
}
// Its inverse (unnormalised), from the digit-reversed order back to x[t + q M/8].
template <int L, class Line>
__device__ __forceinline__ void fft_inv(double2 (&v)[8], int t, double2* sm, const double2* __restrict__ tw) {
  if constexpr (L > 8) {
    constexpr int S = L / 8;
    fft_inv<S, Line>(v, t, sm, tw + 7 * S);
    double2 w[7];
#pragma unroll
    for (int r = 1; r < 8; ++r) w[r - 1] = Line::table(&tw[(r - 1) * S + t % S]);
    exchange<S, L, Line>(v, t, sm);
#pragma unroll
    for (int r = 1; r < 8; ++r) v[r] = cmulc(v[r], w[r - 1]);
    dft8<true>(v);
  } else {
    last_pass<L, true>(v);
  }
}
// Frequency at position p of the digit-reversed order.
template <int L>
__host__ __device__ __forceinline__ constexpr int frequency(int p) {
  if constexpr (L > 8)
    return p / (L / 8) + 8 * frequency<L / 8>(p % (L / 8));
  else
    return p;
}

// Tables of a size (Inst::tw): the passes' twiddles, then for Bluestein the kernel's
// transform over M in the order [q][t] of the threads' elements and the chirp w_j, j < n.
template <int M>
struct Tables {
  const double2 *tw, *kernel, *chirp;
  __device__ __forceinline__ explicit Tables(const double2* base)
      : tw(base), kernel(base + Passes<M>::twiddles()), chirp(base + Passes<M>::twiddles() + M) {}
};

// n-point DFT of the line pair: v[q] = x[t + q T] (zero from n on) on entry; Z_k, k < n, in
// sm[slot(k)] on return (after the closing barrier).
template <int M, bool CHIRP, class Line>
__device__ __forceinline__ void line_dft(double2 (&v)[8], int n, int t, double2* sm, const Tables<M>& tab) {
  constexpr int T = M / 8;
  if (CHIRP) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int m = t + q * T;
      v[q] = m < n ? cmul(v[q], Line::table(&tab.chirp[m])) : make_double2(0.0, 0.0);
    }
    fft_fwd<M, Line>(v, t, sm, tab.tw);
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = cmul(v[q], Line::table(&tab.kernel[q * T + t]));
    fft_inv<M, Line>(v, t, sm, tab.tw);
    Line::sync();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = t + q * T;
      if (k < n) sm[slot(k)] = cmul(v[q], Line::table(&tab.chirp[k]));
    }
  } else {
    fft_fwd<M, Line>(v, t, sm, tab.tw);
    Line::sync();
#pragma unroll
    for (int q = 0; q < 8; ++q) sm[slot(frequency<M>(8 * t + q))] = v[q];
  }
  Line::sync();
}

// Source of sample m of the reordered sequence.
__device__ __forceinline__ int makhoul(int m, int n) { return m < (n + 1) / 2 ? 2 * m : 2 * (n - 1 - m) + 1; }

// X_k of both lines from Z_k and Z_{n-k}
__device__ __forceinline__ double2 dct2_post(double2 Z, double2 P, double2 pt, double sk) {
  const double ax = 0.5 * (Z.x + P.x), ay = 0.5 * (Z.y - P.y), bx = 0.5 * (Z.y + P.y), by = 0.5 * (P.x - Z.x);
  return make_double2(sk * fma(ax, pt.x, ay * pt.y), sk * fma(bx, pt.x, by * pt.y));
}
// conj(W^a_k + i W^b_k) from Y_k and Y_{n-k} of both lines: the inverse DFT is the conjugate
// of the DFT of the conjugate
__device__ __forceinline__ double2 dct3_pre(int k, double2 y, double2 ym, double2 pt) {
  if (k == 0) return make_double2(y.x, -y.y);
  const double ax = 0.5 * fma(y.x, pt.x, ym.x * pt.y), ay = 0.5 * fma(y.x, pt.y, -ym.x * pt.x);
  const double bx = 0.5 * fma(y.y, pt.x, ym.y * pt.y), by = 0.5 * fma(y.y, pt.y, -ym.y * pt.x);
  return make_double2(ax - by, -(ay + bx));
}

// ---- the passes for one line pair ----

// Rows i and i + 1 of src (n x n) -> their coefficients in T.
template <int M, bool CHIRP, class Line>
__device__ __forceinline__ void row_pair_fwd(const double* src, double* T, int n, int i, int t, double2* sm,
                                             const Tables<M>& tab, const double2* pt) {
  constexpr int LT = M / 8;
  const bool a = i < n, b = i + 1 < n;
  double2 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int m = t + q * LT;
    v[q] = make_double2(0.0, 0.0);
    if (m < n) {
      const double* p = src + (size_t)i * n + makhoul(m, n);
      if (a) v[q].x = p[0];
      if (b) v[q].y = p[n];
    }
  }
  line_dft<M, CHIRP, Line>(v, n, t, sm, tab);
  Line::computed();
  const double s0 = sqrt(1.0 / n), s1 = sqrt(2.0 / n);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = t + q * LT;
    if (k >= n) continue;
    const double2 X = dct2_post(sm[slot(k)], sm[slot(k ? n - k : 0)], Line::table(&pt[k]), k ? s1 : s0);
    if (a) T[(size_t)i * n + k] = X.x;
    if (b) T[(size_t)(i + 1) * n + k] = X.y;
  }
}

// Columns l and l + 1 of T, in place: coefficients, division by lambda, and back.
template <int M, bool CHIRP, class Line>
__device__ __forceinline__ void column_pair(double* T, int n, int l, int t, double2* sm, const Tables<M>& tab,
                                            const double2* pt, const double* cosk) {
  constexpr int LT = M / 8;
  const bool a = l < n, b = l + 1 < n;
  double2 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int m = t + q * LT;
    v[q] = make_double2(0.0, 0.0);
    if (m < n) {
      const double* p = T + (size_t)makhoul(m, n) * n + l;
      if (a) v[q].x = p[0];
      if (b) v[q].y = p[1];
    }
  }
  line_dft<M, CHIRP, Line>(v, n, t, sm, tab);
  // the coefficients over lambda, times s_k for the way back
  const double s0 = sqrt(1.0 / n), s1 = sqrt(2.0 / n);
  const double ca = a ? cosk[l] : 0.0, cb = b ? cosk[l + 1] : 0.0;
  double2 u[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = t + q * LT;
    u[q] = make_double2(0.0, 0.0);
    if (k >= n) continue;
    const double sk = k ? s1 : s0, ck = cosk[k];
    const double2 X = dct2_post(sm[slot(k)], sm[slot(k ? n - k : 0)], Line::table(&pt[k]), sk);
    const double la = 2.0 - 2.0 * ck * ca, lb = 2.0 - 2.0 * ck * cb;
    u[q] = make_double2(k == 0 && l == 0 ? 0.0 : sk * (X.x / la), sk * (X.y / lb));
  }
  Line::sync();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = t + q * LT;
    if (k < n) sm[slot(k)] = u[q];
  }
  Line::sync();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = t + q * LT;
    v[q] = make_double2(0.0, 0.0);
    if (k < n) v[q] = dct3_pre(k, u[q], sm[slot(k ? n - k : 0)], Line::table(&pt[k]));
  }
  line_dft<M, CHIRP, Line>(v, n, t, sm, tab);
  Line::computed();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int m = t + q * LT;
    if (m >= n) continue;
    const double2 z = sm[slot(m)];
    double* p = T + (size_t)makhoul(m, n) * n + l;
    if (a) p[0] = z.x;
    if (b) p[1] = -z.y;
  }
}

// Rows i and i + 1 of T -> their samples in out.
template <int M, bool CHIRP, class Line>
__device__ __forceinline__ void row_pair_inv(const double* T, double* out, int n, int i, int t, double2* sm,
                                             const Tables<M>& tab, const double2* pt) {
  constexpr int LT = M / 8;
  const bool a = i < n, b = i + 1 < n;
  const double s0 = sqrt(1.0 / n), s1 = sqrt(2.0 / n);
  double2 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = t + q * LT;
    v[q] = make_double2(0.0, 0.0);
    if (k >= n) continue;
    const double* p = T + (size_t)i * n;
    const double sk = k ? s1 : s0;
    double2 y = make_double2(0.0, 0.0), ym = y;
    if (a) {
      y.x = sk * p[k];
      if (k) ym.x = s1 * p[n - k];
    }
    if (b) {
      y.y = sk * p[n + k];
      if (k) ym.y = s1 * p[n + n - k];
    }
    v[q] = dct3_pre(k, y, ym, Line::table(&pt[k]));
  }
  line_dft<M, CHIRP, Line>(v, n, t, sm, tab);
  Line::computed();
  // sample j of a row is element j/2 or n-1-j/2 of the reordered sequence
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int j = t + q * LT;
    if (j >= n) continue;
    const double2 z = sm[slot((j & 1) ? n - 1 - (j >> 1) : (j >> 1))];
    if (a) out[(size_t)i * n + j] = z.x;
    if (b) out[(size_t)(i + 1) * n + j] = -z.y;
  }
}

template <int M, bool CHIRP>
__global__ __launch_bounds__(Geom<M, false>::THREADS, Geom<M, false>::MIN_BLOCKS) void k_fft_rows_fwd(const Inst* insts, const int* row_inst, int seg) {
  using G = Geom<M, false>;
  constexpr int T = G::T;
  extern __shared__ double2 smem[];
  const int item = seg + blockIdx.x;
  overlap_wait();
  const Inst& I = insts[row_inst[item]];
  if (!I.active) return;
  const int n = I.n, line = threadIdx.x / T, t = threadIdx.x % T;
  const int i = 2 * ((item - I.row0) * G::LB + line);  // rows i and i + 1
  double2* sm = smem + line * G::SLOTS;
  row_pair_fwd<M, CHIRP, BlockLine>(I.r[I.it % 3], I.t1, n, i, t, sm, Tables<M>(I.tw), I.pt);
}

// In place on t1, two adjacent columns per line; consecutive threads take the block's lines
// in turn, so that they read consecutive columns.
template <int M, bool CHIRP>
__global__ __launch_bounds__(Geom<M, true>::THREADS, Geom<M, true>::MIN_BLOCKS) void k_fft_cols(const Inst* insts, const int* col_inst, int seg) {
  using G = Geom<M, true>;
  constexpr int T = G::T, LB = G::LB;
  extern __shared__ double2 smem[];
  const int item = seg + blockIdx.x;
  overlap_wait();
  const Inst& I = insts[col_inst[item]];
  if (!I.active) return;
  const int n = I.n, line = threadIdx.x % LB, t = threadIdx.x / LB;
  const int l = 2 * ((item - I.col0) * LB + line);  // columns l and l + 1
  double2* sm = smem + line * G::SLOTS;
  column_pair<M, CHIRP, BlockLine>(I.t1, n, l, t, sm, Tables<M>(I.tw), I.pt, I.cosk);
}

template <int M, bool CHIRP>
__global__ __launch_bounds__(Geom<M, false>::THREADS, Geom<M, false>::MIN_BLOCKS) void k_fft_rows_inv(const Inst* insts, const int* row_inst, int seg) {
  using G = Geom<M, false>;
  constexpr int T = G::T;
  extern __shared__ double2 smem[];
  const int item = seg + blockIdx.x;
  overlap_wait();
  const Inst& I = insts[row_inst[item]];
  if (!I.active) return;
  const int n = I.n, line = threadIdx.x / T, t = threadIdx.x % T;
  const int i = 2 * ((item - I.row0) * G::LB + line);
  double2* sm = smem + line * G::SLOTS;
  row_pair_inv<M, CHIRP, BlockLine>(I.t1, I.dhat, n, i, t, sm, Tables<M>(I.tw), I.pt);
}

// ---- the passes for the one-cluster solve (cluster.cuh): lines of at most a warp ----

template <int M, bool CHIRP>
struct ClusterFft {
  static constexpr int T = M / 8, LPW = 32 / T, SLOTS = Geom<M, false>::SLOTS, MAX_N = M;
  static_assert(T <= 32 && LPW * SLOTS * sizeof(double2) <= CL_WARP_BYTES, "a warp's lines fit in its region");
  static __host__ __device__ int entries(int n) { return Passes<M>::twiddles() + (CHIRP ? M + n : 0); }
  static int table_bytes(int n) { return (int)(sizeof(double2) * (entries(n) + n) + (sizeof(double) * n + 15) / 16 * 16); }
  const int n, sub = (threadIdx.x & 31) / T, t = (threadIdx.x & 31) % T, items;
  double2 *tab, *pt;
  double* cosk;
  __device__ __forceinline__ ClusterFft(const Inst& I, unsigned char* smem)
      : n(I.n), items(((I.n + 1) / 2 + LPW - 1) / LPW), tab(reinterpret_cast<double2*>(smem)) {
    pt = tab + entries(n);
    cosk = reinterpret_cast<double*>(pt + n);
    for (int e = threadIdx.x; e < entries(n); e += CL_T) tab[e] = I.tw[e];
    for (int e = threadIdx.x; e < n; e += CL_T) {
      pt[e] = I.pt[e];
      cosk[e] = I.cosk[e];
    }
  }
  __device__ __forceinline__ double2* line(const ClusterBlock& B) const {
    return reinterpret_cast<double2*>(B.region()) + sub * SLOTS;
  }
  __device__ __forceinline__ void rows_fwd(const ClusterBlock& B, int it) const {
    B.items(items, [&](int item) {
      row_pair_fwd<M, CHIRP, WarpLine>(B.I.r[it % 3], B.I.t1, n, 2 * (item * LPW + sub), t, line(B), Tables<M>(tab), pt);
    });
  }
  __device__ __forceinline__ void cols(const ClusterBlock& B) const {
    B.items(items, [&](int item) {
      column_pair<M, CHIRP, WarpLine>(B.I.t1, n, 2 * (item * LPW + sub), t, line(B), Tables<M>(tab), pt, cosk);
    });
  }
  __device__ __forceinline__ void rows_inv(const ClusterBlock& B) const {
    B.items(items, [&](int item) {
      row_pair_inv<M, CHIRP, WarpLine>(B.I.t1, B.I.dhat, n, 2 * (item * LPW + sub), t, line(B), Tables<M>(tab), pt);
    });
  }
};

// ---- host ----

bool pow2(int n) { return (n & (n - 1)) == 0; }

// Transform length of size n: n itself for a power of two, else Bluestein's M >= 2n - 1.
int length_of(int n) {
  if (pow2(n)) return n;
  int m = 32;
  while (m < 2 * n - 1) m *= 2;
  return m;
}

// f(M, CHIRP) with the size's length and kind as compile-time constants
template <class F>
void dispatch(int n, F&& f) {
  const int M = length_of(n);
#define OTM_FFT_CASE(LEN, CH) \
  case LEN: return f(std::integral_constant<int, LEN>(), std::integral_constant<bool, CH>())
  if (pow2(n)) {
    switch (M) {
      OTM_FFT_CASE(8, false);
      OTM_FFT_CASE(16, false);
      OTM_FFT_CASE(32, false);
      OTM_FFT_CASE(2048, false);
      OTM_FFT_CASE(4096, false);
    }
  } else {
    switch (M) {
      OTM_FFT_CASE(32, true);
      OTM_FFT_CASE(64, true);
      OTM_FFT_CASE(128, true);
      OTM_FFT_CASE(256, true);
      OTM_FFT_CASE(512, true);
      OTM_FFT_CASE(1024, true);
      OTM_FFT_CASE(2048, true);
      OTM_FFT_CASE(4096, true);
      OTM_FFT_CASE(8192, true);
    }
  }
#undef OTM_FFT_CASE
  throw BadArg{"poisson_fft: unsupported size"};
}

using ld = long double;
struct Cld {
  ld x, y;
};
const ld kPi = 3.14159265358979323846264338327950288L;
Cld unit(long num, long den) {  // exp(-2 pi i num / den)
  num %= den;
  const ld a = 2.0L * kPi * (ld)num / (ld)den;
  return {std::cos(a), -std::sin(a)};
}

// In-place radix-2 DFT of a power-of-two number of points, extended precision.
void dft_host(std::vector<Cld>& x) {
  const size_t M = x.size();
  for (size_t i = 1, j = 0; i < M; ++i) {
    size_t bit = M >> 1;
    for (; j & bit; bit >>= 1) j ^= bit;
    j ^= bit;
    if (i < j) std::swap(x[i], x[j]);
  }
  std::vector<Cld> w(M / 2);
  for (size_t k = 0; k < M / 2; ++k) w[k] = unit((long)k, (long)M);
  for (size_t len = 2; len <= M; len *= 2)
    for (size_t s = 0; s < M; s += len)
      for (size_t k = 0; k < len / 2; ++k) {
        const Cld c = w[k * (M / len)], b = x[s + k + len / 2];
        const Cld t = {b.x * c.x - b.y * c.y, b.x * c.y + b.y * c.x}, a = x[s + k];
        x[s + k] = {a.x + t.x, a.y + t.y};
        x[s + k + len / 2] = {a.x - t.x, a.y - t.y};
      }
}

}  // namespace

int fft_family(int n) { return 2 * length_of(n) + (pow2(n) ? 0 : 1); }

int fft_lines(int n, bool cols) {
  int lines = 0;
  dispatch(n, [&](auto Mc, auto) {
    constexpr int M = decltype(Mc)::value;
    lines = 2 * (cols ? Geom<M, true>::LB : Geom<M, false>::LB);
  });
  return lines;
}

void fft_tables(int n, std::vector<double2>& out) {
  out.clear();
  dispatch(n, [&](auto Mc, auto chirp) {
    constexpr int M = decltype(Mc)::value;
    auto put = [&](Cld c) { out.push_back(make_double2((double)c.x, (double)c.y)); };
    for (int L = M; L > 8; L /= 8)
      for (int r = 1; r < 8; ++r)
        for (int t = 0; t < L / 8; ++t) put(unit((long)r * t, L));
    if (!decltype(chirp)::value) return;
    std::vector<Cld> w(n), k(M, {0.0L, 0.0L});
    for (int j = 0; j < n; ++j) w[j] = unit((long)j * j % (2 * n), 2 * n);
    for (int j = 0; j < n; ++j) k[j] = k[(M - j) % M] = {w[j].x, -w[j].y};
    dft_host(k);
    for (int q = 0; q < 8; ++q)
      for (int t = 0; t < M / 8; ++t) {
        const Cld c = k[frequency<M>(8 * t + q)];
        put({c.x / M, c.y / M});
      }
    for (int j = 0; j < n; ++j) put(w[j]);
  });
}

void poisson_fft_attrs(int device) {
  static bool attr[64] = {};  // per device ordinal
  if (device < 64 && attr[device]) return;
  for (int n : {8, 16, 32, 2048, 4096, 9, 17, 33, 65, 129, 257, 513, 1025, 2049})
    dispatch(n, [&](auto Mc, auto ch) {
      constexpr int M = decltype(Mc)::value;
      constexpr bool C = decltype(ch)::value;
      constexpr auto key = cudaFuncAttributeMaxDynamicSharedMemorySize;
      OTM_CUDA(cudaFuncSetAttribute(k_fft_rows_fwd<M, C>, key, (int)Geom<M, false>::SMEM));
      OTM_CUDA(cudaFuncSetAttribute(k_fft_cols<M, C>, key, (int)Geom<M, true>::SMEM));
      OTM_CUDA(cudaFuncSetAttribute(k_fft_rows_inv<M, C>, key, (int)Geom<M, false>::SMEM));
    });
  if (device < 64) attr[device] = true;
}

void poisson_fft(otm_context* ctx, int n, Inst* d_insts, const int* row_inst, int roff, int nrow_items,
                 const int* col_inst, int coff, int ncol_items) {
  poisson_fft_attrs(ctx->device);
  if (nrow_items <= 0) return;
  dispatch(n, [&](auto Mc, auto ch) {
    constexpr int M = decltype(Mc)::value;
    constexpr bool C = decltype(ch)::value;
    using GR = Geom<M, false>;
    using GC = Geom<M, true>;
    launch_smem(ctx, "fft_rows_fwd", k_fft_rows_fwd<M, C>, nrow_items, GR::THREADS, GR::SMEM, (const Inst*)d_insts,
                row_inst, roff);
    launch_smem(ctx, "fft_cols", k_fft_cols<M, C>, ncol_items, GC::THREADS, GC::SMEM, (const Inst*)d_insts, col_inst,
                coff);
    launch_smem(ctx, "fft_rows_inv", k_fft_rows_inv<M, C>, nrow_items, GR::THREADS, GR::SMEM, (const Inst*)d_insts,
                row_inst, roff);
  });
}

// Largest size solved by a cluster: above it a line takes more threads than a warp has (at 127^2
// the cluster is 1.15 times as fast as the kernels: cluster.cuh).
constexpr int CLUSTER_MAX = 128;

int poisson_cluster_blocks(otm_context* ctx, int n, int count) {
  int blocks = 0;
  if (n <= CLUSTER_MAX)
    dispatch(n, [&](auto Mc, auto ch) {
      constexpr int M = decltype(Mc)::value;
      if constexpr (M <= 256) blocks = cluster_blocks<ClusterFft<M, decltype(ch)::value>>(ctx, n, count);
    });
  return blocks;
}

void poisson_cluster(otm_context* ctx, int n, int count, int blocks, Inst* d_insts, double* partials) {
  dispatch(n, [&](auto Mc, auto ch) {
    constexpr int M = decltype(Mc)::value;
    if constexpr (M <= 256)
      cluster_launch<ClusterFft<M, decltype(ch)::value>>(ctx, n, count, blocks, d_insts, partials);
  });
}

}  // namespace otm
