// Point location in the forward mesh (TransportMap inversion) and rasterization of
// the deformed grid mesh or of any triangle/quad mesh, for sm_100a.
//
// Inversion runs on a uniform bin grid built on the GPU: faces are binned by their
// bounding boxes (count, exclusive scan, scatter) and each query point tests only the
// faces of its bin. Rasterization is face-parallel: each face tests the pixel centres
// of its box and keeps the highest accepting face index per pixel with an integer
// atomicMax; a per-pixel pass then writes the values. This file is compiled without FMA contraction: the geometric
// predicates (utils/mesh_utils.cpp:18-88) then round exactly as the reference's
// scalar x86-64 build does, and the reference's BVH face order and leaf boxes are
// rebuilt on the GPU (build_bvh_order), which makes the located faces, hit counts,
// weights, inverse positions and pixel values bit-identical to the reference.

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "context.h"
#include "place_list.cuh"

namespace otm {

// ---- geometry (utils/eigen_addons.h:15-22, utils/mesh_utils.h:18-25, mesh_utils.cpp:18-88) ----

__device__ __forceinline__ double cross2(double ax, double ay, double bx, double by) { return ax * by - ay * bx; }

__device__ __forceinline__ double signed_area3(double ax, double ay, double bx, double by, double cx, double cy) {
  return 0.5 * cross2(bx - ax, by - ay, cx - ax, cy - ay);
}

struct Quad {
  double x[4], y[4];
};

__device__ __forceinline__ bool inside_tri(double qx, double qy, double p0x, double p0y, double p1x, double p1y,
                                           double p2x, double p2y) {
  double q2x = qx - p2x, q2y = qy - p2y;
  double eux = p1x - p2x, euy = p1y - p2y;
  double evx = p0x - p2x, evy = p0y - p2y;
  double area2 = cross2(evx, evy, eux, euy);
  double u = cross2(q2x, q2y, eux, euy) / area2;
  double v = cross2(evx, evy, q2x, q2y) / area2;
  const double eps = 1e-8;
  return u >= -eps && v >= -eps && u + v <= 1. + eps;
}

// inside_quad (mesh_utils.cpp:62-74)
__device__ __forceinline__ bool inside_quad(double qx, double qy, const Quad& p) {
  return inside_tri(qx, qy, p.x[0], p.y[0], p.x[1], p.y[1], p.x[2], p.y[2]) ||
         inside_tri(qx, qy, p.x[0], p.y[0], p.x[2], p.y[2], p.x[3], p.y[3]);
}

// bilinear_coordinates_in_quad, weights form (mesh_utils.cpp:18-59, 76-88), in two parts: the
// terms of the two solution pairs (u, v) = (2 A3 / E3, 2 A0 / E0) and their conjugates
// (false: no real solution), and the weights from them.
struct Bilinear {
  double A0, A3, E0, E3, E0p, E3p;
};
constexpr double kBilinearZero = 4 * DBL_MIN;

__device__ __forceinline__ bool bilinear_terms(double qx, double qy, const Quad& p, Bilinear& t) {
  double A0 = signed_area3(qx, qy, p.x[0], p.y[0], p.x[1], p.y[1]);
  double A1 = signed_area3(qx, qy, p.x[1], p.y[1], p.x[2], p.y[2]);
  double A2 = signed_area3(qx, qy, p.x[2], p.y[2], p.x[3], p.y[3]);
  double A3 = signed_area3(qx, qy, p.x[3], p.y[3], p.x[0], p.y[0]);
  double B0 = signed_area3(qx, qy, p.x[3], p.y[3], p.x[1], p.y[1]);
  double B1 = signed_area3(qx, qy, p.x[0], p.y[0], p.x[2], p.y[2]);
  double B3 = signed_area3(qx, qy, p.x[2], p.y[2], p.x[0], p.y[0]);
  double D = B0 * B0 + B1 * B1 + 2 * A0 * A2 + 2 * A1 * A3;
  if (D < 0) return false;
  double sD = sqrt(D);
  t.A0 = A0;
  t.A3 = A3;
  t.E0 = 2 * A0 - B0 - B1 + sD;
  t.E3 = 2 * A3 - B3 - B0 + sD;
  t.E0p = 2 * A0 - B0 - B1 - sD;
  t.E3p = 2 * A3 - B3 - B0 - sD;
  return true;
}

// What weights_inside will say of a point, where it is certain without the four divisions and
// the snapping of bilinear_from_terms (half of a pixel test's instructions): 1 accepted, -1
// rejected, 0 to be computed. The snapping tolerance is 1.5e-8 and a division rounds by 1e-16,
// so a ratio beyond [0, 1] by 1e-7 stays outside and one 1e-7 within stays inside. A pair with u
// or v outside leaves one of the four weights negative by at least 1e-8, or NaN; the second
// pair only counts when the first is outside. NaN in any term compares false: computed.
struct Verdict {
  bool in, out;
};
__device__ __forceinline__ Verdict ratio_verdict(double num, double den) {
  const double a = fabs(num), b = fabs(den), low = b * 1e-7;
  const bool same = (__double2hiint(num) ^ __double2hiint(den)) >= 0;
  const bool above = a > low;
  return {bool(same & above & (a < b * (1. - 1e-7))), bool((a > b * (1. + 1e-7)) | (!same & above))};
}
__device__ __forceinline__ int bilinear_verdict(const Bilinear& t) {
  // |A| within `zero` makes the ratio an exact 0: on the border, computed
  const bool v0 = fabs(t.A0) > kBilinearZero, u0 = fabs(t.A3) > kBilinearZero;
  const double nv = 2 * t.A0, nu = 2 * t.A3;
  const Verdict v = ratio_verdict(nv, t.E0), u = ratio_verdict(nu, t.E3);
  if (v0 & u0 & v.in & u.in) return 1;
  const Verdict va = ratio_verdict(nv, t.E0p), ua = ratio_verdict(nu, t.E3p);
  return ((v0 & v.out) | (u0 & u.out)) & ((v0 & va.out) | (u0 & ua.out)) ? -1 : 0;
}

__device__ __forceinline__ void bilinear_from_terms(const Bilinear& t, double w[4]) {
  const double A0 = t.A0, A3 = t.A3;
  const double zero = kBilinearZero;
  double v = fabs(A0) <= zero ? 0 : 2 * A0 / t.E0;
  double u = fabs(A3) <= zero ? 0 : 2 * A3 / t.E3;
  double v_alt = fabs(A0) <= zero ? 0 : 2 * A0 / t.E0p;
  double u_alt = fabs(A3) <= zero ? 0 : 2 * A3 / t.E3p;
  const double eps = 1.4901161193847656e-08;  // sqrt(DBL_EPSILON), exact
  if (fabs(u) < eps) u = 0;
  if (fabs(v) < eps) v = 0;
  if (fabs(u - 1.) < eps) u = 1;
  if (fabs(v - 1.) < eps) v = 1;
  if (fabs(u_alt) < eps) u_alt = 0;
  if (fabs(v_alt) < eps) v_alt = 0;
  if (fabs(u_alt - 1.) < eps) u_alt = 1;
  if (fabs(v_alt - 1.) < eps) v_alt = 1;
  if ((u < 0 || v < 0 || u > 1 || v > 1) && (u_alt >= 0 && v_alt >= 0 && u_alt <= 1 && v_alt <= 1)) {
    u = u_alt;
    v = v_alt;
  }
  const double weps = 4 * DBL_EPSILON;
  w[0] = (1. - u) * (1 - v);
  w[1] = (u) * (1. - v);
  w[2] = (u) * (v);
  w[3] = (1. - u) * (v);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (fabs(w[k]) <= weps)
      w[k] = 0;
    else if (fabs(w[k] - 1.) <= weps)
      w[k] = 1;
  }
}

__device__ bool bilinear_weights(double qx, double qy, const Quad& p, double w[4]) {
  Bilinear t;
  if (!bilinear_terms(qx, qy, p, t)) return false;
  bilinear_from_terms(t, w);
  return true;
}

__device__ __forceinline__ bool weights_inside(const double w[4]) {
  return w[0] <= 1.0f && w[1] <= 1.0f && w[2] <= 1.0f && w[3] <= 1.0f && w[0] >= 0.0f && w[1] >= 0.0f &&
         w[2] >= 0.0f && w[3] >= 0.0f;
}

// Corners of face f = j + i*n of an (n+1)^2 grid mesh: (i,j), (i+1,j), (i+1,j+1), (i,j+1).
__device__ __forceinline__ void load_quad(const double* xy, int n, int f, Quad& p, int vid[4]) {
  int i = f / n, j = f - (f / n) * n;
  vid[0] = j + i * (n + 1);
  vid[1] = j + (i + 1) * (n + 1);
  vid[2] = (j + 1) + (i + 1) * (n + 1);
  vid[3] = (j + 1) + i * (n + 1);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    p.x[k] = xy[2 * (size_t)vid[k]];
    p.y[k] = xy[2 * (size_t)vid[k] + 1];
  }
}

// ---- exclusive scan of int counts ----
//
// Chunks of SCAN_B values: a block scans one (four values per thread, warp shuffles), one
// block scans the chunks' sums, and a value's prefix is its chunk-local one plus its chunk's.

constexpr int SCAN_B = 1024, SCAN_T = SCAN_B / 4;

// Exclusive prefix of v over the block (a multiple of 32 threads, at most 1024); *total its sum.
// warp_total: 32 ints of shared memory, free for reuse after the next barrier.
__device__ __forceinline__ int block_prefix(int v, int* warp_total, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += u;
  }
  if (lane == 31) warp_total[warp] = s;
  __syncthreads();
  int w = lane < nw ? warp_total[lane] : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) w += u;
  }
  *total = __shfl_sync(0xffffffffu, w, 31);
  const int before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
  return (warp ? before : 0) + s - v;
}

// Chunk-local prefixes of a chunk's values v[k] = value(4 t + k of the chunk).
template <class F>
__device__ __forceinline__ void scan_chunk(F value, int* out, int* sums, int count) {
  __shared__ int warp_total[32];
  const int g = blockIdx.x * SCAN_B + threadIdx.x * 4;
  int v[4], t = 0, total;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = g + k < count ? value(g + k) : 0;
    t += v[k];
  }
  int p = block_prefix(t, warp_total, &total);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (g + k < count) out[g + k] = p;
    p += v[k];
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ __launch_bounds__(SCAN_T) void k_scan_local(const int* in, int* out, int* sums, int count) {
  scan_chunk([&](int i) { return in[i]; }, out, sums, count);
}

// The chunk sums' prefixes in place, one block of 1024 threads; returns the grand total.
__device__ __forceinline__ int scan_sums(int* sums, int n) {
  __shared__ int warp_total[32];
  int carry = 0;
  for (int c0 = 0; c0 < n; c0 += 4096) {
    const int g = c0 + threadIdx.x * 4;
    int v[4], t = 0, total;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = g + k < n ? sums[g + k] : 0;
      t += v[k];
    }
    int p = carry + block_prefix(t, warp_total, &total);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (g + k < n) sums[g + k] = p;
      p += v[k];
    }
    carry += total;
    __syncthreads();
  }
  return carry;
}

__global__ __launch_bounds__(1024) void k_scan_sums(int* sums, int nblocks, int* out, int count) {
  const int total = scan_sums(sums, nblocks);
  if (threadIdx.x == 0) out[count] = total;
}

__global__ __launch_bounds__(SCAN_T) void k_scan_add(int* out, const int* sums, int count) {
  const int g = blockIdx.x * SCAN_B + threadIdx.x * 4, add = sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (g + k < count) out[g + k] += add;
}

static void exclusive_scan(cudaStream_t st, const int* counts, int* starts, int* block_sums, int count) {
  int nb = (count + SCAN_B - 1) / SCAN_B;
  k_scan_local<<<nb, SCAN_T, 0, st>>>(counts, starts, block_sums, count);
  k_scan_sums<<<1, 1024, 0, st>>>(block_sums, nb, starts, count);
  k_scan_add<<<nb, SCAN_T, 0, st>>>(starts, block_sums, count);
}

// ---- the reference's BVH face order (utils/bvh2d.cpp:29-64, 165-242) ----
//
// The reference's locator is a BVH over face centroids (leaves of <= 4 faces, depth <= 24,
// TransportMap::init_inverse, transport_map.cpp:36-43). Two of its properties are visible in
// results: the order of the hits of a point (increasing position in its permuted face
// array, the order of the depth-first traversal, bvh2d.cpp:94-162), and that a face is
// only tested where the point lies in the (slightly enlarged) box of the face's leaf.
// Both follow from the permutation the build leaves in its face array, which is
// computed here level by level, all nodes of a level at once:
//   * node box: min / max over its faces' vertices (order-free, exact), enlarged by
//     2 eps diag + eps; split dimension = the first largest extent, split value =
//     float(0.5 (max + min)) of the enlarged box (bvh2d.cpp:178-212);
//   * split() (bvh2d.cpp:167-176) is a two-ended partition. With S the number of
//     "small" centroids (c < split value) in [start, end), the k-th "big" element from
//     the left among the first S positions trades places with the k-th small element
//     from the right among the others -- exactly the pairs its loop swaps -- so prefix
//     counts give every element's final position. Its return value is start + S, plus
//     one when the element then at start + S equals the split value, except in the one
//     loop exit that skips the final scan (last swap at start + S - 2 and start + S);
//   * leaves: <= 4 faces, level >= 24, or a split that leaves one side empty.
// Result per face: rank (position in the final face array) and the box of its leaf.
//
// The build runs in two phases. Nodes of more than BVH_SUB faces are split level by level
// over the whole array, five kernels a level in the body of a WHILE node, windows of
// positions without such a node passed over; a node of at most BVH_SUB faces is set aside
// with its level. Only the face order moves (4 bytes a face); centroids and boxes are read
// where they lie. Then each block takes the subtrees that start in its window of BVH_SUB
// positions through all their remaining levels in shared memory. All 25 levels over the whole
// array, nine kernels and two copies each and 52 bytes moved a face, took 1.73 ms for a
// 1024^2 map, nearly all of it in passes over positions whose nodes were small. Now 0.56 ms go to the 20
// levels of the first phase (bound by launches and by the dependent loads of each kernel: 28
// us a level, 37 launched plainly, where the 20 MB it moves would take 4) and 0.25 ms to the
// second (bound by its barriers; 512 threads on subtrees of up to 512 faces measured best among 128 .. 512 and
// 128 .. 1024).

constexpr int BVH_LEAF = 4, BVH_DEPTH = 24, BVH_SUB = 512;

struct BvhNode {  // a node of more than BVH_SUB faces
  int start, end;
  int leaf, mid;
  int lo, hi;  // children in the next level's list, or -1: set aside
  unsigned long long kmin[2], kmax[2];  // order-preserving keys of the box (atomics)
};

// State of a build: its buffers (set for each build) and the level being split.
struct BvhCtl {
  const double* xy;
  int* rank;
  double4* lbox;
  int level;
};

// node_of of a position: the node's index in its level's list; ~start once its node has been
// set aside; BVH_DONE when the face's leaf is recorded.
constexpr int BVH_DONE = INT_MIN;

__device__ __forceinline__ unsigned long long dkey(double x) {
  unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double dkey_inv(unsigned long long k) {
  unsigned long long u = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
  return __longlong_as_double((long long)u);
}

__device__ __forceinline__ void bvh_node_init(BvhNode& b, int start, int end) {
  b.start = start;
  b.end = end;
  b.leaf = 0;
  b.lo = b.hi = -1;
  b.kmin[0] = b.kmin[1] = ~0ull;
  b.kmax[0] = b.kmax[1] = 0ull;
}

// Enlarged box, split dimension and value of a node from the box of its faces (bvh2d.cpp:178-212).
struct BvhSplit {
  double4 box;  // min x, min y, max x, max y
  int dim;
  double sv;  // a float's value
};
__device__ __forceinline__ BvhSplit bvh_split(const double4& b) {
  const double mn[2] = {b.x, b.y}, mx[2] = {b.z, b.w};
  double diag[2], lo[2], hi[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    diag[c] = mx[c] - mn[c];
    const double en = diag[c] * (2. * DBL_EPSILON) + DBL_EPSILON;
    lo[c] = mn[c] - en;
    hi[c] = mx[c] + en;
  }
  BvhSplit r;
  r.box = make_double4(lo[0], lo[1], hi[0], hi[1]);
  r.dim = diag[1] > diag[0] ? 1 : 0;  // Eigen's maxCoeff: the first of equal maxima
  r.sv = (double)(float)(0.5 * (r.dim ? hi[1] + lo[1] : hi[0] + lo[0]));
  return r;
}
__device__ __forceinline__ BvhSplit bvh_split(const BvhNode& nd) {
  return bvh_split(make_double4(dkey_inv(nd.kmin[0]), dkey_inv(nd.kmin[1]), dkey_inv(nd.kmax[0]), dkey_inv(nd.kmax[1])));
}

// split()'s return value (bvh2d.cpp:175) for a node [start, end) with S small centroids: q =
// start + S, m swapped pairs, eq: the element now at q equals the split value, last: the last
// pair's positions were q - 2 and q (the loop then exits right after its last swap without
// the final scan: it tests the small element at q - 1 and returns q).
__device__ __forceinline__ int bvh_mid(int q, int m, bool eq, bool last) { return q + (eq && !(m >= 1 && last) ? 1 : 0); }

// Boxes hold no NaN (box_of_quad), so a comparison and a selection serve.
__device__ __forceinline__ double4 box_join(double4 a, double4 b) {
  return make_double4(b.x < a.x ? b.x : a.x, b.y < a.y ? b.y : a.y, b.z > a.z ? b.z : a.z, b.w > a.w ? b.w : a.w);
}
__device__ __forceinline__ double4 box_shfl_xor(double4 b, int o, unsigned lanes = 0xffffffffu) {
  return make_double4(__shfl_xor_sync(lanes, b.x, o), __shfl_xor_sync(lanes, b.y, o), __shfl_xor_sync(lanes, b.z, o),
                      __shfl_xor_sync(lanes, b.w, o));
}
__device__ __forceinline__ double4 box_shfl_up(double4 b, int o) {
  return make_double4(__shfl_up_sync(0xffffffffu, b.x, o), __shfl_up_sync(0xffffffffu, b.y, o),
                      __shfl_up_sync(0xffffffffu, b.z, o), __shfl_up_sync(0xffffffffu, b.w, o));
}
__device__ __forceinline__ double4 box_none() { return make_double4(INFINITY, INFINITY, -INFINITY, -INFINITY); }
// Box of a face's corners, NaN coordinates passed over (all of them: the empty box).
__device__ __forceinline__ double4 box_of_quad(const Quad& p) {
  const double4 b = make_double4(fmin(fmin(p.x[0], p.x[1]), fmin(p.x[2], p.x[3])),
                                 fmin(fmin(p.y[0], p.y[1]), fmin(p.y[2], p.y[3])),
                                 fmax(fmax(p.x[0], p.x[1]), fmax(p.x[2], p.x[3])),
                                 fmax(fmax(p.y[0], p.y[1]), fmax(p.y[2], p.y[3])));
  const bool x = b.x == b.x, y = b.y == b.y;
  return make_double4(x ? b.x : INFINITY, y ? b.y : INFINITY, x ? b.z : -INFINITY, y ? b.w : -INFINITY);
}
__device__ __forceinline__ void box_atomic(BvhNode& nd, const double4& b) {
  atomicMin(&nd.kmin[0], dkey(b.x));
  atomicMin(&nd.kmin[1], dkey(b.y));
  atomicMax(&nd.kmax[0], dkey(b.z));
  atomicMax(&nd.kmax[1], dkey(b.w));
}

// A block's window of the array: BVH_PER positions per thread, BVH_BT apart.
constexpr int BVH_BT = 256, BVH_PER = SCAN_B / BVH_BT;

// Folds the boxes of the window's positions (id: their nodes, -1 for none) into the nodes with
// 64-bit atomics on order-preserving keys. A node's positions are contiguous: a window that
// lies in one node (the upper levels) is reduced first and issues one set of atomics;
// otherwise every warp folds each run of equal nodes with a segmented shuffle scan and the
// last lane of a run issues its atomics. Returns whether the window has any node. All threads
// call it.
__device__ __forceinline__ bool window_boxes(BvhNode* nodes, const int (&id)[BVH_PER], double4 (&box)[BVH_PER]) {
  __shared__ int s_first;
  __shared__ double4 s_box[BVH_BT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool same = true, some = false;
#pragma unroll
  for (int j = 0; j < BVH_PER; ++j) {
    same = same && id[j] == id[0];
    some = some || id[j] >= 0;
  }
  if (threadIdx.x == 0) s_first = id[0];
  if (!__syncthreads_or(some)) return false;
  const int first = s_first;
  if (__syncthreads_and(same && id[0] == first)) {
    double4 b = box_join(box_join(box[0], box[1]), box_join(box[2], box[3]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = box_join(b, box_shfl_xor(b, o));
    if (lane == 0) s_box[warp] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
      double4 t = s_box[0];
#pragma unroll
      for (int w = 1; w < BVH_BT / 32; ++w) t = box_join(t, s_box[w]);
      box_atomic(nodes[first], t);
    }
    return true;
  }
#pragma unroll
  for (int j = 0; j < BVH_PER; ++j) {
    const int k = id[j];
    if (!__any_sync(0xffffffffu, k >= 0)) continue;
    double4 b = box[j];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double4 u = box_shfl_up(b, o);
      const int ku = __shfl_up_sync(0xffffffffu, k, o);
      if (lane >= o && ku == k) b = box_join(b, u);
    }
    const int kn = __shfl_down_sync(0xffffffffu, k, 1);
    if (k >= 0 && (lane == 31 || kn != k)) box_atomic(nodes[k], b);
  }
  return true;
}

__global__ void k_bvh_root(BvhCtl* ctl, int N, BvhNode* root, int* sub_end, unsigned char* sub_level) {
  bvh_node_init(*root, 0, N);
  ctl->level = 0;
  sub_end[0] = N;
  sub_level[0] = 0;
}

// Face centroids (bvh2d.cpp:44-58: zero + the corners in circulator order, / 4), face
// boxes, identity permutation, every position in the root node with its box -- or, for a
// mesh of at most BVH_SUB faces, the root set aside.
__global__ __launch_bounds__(BVH_BT) void k_bvh_init(const BvhCtl* ctl, int n, int* fac, int* final_fac, double2* cen,
                                                     double4* fbox, int* node_of, BvhNode* root,
                                                     unsigned char* window) {
  const int N = n * n;
  const double* xy = ctl->xy;
  int id[BVH_PER];
  double4 box[BVH_PER];
#pragma unroll
  for (int j = 0; j < BVH_PER; ++j) {
    const int f = (blockIdx.x * BVH_PER + j) * BVH_BT + threadIdx.x;
    id[j] = -1;
    box[j] = box_none();
    if (f >= N) continue;
    Quad p;
    int vid[4];
    load_quad(xy, n, f, p, vid);
    double cx = 0.0, cy = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      cx += p.x[k];
      cy += p.y[k];
    }
    cen[f] = make_double2(cx / 4, cy / 4);
    box[j] = box_of_quad(p);
    fbox[f] = box[j];
    if (N > BVH_SUB) {
      fac[f] = f;
      node_of[f] = id[j] = 0;
    } else {
      final_fac[f] = f;
      node_of[f] = ~0;
    }
  }
  const bool some = window_boxes(root, id, box);
  if (threadIdx.x == 0) window[blockIdx.x] = some ? 1 : 0;
}

// small[p] = 1 when position p's centroid lies below its node's split value, and the window-
// local prefix counts lpre (N + 1 of them; a window's first is 0 from the first level on).
__global__ __launch_bounds__(SCAN_T) void k_bvh_classify(int N, const BvhCtl* ctl, const int* node_of, const int* fac0,
                                                         const int* fac1, const double2* cen, const BvhNode* even,
                                                         const BvhNode* odd, const unsigned char* window0,
                                                         const unsigned char* window1, unsigned char* small, int* lpre,
                                                         int* sums) {
  overlap_wait();
  const int level = ctl->level;
  const bool at_end = (long)blockIdx.x * SCAN_B >= N;  // the window of p = N alone
  if (level > 0 && (at_end || !(level & 1 ? window1 : window0)[blockIdx.x])) {
    if (threadIdx.x == 0) sums[blockIdx.x] = 0;
    return;
  }
  const BvhNode* nodes = level & 1 ? odd : even;
  const int* fac = level & 1 ? fac1 : fac0;
  int last = -1;
  BvhSplit sp;
  scan_chunk(
      [&](int p) {
        const int k = p < N ? node_of[p] : -1;
        if (k < 0) return 0;
        if (k != last) {
          sp = bvh_split(nodes[k]);
          last = k;
        }
        const double2 c = cen[fac[p]];
        const int s = (sp.dim ? c.y : c.x) < sp.sv ? 1 : 0;
        small[p] = (unsigned char)s;
        return s;
      },
      lpre, sums, N + 1);
}

__global__ __launch_bounds__(1024) void k_bvh_sums(int* sums, int nsums) {
  overlap_wait();
  scan_sums(sums, nsums);
}

// Small positions before p.
struct BvhPrefix {
  const int *lpre, *sums;
  __device__ __forceinline__ int operator()(int p) const { return lpre[p] + sums[p / SCAN_B]; }
};

// The partition's pairs: big elements among the first S positions (rank from the left)
// and small elements after them (rank from the right) record their positions by rank.
__global__ __launch_bounds__(BVH_BT) void k_bvh_slots(int N, const BvhCtl* ctl, const int* node_of,
                                                      const BvhNode* even, const BvhNode* odd,
                                                      const unsigned char* window0, const unsigned char* window1,
                                                      const unsigned char* small, BvhPrefix pre, int* slot_big,
                                                      int* slot_small) {
  overlap_wait();
  const int level = ctl->level;
  if (!(level & 1 ? window1 : window0)[blockIdx.x]) return;
#pragma unroll
  for (int j = 0; j < BVH_PER; ++j) {
    const int p = (blockIdx.x * BVH_PER + j) * BVH_BT + threadIdx.x, k = p < N ? node_of[p] : -1;
    if (k < 0) continue;
    const BvhNode& nd = (level & 1 ? odd : even)[k];
    const int start = nd.start, before = pre(start), upto = pre(nd.end), q = start + upto - before;
    if (!small[p] && p < q) {
      slot_big[start + (p - start) - (pre(p) - before)] = p;
    } else if (small[p] && p >= q) {
      slot_small[start + upto - pre(p) - 1] = p;
    }
  }
}

// Position whose element stands at p once the pairs have traded places.
__device__ __forceinline__ int bvh_source(int p, int start, int before, int upto, int pre_p, bool small,
                                          const int* slot_big, const int* slot_small) {
  const int q = start + upto - before;
  if (!small && p < q) return slot_small[start + (p - start) - (pre_p - before)];
  if (small && p >= q) return slot_big[start + upto - pre_p - 1];
  return p;
}

// The leaf tests by depth and no improvement (:214-221), the children -- listed for the next
// level or set aside -- the level count and the loop test (one block).
__global__ __launch_bounds__(1024) void k_bvh_children(BvhCtl* ctl, int* counts, BvhNode* even, BvhNode* odd,
                                                       const int* fac0, const int* fac1, const unsigned char* small,
                                                       BvhPrefix pre, const int* slot_big, const int* slot_small,
                                                       const double2* cen, int* sub_end, unsigned char* sub_level,
                                                       cudaGraphConditionalHandle handle, int in_graph) {
  __shared__ int s_next;
  overlap_wait();
  const int level = ctl->level, count = level ? counts[level & 1] : 1;
  BvhNode* nodes = level & 1 ? odd : even;
  BvhNode* next = level & 1 ? even : odd;
  const int* fac = level & 1 ? fac1 : fac0;
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < count; k += blockDim.x) {
    BvhNode& nd = nodes[k];
    const int start = nd.start, end = nd.end;
    if (level >= BVH_DEPTH) {
      nd.leaf = 1;
      continue;
    }
    const int before = pre(start), upto = pre(end), S = upto - before;
    int mid = end;  // no big element: the loop runs to `end` and both branches give end
    if (S != end - start) {
      const BvhSplit sp = bvh_split(nd);
      const int q = start + S, pre_q = pre(q), m = S - (pre_q - before);
      const double2 c = cen[fac[bvh_source(q, start, before, upto, pre_q, small[q] != 0, slot_big, slot_small)]];
      const bool last = m >= 1 && slot_big[start + m - 1] == q - 2 && slot_small[start + m - 1] == q;
      mid = bvh_mid(q, m, (sp.dim ? c.y : c.x) == sp.sv, last);
    }
    nd.mid = mid;
    if (mid == start || mid == end) {
      nd.leaf = 1;
      continue;
    }
    auto child = [&](int s, int e) {
      if (e - s > BVH_SUB) {
        const int c = atomicAdd(&s_next, 1);
        bvh_node_init(next[c], s, e);
        return c;
      }
      sub_end[s] = e;
      sub_level[s] = (unsigned char)(level + 1);
      return -1;
    };
    nd.lo = child(start, mid);
    nd.hi = child(mid, end);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ctl->level = level + 1;
    counts[(level + 1) & 1] = s_next;
    if (in_graph) cudaGraphSetConditional(handle, s_next > 0 ? 1u : 0u);
  }
}

// End of a level: the pairs trade places and every position moves to its child -- or, where the
// node became a leaf, records its face's rank and leaf box -- with the boxes of the next
// level's nodes.
__global__ __launch_bounds__(BVH_BT) void k_bvh_move(int N, const BvhCtl* ctl, int* node_of, int* fac0, int* fac1,
                                                     int* final_fac, const double4* fbox, BvhNode* even, BvhNode* odd,
                                                     unsigned char* window0, unsigned char* window1,
                                                     const unsigned char* small, BvhPrefix pre, const int* slot_big,
                                                     const int* slot_small) {
  overlap_wait();
  const int level = ctl->level - 1;  // k_bvh_children has counted it
  unsigned char* to = level & 1 ? window0 : window1;
  if (!(level & 1 ? window1 : window0)[blockIdx.x]) {
    if (threadIdx.x == 0) to[blockIdx.x] = 0;
    return;
  }
  const BvhNode* nodes = level & 1 ? odd : even;
  const int* from = level & 1 ? fac1 : fac0;
  int* into = level & 1 ? fac0 : fac1;
  int id[BVH_PER];
  double4 box[BVH_PER];
#pragma unroll
  for (int j = 0; j < BVH_PER; ++j) {
    const int p = (blockIdx.x * BVH_PER + j) * BVH_BT + threadIdx.x, k = p < N ? node_of[p] : -1;
    id[j] = -1;
    box[j] = box_none();
    if (k < 0) continue;
    const BvhNode& nd = nodes[k];
    const int start = nd.start;
    const int src = level >= BVH_DEPTH ? p
                                       : bvh_source(p, start, pre(start), pre(nd.end), pre(p), small[p] != 0, slot_big,
                                                    slot_small);
    const int f = from[src];
    if (nd.leaf) {
      ctl->rank[f] = p;
      ctl->lbox[f] = bvh_split(nd).box;
      node_of[p] = BVH_DONE;
      continue;
    }
    const bool low = p < nd.mid;
    const int child = low ? nd.lo : nd.hi;
    if (child >= 0) {
      into[p] = f;
      node_of[p] = id[j] = child;
      box[j] = fbox[f];
    } else {
      final_fac[p] = f;
      node_of[p] = ~(low ? start : nd.mid);
    }
  }
  const bool some = window_boxes(level & 1 ? even : odd, id, box);
  if (threadIdx.x == 0) to[blockIdx.x] = some ? 1 : 0;
}

// Second phase: block b takes the subtrees set aside that start in positions
// [b BVH_SUB, (b+1) BVH_SUB) -- at most 2 BVH_SUB - 1 positions -- through their remaining
// levels, all nodes of a level at once as in the first phase, on a permutation in shared
// memory. Nodes of at most BVH_LEAF faces are recorded when they appear. A node's box is folded
// by eight lanes when it has at most SMALL_NODE faces, else by a warp.
constexpr int SMALL_NODE = 64;
constexpr int BVH_WIN = 2 * BVH_SUB, BVH_T = 512, BVH_NODES = BVH_WIN / (BVH_LEAF + 1) + 1;

struct BvhWindow {
  double4 fbox[BVH_WIN];                   // by original position
  double2 cen[BVH_WIN];
  BvhSplit split[BVH_NODES];
  int face[BVH_WIN];
  unsigned short perm[BVH_WIN];            // original position of the element at a position
  unsigned short node[BVH_WIN];            // the position's node, or NONE
  unsigned short pre[BVH_WIN + 1];         // small positions before it
  unsigned short slot_big[BVH_WIN], slot_small[BVH_WIN];
  unsigned char small[BVH_WIN];
  struct Node {
    unsigned short start, end, mid, lo, hi;
    unsigned char level, leaf;
  } nodes[2][BVH_NODES];
  int warp_total[32], count, lo, hi;
};

__global__ __launch_bounds__(BVH_T) void k_bvh_subtrees(int N, const BvhCtl* ctl, const int* node_of,
                                                        const int* final_fac, const double2* cen, const double4* fbox,
                                                        const int* sub_end, const unsigned char* sub_level) {
  extern __shared__ __align__(16) unsigned char s_window[];
  BvhWindow& W = *reinterpret_cast<BvhWindow*>(s_window);
  constexpr unsigned short NONE = 0xffff;
  constexpr int PER = BVH_WIN / BVH_T;
  int* rank = ctl->rank;
  double4* lbox = ctl->lbox;
  const int w0 = blockIdx.x * BVH_SUB, w1 = min(w0 + BVH_SUB, N), lane = threadIdx.x & 31;
  // the window's subtrees: the first starts at the first position that is its node's start,
  // the last ends where the node of the last position starting in the window ends
  if (threadIdx.x == 0) {
    W.lo = N;
    W.hi = 0;
    W.count = 0;
  }
  __syncthreads();
  for (int p = w0 + threadIdx.x; p < w1; p += BVH_T)
    if (node_of[p] == ~p) {
      atomicMin(&W.lo, p);
      atomicMax(&W.hi, sub_end[p]);
    }
  __syncthreads();
  const int base = W.lo, M = W.hi - W.lo;
  if (M <= 0) return;
  // a node of at most BVH_LEAF faces: its box over them, ranks and leaf boxes (one thread)
  auto box_of = [&](int s, int e, int step) {
    double4 b = W.fbox[W.perm[s]];
    for (int p = s + step; p < e; p += step) b = box_join(b, W.fbox[W.perm[p]]);
    return b;
  };
  auto record_leaf = [&](int s, int e) {
    const double4 b = bvh_split(box_of(s, e, 1)).box;
    for (int p = s; p < e; ++p) {
      const int f = W.face[W.perm[p]];
      rank[f] = base + p;
      lbox[f] = b;
    }
  };
  // load; every start makes its node, then every position finds it (slot_big: node of a start)
  for (int p = threadIdx.x; p < M; p += BVH_T) {
    W.perm[p] = (unsigned short)p;
    if (node_of[base + p] == BVH_DONE) continue;  // of a leaf between subtrees
    const int f = final_fac[base + p];
    W.face[p] = f;
    W.cen[p] = cen[f];
    W.fbox[p] = fbox[f];
  }
  __syncthreads();
  for (int p = threadIdx.x; p < M; p += BVH_T) {
    if (node_of[base + p] != ~(base + p)) continue;
    const int e = sub_end[base + p] - base;
    unsigned short id = NONE;
    if (e - p <= BVH_LEAF) {
      record_leaf(p, e);
    } else {
      id = (unsigned short)atomicAdd(&W.count, 1);
      W.nodes[0][id] = {(unsigned short)p, (unsigned short)e, 0, 0, 0, sub_level[base + p], 0};
    }
    W.slot_big[p] = id;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < M; p += BVH_T) {
    const int k = node_of[base + p];
    W.node[p] = k == BVH_DONE ? NONE : W.slot_big[~k - base];
  }
  int count = W.count;
  for (int par = 0; count > 0; par ^= 1) {
    auto* nodes = W.nodes[par];
    auto* next = W.nodes[par ^ 1];
    __syncthreads();
    if (threadIdx.x == 0) W.count = 0;
    for (int k = threadIdx.x >> 3; k < count; k += BVH_T / 8) {
      const int s = nodes[k].start + (lane & 7), e = nodes[k].end;
      if (e - nodes[k].start > SMALL_NODE) continue;
      double4 b = s < e ? box_of(s, e, 8) : box_none();
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) b = box_join(b, box_shfl_xor(b, o, 0xffu << (lane & 24)));
      if ((lane & 7) == 0) W.split[k] = bvh_split(b);
    }
    for (int k = threadIdx.x >> 5; k < count; k += BVH_T / 32) {
      const int s = nodes[k].start + lane, e = nodes[k].end;
      if (e - nodes[k].start <= SMALL_NODE) continue;
      double4 b = s < e ? box_of(s, e, 32) : box_none();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) b = box_join(b, box_shfl_xor(b, o));
      if (lane == 0) W.split[k] = bvh_split(b);
    }
    __syncthreads();
    // classify and count: thread t takes positions PER t .. PER t + PER - 1
    {
      int v[PER], t = 0, total;
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int p = threadIdx.x * PER + j, k = p < M ? W.node[p] : NONE;
        v[j] = 0;
        if (k != NONE) {
          const double2 c = W.cen[W.perm[p]];
          v[j] = (W.split[k].dim ? c.y : c.x) < W.split[k].sv ? 1 : 0;
          W.small[p] = (unsigned char)v[j];
        }
        t += v[j];
      }
      int x = block_prefix(t, W.warp_total, &total);
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int p = threadIdx.x * PER + j;
        if (p < M) W.pre[p] = (unsigned short)x;
        x += v[j];
      }
      if (threadIdx.x == 0) W.pre[M] = (unsigned short)total;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < M; p += BVH_T) {
      const int k = W.node[p];
      if (k == NONE) continue;
      const int s = nodes[k].start, before = W.pre[s], upto = W.pre[nodes[k].end], q = s + upto - before;
      if (!W.small[p] && p < q)
        W.slot_big[s + (p - s) - (W.pre[p] - before)] = (unsigned short)p;
      else if (W.small[p] && p >= q)
        W.slot_small[s + upto - W.pre[p] - 1] = (unsigned short)p;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < M; p += BVH_T) {
      const int k = W.node[p];
      if (k == NONE || W.small[p] || nodes[k].level >= BVH_DEPTH) continue;
      const int s = nodes[k].start, before = W.pre[s];
      if (p >= s + W.pre[nodes[k].end] - before) continue;
      const int r = W.slot_small[s + (p - s) - (W.pre[p] - before)];
      const unsigned short t = W.perm[p];
      W.perm[p] = W.perm[r];
      W.perm[r] = t;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < count; k += BVH_T) {
      auto& nd = nodes[k];
      const int s = nd.start, e = nd.end;
      nd.leaf = 1;
      if (nd.level >= BVH_DEPTH) continue;
      const int before = W.pre[s], S = W.pre[e] - before;
      int mid = e;
      if (S != e - s) {
        const int q = s + S, m = S - (W.pre[q] - before);
        const double2 c = W.cen[W.perm[q]];
        const bool last = m >= 1 && W.slot_big[s + m - 1] == q - 2 && W.slot_small[s + m - 1] == q;
        mid = bvh_mid(q, m, (W.split[k].dim ? c.y : c.x) == W.split[k].sv, last);
      }
      if (mid == s || mid == e) continue;
      nd.leaf = 0;
      nd.mid = (unsigned short)mid;
      auto child = [&](int cs, int ce) -> unsigned short {
        if (ce - cs <= BVH_LEAF) return NONE;
        const int c = atomicAdd(&W.count, 1);
        next[c] = {(unsigned short)cs, (unsigned short)ce, 0, 0, 0, (unsigned char)(nd.level + 1), 0};
        return (unsigned short)c;
      };
      nd.lo = child(s, mid);
      nd.hi = child(mid, e);
    }
    __syncthreads();
    for (int p = threadIdx.x; p < M; p += BVH_T) {
      const int k = W.node[p];
      if (k == NONE) continue;
      const auto& nd = nodes[k];
      if (nd.leaf) {
        const int f = W.face[W.perm[p]];
        rank[f] = base + p;
        lbox[f] = W.split[k].box;
        W.node[p] = NONE;
      } else {
        const bool low = p < nd.mid;
        const unsigned short c = low ? nd.lo : nd.hi;
        W.node[p] = c;
        if (c == NONE && p == (low ? nd.start : nd.mid)) record_leaf(p, low ? nd.mid : nd.end);
      }
    }
    count = W.count;
  }
}

// Levels per body of the first phase's WHILE node. A body costs about 3 us beside its kernels, a
// level after the last one five launches that return at once; the kernels overlap their
// predecessor's end (common.cuh). A query of 2^20 points on a new mesh of 64^2, 256^2 and 1024^2
// faces: one level per body with plain launches 455, 704 and 1477 us, overlapped 442, 674 and
// 1446, two levels 422, 670 and 1408, three 418, 648 and 1408, four 432, 668 and 1399.
constexpr int LEVELS_PER_BODY = 3;

// rank[f] and the leaf box of f for the n^2 quads of the forward mesh xy (device). The launches
// run as one CUDA graph per size (captured on first use, kept in the context) on the
// context's grow-only scratch; a build's own buffers reach it through the control block.
// With profiling on, the same launches are issued one by one so that each is timed.
static void build_bvh_order(otm_context* ctx, const double* xy, int n, int* rank, double4* lbox) {
  cudaStream_t st = ctx->stream;
  const int N = n * n;
  const int cap = N / (BVH_SUB + 1) + 2;  // nodes of a level in the first phase
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  const int windows = (N + SCAN_B - 1) / SCAN_B, nsums = N / SCAN_B + 1;
  const size_t b_int = al(sizeof(int) * ((size_t)N + 1)), b_byte = al((size_t)N), b_nodes = al(sizeof(BvhNode) * cap);
  const size_t b_cen = al(sizeof(double2) * N), b_box = al(sizeof(double4) * N), b_sums = al(sizeof(int) * nsums);
  const size_t b_win = al((size_t)windows);
  DevBuf& buf = ctx->bvh_scratch;  // grow-only: no allocation once a size has been built
  buf.reserve(8 * b_int + 2 * b_byte + b_cen + b_box + 2 * b_nodes + b_sums + 2 * b_win + 256);
  char* q = buf.as<char>();
  auto take = [&](size_t b) {
    char* r = q;
    q += b;
    return r;
  };
  BvhCtl* ctl = reinterpret_cast<BvhCtl*>(take(256));
  int* counts = reinterpret_cast<int*>(ctl + 1);  // nodes in the lists of even and odd levels
  double2* cen = reinterpret_cast<double2*>(take(b_cen));
  double4* fbox = reinterpret_cast<double4*>(take(b_box));
  int* fac0 = reinterpret_cast<int*>(take(b_int));
  int* fac1 = reinterpret_cast<int*>(take(b_int));
  int* final_fac = reinterpret_cast<int*>(take(b_int));
  int* node_of = reinterpret_cast<int*>(take(b_int));
  int* lpre = reinterpret_cast<int*>(take(b_int));
  int* slot_big = reinterpret_cast<int*>(take(b_int));
  int* slot_small = reinterpret_cast<int*>(take(b_int));
  int* sub_end = reinterpret_cast<int*>(take(b_int));
  unsigned char* small = reinterpret_cast<unsigned char*>(take(b_byte));
  unsigned char* sub_level = reinterpret_cast<unsigned char*>(take(b_byte));
  BvhNode* even = reinterpret_cast<BvhNode*>(take(b_nodes));
  BvhNode* odd = reinterpret_cast<BvhNode*>(take(b_nodes));
  int* sums = reinterpret_cast<int*>(take(b_sums));
  unsigned char* win0 = reinterpret_cast<unsigned char*>(take(b_win));
  unsigned char* win1 = reinterpret_cast<unsigned char*>(take(b_win));
  const BvhPrefix pre{lpre, sums};
  using CBytes = const unsigned char*;
  auto level = [&](cudaGraphConditionalHandle handle, int in_graph) {
    launch(ctx, "bvh_classify", k_bvh_classify, nsums, SCAN_T, N, (const BvhCtl*)ctl, (const int*)node_of,
           (const int*)fac0, (const int*)fac1, (const double2*)cen, (const BvhNode*)even, (const BvhNode*)odd,
           (CBytes)win0, (CBytes)win1, small, lpre, sums);
    launch(ctx, "bvh_sums", k_bvh_sums, 1, 1024, sums, nsums);
    launch(ctx, "bvh_slots", k_bvh_slots, windows, BVH_BT, N, (const BvhCtl*)ctl, (const int*)node_of,
           (const BvhNode*)even, (const BvhNode*)odd, (CBytes)win0, (CBytes)win1, (CBytes)small, pre, slot_big,
           slot_small);
    launch(ctx, "bvh_children", k_bvh_children, 1, 1024, ctl, counts, even, odd, (const int*)fac0, (const int*)fac1,
           (CBytes)small, pre, (const int*)slot_big, (const int*)slot_small, (const double2*)cen, sub_end, sub_level,
           handle, in_graph);
    launch(ctx, "bvh_move", k_bvh_move, windows, BVH_BT, N, (const BvhCtl*)ctl, node_of, fac0, fac1, final_fac,
           (const double4*)fbox, even, odd, win0, win1, (CBytes)small, pre, (const int*)slot_big,
           (const int*)slot_small);
  };
  auto begin = [&] {
    launch(ctx, "bvh_root", k_bvh_root, 1, 1, ctl, N, even, sub_end, sub_level);
    launch(ctx, "bvh_init", k_bvh_init, windows, BVH_BT, (const BvhCtl*)ctl, n, fac0, final_fac, cen, fbox, node_of,
           even, win0);
  };
  auto finish = [&] {
    launch_smem(ctx, "bvh_subtrees", k_bvh_subtrees, (unsigned)((N + BVH_SUB - 1) / BVH_SUB), BVH_T, sizeof(BvhWindow),
                N, (const BvhCtl*)ctl, (const int*)node_of, (const int*)final_fac, (const double2*)cen,
                (const double4*)fbox, (const int*)sub_end, (CBytes)sub_level);
  };
  static bool attr[64] = {};  // per device ordinal
  if (ctx->device >= 64 || !attr[ctx->device]) {
    OTM_CUDA(cudaFuncSetAttribute(k_bvh_subtrees, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BvhWindow)));
    if (ctx->device < 64) attr[ctx->device] = true;
  }
  BvhCtl h = {xy, rank, lbox, 0};
  OTM_CUDA(cudaMemcpyAsync(ctl, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  if (ctx->prof.on) {
    begin();
    int left[2] = {1, 1};
    for (int l = 0; N > BVH_SUB && left[l & 1]; ++l) {
      level((cudaGraphConditionalHandle)0, 0);
      OTM_CUDA(cudaMemcpyAsync(left, counts, sizeof(left), cudaMemcpyDeviceToHost, st));
      OTM_CUDA(cudaStreamSynchronize(st));
    }
    finish();
  } else {
    auto& slot = ctx->bvh_graphs[n];
    if (!slot || slot->base != buf.p) {
      slot.reset(new otm_context::GraphExec());
      slot->base = buf.p;
      cudaGraph_t g = nullptr;
      const long before = ctx->launches;
      OTM_CUDA(cudaGraphCreate(&g, 0));
      auto capture = [&](cudaGraph_t to, const cudaGraphNode_t* after, auto&& body) {
        cudaGraph_t done = nullptr;
        OTM_CUDA(cudaStreamBeginCaptureToGraph(st, to, after, nullptr, after ? 1 : 0, cudaStreamCaptureModeThreadLocal));
        try {
          body();
        } catch (...) {
          cudaStreamEndCapture(st, &done);
          throw;
        }
        OTM_CUDA(cudaStreamEndCapture(st, &done));
      };
      try {
        // begin and finish around the loop: child graphs, so that each is one node
        cudaGraph_t part = nullptr;
        cudaGraphNode_t last;
        auto add_part = [&](const cudaGraphNode_t* after, auto&& body) {
          OTM_CUDA(cudaGraphCreate(&part, 0));
          capture(part, nullptr, body);
          OTM_CUDA(cudaGraphAddChildGraphNode(&last, g, after, after ? 1 : 0, part));
          cudaGraphDestroy(part);
          part = nullptr;
        };
        try {
          add_part(nullptr, begin);
          if (N > BVH_SUB) {
            cudaGraphConditionalHandle handle;
            OTM_CUDA(cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault));
            cudaGraphNodeParams params = {};
            params.type = cudaGraphNodeTypeConditional;
            params.conditional.handle = handle;
            params.conditional.type = cudaGraphCondTypeWhile;
            params.conditional.size = 1;
            cudaGraphNode_t loop;
            OTM_CUDA(cudaGraphAddNode(&loop, g, &last, 1, &params));
            capture(params.conditional.phGraph_out[0], nullptr, [&] {
              const Overlap overlap(ctx, true, N);
              for (int l = 0; l < LEVELS_PER_BODY; ++l) level(handle, 1);
            });
            last = loop;
          }
          const cudaGraphNode_t after = last;
          add_part(&after, finish);
        } catch (...) {
          if (part) cudaGraphDestroy(part);
          throw;
        }
        slot->kernels = ctx->launches - before;
        ctx->launches = before;  // captured, not executed
        OTM_CUDA(cudaGraphInstantiate(&slot->exec, g, 0));
      } catch (...) {
        ctx->launches = before;
        slot.reset();
        cudaGraphDestroy(g);
        throw;
      }
      cudaGraphDestroy(g);
    }
    OTM_CUDA(cudaGraphLaunch(slot->exec, st));
    ctx->launches += slot->kernels;  // one body of levels: how many ran stays on the device
  }
  OTM_CUDA(cudaGetLastError());
}

// ---- point location (TransportMap::init_inverse / inv_impl) ----

// Bin range of face f's bounding box, enlarged so that every point the reference's
// tolerant tests can accept (inside_quad eps 1e-8, weight snapping) lands inside it.
__device__ __forceinline__ void face_bins(const Quad& p, int B, int& bx0, int& bx1, int& by0, int& by1,
                                          double4& box) {
  double mnx = fmin(fmin(p.x[0], p.x[1]), fmin(p.x[2], p.x[3]));
  double mxx = fmax(fmax(p.x[0], p.x[1]), fmax(p.x[2], p.x[3]));
  double mny = fmin(fmin(p.y[0], p.y[1]), fmin(p.y[2], p.y[3]));
  double mxy = fmax(fmax(p.y[0], p.y[1]), fmax(p.y[2], p.y[3]));
  double m = 1e-6 * fmax(mxx - mnx, mxy - mny) + 1e-12;
  box = make_double4(mnx - m, mny - m, mxx + m, mxy + m);
  auto cl = [B](double v) {
    double t = floor(v * (double)B);
    return t >= B ? B - 1 : (t > 0 ? (int)t : 0);  // 0 for NaN
  };
  bx0 = cl(box.x);
  bx1 = cl(box.z);
  by0 = cl(box.y);
  by1 = cl(box.w);
}

// The bins' counts, and their sum in 64 bits. Once that is beyond an int the bins are too many
// (build_locator) and faces of many bins leave theirs out.
constexpr int BIN_T = 256;
__global__ __launch_bounds__(BIN_T) void k_bin_count(const double* xy, int n, int B, int* counts, double4* boxes,
                                                     unsigned long long* sum) {
  __shared__ unsigned long long s_all[BIN_T / 32];
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long bins = 0;
  int bx0 = 0, bx1 = -1, by0 = 0, by1 = -1;
  if (f < n * n) {
    Quad p;
    int vid[4];
    load_quad(xy, n, f, p, vid);
    double4 box;
    face_bins(p, B, bx0, bx1, by0, by1, box);
    boxes[f] = box;
    bins = (unsigned long long)(bx1 - bx0 + 1) * (by1 - by0 + 1);
  }
  unsigned long long all = bins;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
  if ((threadIdx.x & 31) == 0) s_all[threadIdx.x >> 5] = all;
  __syncthreads();
  if (threadIdx.x == 0) {  // an add per block: one per warp took 0.7 ms at 4096^2
    for (int w = 1; w < BIN_T / 32; ++w) all += s_all[w];
    atomicAdd(sum, all);
  }
  __syncthreads();
  for (int by = by0; by <= by1; ++by) {
    if (bins > 64 && __ldcg(sum) > (unsigned long long)INT_MAX) return;
    for (int bx = bx0; bx <= bx1; ++bx) atomicAdd(&counts[by * B + bx], 1);
  }
}

__global__ void k_bin_fill(const double* xy, int n, int B, const int* starts, int* cursor, int* faces) {
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n * n) return;
  Quad p;
  int vid[4];
  load_quad(xy, n, f, p, vid);
  int bx0, bx1, by0, by1;
  double4 box;
  face_bins(p, B, bx0, bx1, by0, by1, box);
  for (int by = by0; by <= by1; ++by)
    for (int bx = bx0; bx <= bx1; ++bx) {
      int b = by * B + bx;
      faces[starts[b] + atomicAdd(&cursor[b], 1)] = f;
    }
}

constexpr int MAXHITS = 8;

// inside_tri's answer where it is certain without its two divisions: 1 inside, -1 outside, 0 to
// be computed. The test's tolerance is 1e-8; a term 1e-7 beyond it decides (NaN decides nothing).
__device__ __forceinline__ int tri_verdict(double qx, double qy, double p0x, double p0y, double p1x, double p1y,
                                           double p2x, double p2y) {
  const double q2x = qx - p2x, q2y = qy - p2y;
  const double eux = p1x - p2x, euy = p1y - p2y;
  const double evx = p0x - p2x, evy = p0y - p2y;
  double area2 = cross2(evx, evy, eux, euy);
  double u = cross2(q2x, q2y, eux, euy), v = cross2(evx, evy, q2x, q2y);
  if (area2 < 0) {
    area2 = -area2;
    u = -u;
    v = -v;
  }
  const double m = area2 * 1e-7, s = u + v;
  if ((u < -m) | (v < -m) | (s > area2 + m)) return -1;
  return (u > m) & (v > m) & (s < area2 - m) ? 1 : 0;
}

// Whether point (qx, qy) hits face p: the face tests of bvh2d.cpp:117-142 (inside_quad, then
// the bilinear weights in [0, 1]), by the certain verdicts where they decide.
__device__ __forceinline__ bool hits_face(double qx, double qy, const Quad& p) {
  const int t0 = tri_verdict(qx, qy, p.x[0], p.y[0], p.x[1], p.y[1], p.x[2], p.y[2]);
  if (t0 <= 0) {
    const int t1 = tri_verdict(qx, qy, p.x[0], p.y[0], p.x[2], p.y[2], p.x[3], p.y[3]);
    if (t1 <= 0 && (t0 < 0) & (t1 < 0)) return false;
    if (t1 <= 0 && !inside_quad(qx, qy, p)) return false;
  }
  Bilinear t;
  if (!bilinear_terms(qx, qy, p, t)) return false;
  const int verdict = bilinear_verdict(t);
  if (verdict != 0) return verdict > 0;
  double w[4];
  bilinear_from_terms(t, w);
  return weights_inside(w);
}

// The locator's arrays (build_locator, build_bvh_order).
struct Locator {
  const double* xy;
  const double* density;
  int n, B;
  const int* starts;
  const int* faces;
  const double4* boxes;
  const int* rank;
  const double4* lbox;
};

// The first hit's face and the chosen one for a point with more hits than a warp's lists hold:
// a walk of its bin that keeps the first MAXHITS in the reference's order.
__device__ __noinline__ int many_hits(const Locator& L, int b, double qx, double qy, int densest, int* first) {
  int hf[MAXHITS], hr[MAXHITS], nh = 0;
  for (int k = L.starts[b]; k < L.starts[b + 1]; ++k) {
    const int f = L.faces[k];
    const double4 bb = L.boxes[f];
    if (qx < bb.x || qx > bb.z || qy < bb.y || qy > bb.w) continue;
    Quad p;
    int vid[4];
    load_quad(L.xy, L.n, f, p, vid);
    if (!hits_face(qx, qy, p)) continue;
    const double4 lb = L.lbox[f];
    if (!(lb.x <= qx && lb.y <= qy && qx <= lb.z && qy <= lb.w)) continue;
    const int rk = L.rank[f];
    if (nh >= MAXHITS && rk > hr[MAXHITS - 1]) continue;
    int pos = nh < MAXHITS ? nh : MAXHITS - 1;
    while (pos > 0 && hr[pos - 1] > rk) {
      hf[pos] = hf[pos - 1];
      hr[pos] = hr[pos - 1];
      --pos;
    }
    hf[pos] = f;
    hr[pos] = rk;
    if (nh < MAXHITS) ++nh;
  }
  *first = hf[0];
  int f = hf[0];
  double best = L.density[f];
  for (int k = 1; densest && k < nh; ++k) {
    const double dk = L.density[hf[k]];
    if (dk > best) {
      f = hf[k];
      best = dk > best;
    }
  }
  return f;
}

// inv_impl (transport_map.cpp:50-102) per point. A face of the point's bin is a hit when the
// point lies in the box of the face's BVH leaf (the reference only reaches faces through
// their leaf, bvh2d.cpp:148-161) and passes the face tests; hits are ordered by the face's
// position in the reference's BVH face array, its traversal order. With several hits the
// reference keeps the weights of its first hit and the face of the densest later one
// (transport_map.cpp:70-85); the first-hit mode (inv_fast, bvh2d.cpp:66-81) keeps the first.
//
// The lengths of the points' face lists differ widely (4.6 faces a bin on average, 200 where a
// map squeezes its mesh), so a warp pools the lists of its 32 points: the box tests of all of
// them 32 at a time, the faces that pass queued, and the face tests 32 at a time. Bound by
// the latency of the chains bin, face, box and corners, leaf box from L2. With a thread walking its
// own point's list, ten lanes in 32 worked and 2^20 points on a 1024^2 map took 428 us; now 168.
constexpr int INV_T = 128;

struct InverseWarp {
  double2 q[32];                          // the points
  unsigned long long hit[32][MAXHITS];    // per point: rank << 32 | face
  int hits[32];
  int queue_face[64];
  unsigned char queue_lane[64];
};

__global__ __launch_bounds__(INV_T) void k_inverse(Locator L, double* pts, long P, int first_hit, int* face_out,
                                                   int* hit0_out, int* nhits_out, unsigned long long* missing) {
  __shared__ InverseWarp s_warp[INV_T / 32];
  InverseWarp& W = s_warp[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const long i = (long)blockIdx.x * INV_T + threadIdx.x;
  const int n = L.n, B = L.B;
  double qx = 0., qy = 0.;
  int b = 0, begin = 0, count = 0;
  if (i < P) {
    qx = fmin(fmax(pts[2 * i], 0.), 1.);
    qy = fmin(fmax(pts[2 * i + 1], 0.), 1.);
    if (!(qx == qx)) qx = 0.;  // NaN input: clamp like Eigen's max/min would not; keep it finite
    if (!(qy == qy)) qy = 0.;
    const int bx = (int)fmin(floor(qx * (double)B), (double)(B - 1));
    const int by = (int)fmin(floor(qy * (double)B), (double)(B - 1));
    b = by * B + bx;
    begin = L.starts[b];
    count = L.starts[b + 1] - begin;
  }
  W.q[lane] = make_double2(qx, qy);
  W.hits[lane] = 0;
  __syncwarp();
  auto test = [&](int e) {  // queue entry e
    const int f = W.queue_face[e], l = W.queue_lane[e];
    const double2 q = W.q[l];
    Quad p;
    int vid[4];
    load_quad(L.xy, n, f, p, vid);
    const double4 lb = L.lbox[f];
    if (!(lb.x <= q.x && lb.y <= q.y && q.x <= lb.z && q.y <= lb.w)) return;  // AlignedBox::contains
    if (!hits_face(q.x, q.y, p)) return;
    const int k = atomicAdd(&W.hits[l], 1);
    if (k < MAXHITS) W.hit[l][k] = (unsigned long long)(unsigned)L.rank[f] << 32 | (unsigned)f;
  };
  int queued = 0;
  for (int left = count; __any_sync(0xffffffffu, left > 0);) {  // once but for lists of 2^26 faces
    const int part = pool_part(left);
    int upto = part;  // inclusive prefix over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += u;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31), shift = begin + (count - left) - (upto - part);
    left -= part;
    for (int base = 0; base < total; base += 32) {
      const int item = base + lane;
      int l = 0;  // the point the item belongs to: the first lane with upto > item
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(0xffffffffu, upto, l + o - 1) <= item) l += o;
      l = min(l, 31);
      const int k = item + __shfl_sync(0xffffffffu, shift, l);
      bool pass = false;
      int f = 0;
      if (item < total) {
        f = L.faces[k];
        const double4 bb = L.boxes[f];
        const double2 q = W.q[l];
        pass = !(q.x < bb.x || q.x > bb.z || q.y < bb.y || q.y > bb.w);
      }
      const unsigned m = __ballot_sync(0xffffffffu, pass);
      if (pass) {
        const int e = queued + __popc(m & ((1u << lane) - 1));
        W.queue_face[e] = f;
        W.queue_lane[e] = (unsigned char)l;
      }
      queued += __popc(m);
      __syncwarp();
      if (queued >= 32) {
        queued -= 32;
        test(queued + lane);
        __syncwarp();
      }
    }
  }
  if (lane < queued) test(lane);
  __syncwarp();
  if (i >= P) return;
  const int nh = W.hits[lane];
  if (nhits_out) nhits_out[i] = nh;
  if (nh == 0) {
    if (hit0_out) hit0_out[i] = -1;
    pts[2 * i] = NAN;
    pts[2 * i + 1] = NAN;
    if (face_out) face_out[i] = -1;
    atomicAdd(missing, 1ull);
    return;
  }
  int first, f;
  if (nh <= MAXHITS) {
    for (int k = 1; k < nh; ++k) {  // by rank
      const unsigned long long h = W.hit[lane][k];
      int j = k;
      for (; j > 0 && W.hit[lane][j - 1] > h; --j) W.hit[lane][j] = W.hit[lane][j - 1];
      W.hit[lane][j] = h;
    }
    first = f = (int)(unsigned)W.hit[lane][0];
    if (nh > 1 && !first_hit) {
      double best = L.density[f];
      for (int k = 1; k < nh; ++k) {
        const int g = (int)(unsigned)W.hit[lane][k];
        const double dk = L.density[g];
        if (dk > best) {
          f = g;
          best = dk > best;  // the reference stores the comparison's bool here (transport_map.cpp:82)
        }
      }
    }
  } else {
    f = many_hits(L, b, qx, qy, !first_hit, &first);
  }
  if (hit0_out) hit0_out[i] = first;
  Quad p;
  int vid[4];
  double w[4];
  load_quad(L.xy, n, first, p, vid);
  bilinear_weights(qx, qy, p, w);
  const double dx = 1.0 / (double)n;
  // the corners of face f on the origin grid: (i, j), (i+1, j), (i+1, j+1), (i, j+1)
  const int fi = f / n, fj = f - fi * n;
  double rx = 0, ry = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int vi = fi + (k == 1 || k == 2), vj = fj + (k >= 2);
    double ox = (double)vi * dx, oy = (double)vj * dx;
    if (k == 0) {
      rx = w[0] * ox;
      ry = w[0] * oy;
    } else {
      rx += w[k] * ox;
      ry += w[k] * oy;
    }
  }
  pts[2 * i] = rx;
  pts[2 * i + 1] = ry;
  if (face_out) face_out[i] = f;
}

// ---- rasterization (utils/rasterizer.cpp:36-58, 86-185, 188-302) ----

// A mesh to rasterize: the quads of the (n+1)^2 grid (start == nullptr), or an indexed
// face set of triangles and quads whose face f lists vertices idx[start[f] .. start[f+1])
// in the order the reference's face circulator visits them.
struct MeshRef {
  const double* xy;
  int n;       // grid size (grid meshes only)
  int nf;      // faces
  int nv;      // vertices
  const int* start;
  const int* idx;
};

// Loads face f's corners; returns its valence (3 or 4). Triangles repeat their last
// corner in slot 3, which leaves their bounding box unchanged.
__device__ __forceinline__ int load_face(const MeshRef& m, int f, Quad& p, int vid[4]) {
  if (!m.start) {
    load_quad(m.xy, m.n, f, p, vid);
    return 4;
  }
  const int s = m.start[f];
  const int c = m.start[f + 1] - s;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    vid[k] = m.idx[s + (k < c ? k : c - 1)];
    p.x[k] = m.xy[2 * (size_t)vid[k]];
    p.y[k] = m.xy[2 * (size_t)vid[k] + 1];
  }
  return c;
}

// |area| of a face as rasterize_image takes it (eigen_addons.h:18-23).
__device__ __forceinline__ double face_abs_area(const Quad& p, int c) {
  if (c == 3) return fabs(signed_area3(p.x[0], p.y[0], p.x[1], p.y[1], p.x[2], p.y[2]));
  return fabs(signed_area3(p.x[0], p.y[0], p.x[1], p.y[1], p.x[2], p.y[2]) +
              signed_area3(p.x[0], p.y[0], p.x[2], p.y[2], p.x[3], p.y[3]));
}

// BarycentricTransform (rasterizer.cpp:36-58): T = [s1-s3 | s2-s3], inverted as Eigen
// inverts a 2x2 matrix (adjugate times 1/det), b = T^-1 (q - s3), bary = (b0, b1, 1-b0-b1).
__device__ __forceinline__ void tri_weights(double qx, double qy, const Quad& p, double w[4]) {
  const double m00 = p.x[0] - p.x[2], m10 = p.y[0] - p.y[2];
  const double m01 = p.x[1] - p.x[2], m11 = p.y[1] - p.y[2];
  const double invdet = 1.0 / (m00 * m11 - m10 * m01);
  const double t00 = m11 * invdet, t10 = -m10 * invdet, t01 = -m01 * invdet, t11 = m00 * invdet;
  const double vx = qx - p.x[2], vy = qy - p.y[2];
  const double b0 = t00 * vx + t01 * vy;
  const double b1 = t10 * vx + t11 * vy;
  w[0] = b0;
  w[1] = b1;
  w[2] = 1.0 - b0 - b1;
  w[3] = 0.0;
}

struct FaceBox {
  int x0, x1, y0, y1;  // pixel box [x0,x1) x [y0,y1), as rasterize_face computes it
  __device__ __forceinline__ bool empty() const { return x0 >= x1 || y0 >= y1; }
};

__device__ __forceinline__ FaceBox face_box(const Quad& p, int rows, int cols) {
  double ulx = fmin(fmin(fmin(p.x[0], p.x[1]), p.x[2]), p.x[3]);
  double uly = fmin(fmin(fmin(p.y[0], p.y[1]), p.y[2]), p.y[3]);
  double lrx = fmax(fmax(fmax(p.x[0], p.x[1]), p.x[2]), p.x[3]);
  double lry = fmax(fmax(fmax(p.y[0], p.y[1]), p.y[2]), p.y[3]);
  // Eigen cast<int> truncates toward zero; the boxes are clamped to the image
  double fx0 = ulx * (double)cols, fy0 = uly * (double)rows;
  double fx1 = lrx * (double)cols, fy1 = lry * (double)rows;
  auto trunc_int = [](double v) {
    if (!(v == v)) return 0;
    if (v > 2.0e9) return 2000000000;
    if (v < -2.0e9) return -2000000000;
    return (int)v;
  };
  FaceBox r;
  r.x0 = max(trunc_int(fx0), 0);
  r.y0 = max(trunc_int(fy0), 0);
  r.x1 = min(trunc_int(fx1) + 1, cols);
  r.y1 = min(trunc_int(fy1) + 1, rows);
  return r;
}

// Weights the reference's sequential loop would test at (f, x, y) when its bilinear
// solve fails there (D < 0): its Vector4d is never written, and the optimised build
// then reads the weights of the most recent successful solve. Walk back through the
// loop order -- earlier pixels of face f's box row by row, then earlier quads -- to
// the most recent pixel whose solve succeeds. Bounded; gives zeros (the start state)
// when it runs out, as the sequential emulation does before any solve. Triangles
// never touch that Vector4d and are passed over.
__device__ __noinline__ void stale_weights(const MeshRef& m, int rows, int cols, int f, int x, int y, double w[4]) {
  int steps = 0;
  const int limit = 1 << 22;
  Quad p;
  int vid[4];
  load_face(m, f, p, vid);
  FaceBox r = face_box(p, rows, cols);
  while (steps < limit) {
    // previous pixel in face f's scan
    if (x > r.x0) {
      --x;
    } else if (y > r.y0) {
      --y;
      x = r.x1 - 1;
    } else {
      // last pixel of the previous quad with a non-empty box
      int g = f - 1;
      while (g >= 0 && steps < limit) {
        const int c = load_face(m, g, p, vid);
        r = face_box(p, rows, cols);
        if (!r.empty() && c != 3) break;
        --g;
        ++steps;
      }
      if (g < 0 || steps >= limit) break;
      f = g;
      x = r.x1 - 1;
      y = r.y1 - 1;
    }
    ++steps;
    double qx = ((double)x + 0.5) / (double)cols, qy = ((double)y + 0.5) / (double)rows;
    if (bilinear_weights(qx, qy, p, w)) return;
  }
  w[0] = w[1] = w[2] = w[3] = 0.0;
}

// Weights of face f at the centre of pixel (x, y) as the reference's loop forms them
// (triangles: the barycentric transform; quads: bilinear coordinates, or the stale
// weights where that solve fails). Returns the face's valence; vid gets its corners.
__device__ __forceinline__ int pixel_weights(const MeshRef& m, int rows, int cols, int f, int x, int y, double w[4],
                                             int vid[4]) {
  Quad p;
  const int c = load_face(m, f, p, vid);
  const double qx = ((double)x + 0.5) / (double)cols, qy = ((double)y + 0.5) / (double)rows;
  if (c == 3) {
    tri_weights(qx, qy, p, w);
  } else if (!bilinear_weights(qx, qy, p, w)) {
    stale_weights(m, rows, cols, f, x, y, w);
  }
  return c;
}

// Centres of pixels, (k + 0.5) / count; for a power of two the product with the exact
// reciprocal is the same number.
struct PixelAxis {
  double count, inv;
  bool pow2;
  __device__ __forceinline__ explicit PixelAxis(int n) : count((double)n), inv(1.0 / (double)n), pow2((n & (n - 1)) == 0) {}
  __device__ __forceinline__ double operator()(int k) const {
    const double t = (double)k + 0.5;
    return pow2 ? t * inv : t / count;
  }
};

// Pixel tests whose bilinear solve fails (D < 0), to be decided by stale weights: a walk of any
// length, which k_raster_stale makes with a thread each instead of holding up a warp of the
// owner pass. Tests beyond the list's room are decided on the spot.
struct StaleList {
  PlaceCount* count;  // of the tests that asked for a place, less one: it starts at -1
  uint2* test;        // face, y << 16 | x
  int room;
  // A place of the list for this thread, or one at or beyond `room`.
  __device__ __forceinline__ int place() const {
    return take_place(room, [&] { return atomicAdd(count, 1ull) + 1; });
  }
};

// The owner test: face f (corners p, valence c) records its index at pixel (x, y) when it
// accepts the centre (the weights of pixel_weights lie in [0, 1]).
__device__ __forceinline__ void test_pixel(const MeshRef& m, int rows, int cols, int f, const Quad& p, int c, int x,
                                           int y, double qx, double qy, int* owner, const StaleList& stale) {
  double w[4];
  if (c == 3) {
    tri_weights(qx, qy, p, w);
  } else {
    Bilinear t;
    if (bilinear_terms(qx, qy, p, t)) {
      const int verdict = bilinear_verdict(t);
      if (verdict > 0) atomicMax(&owner[(size_t)y * cols + x], f);
      if (verdict != 0) return;
      bilinear_from_terms(t, w);
    } else {
      const int i = stale.place();
      if (i < stale.room) {
        stale.test[i] = make_uint2((unsigned)f, (unsigned)y << 16 | (unsigned)x);
        return;
      }
      stale_weights(m, rows, cols, f, x, y, w);
    }
  }
  if (weights_inside(w)) atomicMax(&owner[(size_t)y * cols + x], f);
}

// Bound by the latency of the walks' divisions and loads, so it takes four blocks per SM: with one
// block it was 31 us for 256^2 jittered quads drawn at 512^2 and 168 for 1024^2 ones at 1024^2, now 18
// and 62 (the calls 148 -> 134 and 365 -> 259 us; a thread per face, walking inside the owner pass,
// 130 and 494). An empty list takes 6.5 us either way.
constexpr int STALE_BLOCKS = 4;
__global__ __launch_bounds__(128) void k_raster_stale(MeshRef m, int rows, int cols, int* owner, StaleList stale) {
  const int total = (int)min(*stale.count + 1, (PlaceCount)stale.room);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint2 e = stale.test[i];
    const int f = (int)e.x, x = (int)(e.y & 0xffffu), y = (int)(e.y >> 16);
    double w[4];
    stale_weights(m, rows, cols, f, x, y, w);
    if (weights_inside(w)) atomicMax(&owner[(size_t)y * cols + x], f);
  }
}

// The owner pass: every pixel centre of a face's box that the face accepts records the
// face index with atomicMax, so each pixel ends with the highest accepting index -- the
// face the reference's sequential loop writes last (rasterizer.cpp:162-236). A lane per
// face, FACES of a warp, forms its box and value. The tests of the boxes of at most SMALL_BOX
// pixels (a mesh drawn near its own resolution has nothing else) are pooled over the warp, 32
// at a time, whatever the boxes' sizes; larger boxes go on two lists (k_raster_listed), so that
// a stretched face -- the inverse maps of sharp densities have some that span much of the
// image -- does not hold one warp. Bound by instruction issue: about
// 90 FP64 and 150 other instructions for each of 4.6 tests per face. With one thread per
// (face, box row) for every face, found by a binary search over 2^20 row counts, and the
// divisions of bilinear_from_terms in every test, the pass took 148 us at 1024^2 beside 30
// of boxes, counting and scanning; now 67 us in all (a raster call 228 -> 105 us; the owner
// part of a 512^2 barycenter image 83 -> 38 us).
constexpr int SMALL_BOX = 32, RF_T = 128;
// Largest box on the first list: a smooth 100^2 mesh drawn at 1400^2 (boxes of 210 to 260 pixels) takes
// 111 us with 256, 95 with 512, 95 with 1024; a folded 40^2 one at 240^2 98, 107 and 106.
constexpr int MID_BOX = 512;
constexpr int BIG_CHUNK = 128;  // pixels of a face of the second list per warp

// Faces with larger boxes: those of up to MID_BOX pixels from the end of `face` backwards, larger
// ones from its start with their numbers of chunks. Counters start at -1.
struct FaceLists {
  int *mid_count, *big_count;
  int* face;
  int* big_chunks;
};

template <int FACES>
__global__ __launch_bounds__(RF_T) void k_raster_faces(MeshRef m, const double* density, float scale, int rows,
                                                       int cols, double* value, int* owner, FaceLists lists,
                                                       StaleList stale) {
  constexpr int SLOTS = RF_T / 32 * FACES;  // faces of the block
  __shared__ Quad s_quad[SLOTS];
  __shared__ int2 s_corner[SLOTS];                      // first pixel of the face's box
  __shared__ unsigned short s_item[SLOTS * SMALL_BOX];  // per test: lane, dx, dy
  const int lane = threadIdx.x & 31, slot0 = (threadIdx.x >> 5) * FACES, f0 = blockIdx.x * SLOTS + slot0, f = f0 + lane;
  const PixelAxis px(cols), py(rows);
  FaceBox b = {0, 0, 0, 0};
  int c = 4, tests = 0;
  if (lane < FACES && f < m.nf) {
    Quad p;
    int vid[4];
    c = load_face(m, f, p, vid);
    const double in_mass = scale * (density ? density[f] : 1.0);
    value[f] = in_mass / face_abs_area(p, c);  // PerFace value: float(1/N) * density / |area|
    b = face_box(p, rows, cols);
    s_corner[slot0 + lane] = make_int2(b.x0, b.y0);
    s_quad[slot0 + lane] = p;
    if (!b.empty()) {
      const int wx = b.x1 - b.x0, wy = b.y1 - b.y0;
      if (wx > SMALL_BOX || wy > SMALL_BOX || wx * wy > SMALL_BOX) {
        if (wx > MID_BOX || wy > MID_BOX || wx * wy > MID_BOX) {
          const int i = atomicAdd(lists.big_count, 1) + 1;
          lists.face[i] = f;
          lists.big_chunks[i] = (int)(((long long)wx * wy + BIG_CHUNK - 1) / BIG_CHUNK);
        } else {
          lists.face[m.nf - 1 - (atomicAdd(lists.mid_count, 1) + 1)] = f;
        }
      } else {
        tests = wx * wy;
      }
    }
  }
  int upto = tests;  // inclusive prefix over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += u;
  }
  const int total = __shfl_sync(0xffffffffu, upto, 31);
  unsigned short* items = s_item + slot0 * SMALL_BOX;
  for (int k = 0, dx = 0, dy = 0, at = upto - tests; k < tests; ++k) {
    items[at + k] = (unsigned short)(lane | dx << 5 | dy << 10);
    if (++dx == b.x1 - b.x0) {
      dx = 0;
      ++dy;
    }
  }
  const unsigned triangles = __ballot_sync(0xffffffffu, c == 3);
  __syncwarp();
  for (int item = lane; item < total; item += 32) {
    const int e = items[item], l = e & 31;
    const int2 at = s_corner[slot0 + l];
    const int x = at.x + (e >> 5 & 31), y = at.y + (e >> 10);
    test_pixel(m, rows, cols, f0 + l, s_quad[slot0 + l], triangles >> l & 1 ? 3 : 4, x, y, px(x), py(y), owner, stale);
  }
}

// Exclusive prefix of the listed faces' chunks, total at [count] (one block; nothing but the
// total when the list is empty).
__global__ __launch_bounds__(1024) void k_big_scan(const int* big_count, const int* big_chunks, long long* start) {
  __shared__ int warp_total[32];
  const int count = *big_count + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long carry = 0;
  for (int c0 = 0; c0 < count; c0 += 1024) {
    const int i = c0 + threadIdx.x, v = i < count ? big_chunks[i] : 0;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    if (lane == 31) warp_total[warp] = s;
    __syncthreads();
    long long before = 0, total = 0;
    for (int w = 0; w < 32; ++w) {
      const int t = warp_total[w];
      if (w < warp) before += t;
      total += t;
    }
    if (i < count) start[i] = carry + before + s - v;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) start[count] = carry;
}

// The listed faces, in units of work: some boxes of the first list -- as many as give every warp a unit,
// at most 32 -- or a chunk of a box of the second (row by row; chunk t belongs to the last entry with
// start <= t). A warp pools a unit's tests, each found in the prefix of the boxes' sizes. With all
// listed boxes in chunks a smooth 200^2 mesh drawn at 1200^2 (boxes of 49 pixels) took 228 us: 84 in
// one block's scan of 40000 entries, 94 in warps that searched them all and had half their lanes
// idle; now 88, 41 of them here (a thread per box row, the form before that, 89). Three blocks
// of 84 registers per SM: four of 64 took 44 us there, two of 106 registers 48.
constexpr int RL_T = 256, RL_BLOCKS = 3;

__global__ __launch_bounds__(RL_T, RL_BLOCKS) void k_raster_listed(MeshRef m, int rows, int cols, FaceLists lists,
                                                        const long long* start, int* owner, StaleList stale) {
  __shared__ Quad s_quad[RL_T];
  __shared__ int4 s_box[RL_T];  // first row's first pixel and width of a face's box, first test in that row
  __shared__ int s_upto[RL_T];  // inclusive prefix of the tests over the warp
  const int lane = threadIdx.x & 31, warp0 = threadIdx.x & ~31;
  const int warps = gridDim.x * (RL_T / 32), warp = blockIdx.x * (RL_T / 32) + (threadIdx.x >> 5);
  const PixelAxis px(cols), py(rows);
  const int mids = *lists.mid_count + 1, bigs = *lists.big_count + 1;
  const int per = max(1, min((mids + warps - 1) / warps, 32)), groups = (mids + per - 1) / per;
  const long long units = groups + start[bigs];
  for (long long t = warp; t < units; t += warps) {
    int f = 0, c = 4, upto = 0;
    auto take = [&](int face, long long k0, int limit) {
      f = face;
      Quad p;
      int vid[4];
      c = load_face(m, f, p, vid);
      const FaceBox b = face_box(p, rows, cols);
      const long long wx = b.x1 - b.x0, left = wx * (b.y1 - b.y0) - k0;
      const int y0 = (int)(k0 / wx);
      s_box[threadIdx.x] = make_int4(b.x0, b.y0 + y0, (int)wx, (int)(k0 - y0 * wx));
      s_quad[threadIdx.x] = p;
      upto = (int)min(left, (long long)limit);
    };
    if (t < groups) {
      const long long e = t * per + lane;
      if (lane < per && e < mids) take(lists.face[m.nf - 1 - e], 0, MID_BOX);
    } else if (lane == 0) {
      int lo = 0, hi = bigs;  // start[lo] <= chunk < start[hi]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (start[mid] <= t - groups) lo = mid; else hi = mid;
      }
      take(lists.face[lo], (t - groups - start[lo]) * BIG_CHUNK, BIG_CHUNK);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += u;
    }
    s_upto[threadIdx.x] = upto;
    const int tests = __shfl_sync(0xffffffffu, upto, 31);
    const unsigned triangles = __ballot_sync(0xffffffffu, c == 3);
    __syncwarp();
    for (int item0 = 0; item0 < tests; item0 += 32) {
      const int item = item0 + lane;
      int l = 0;  // the box the test belongs to: the first lane with a prefix above the item
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (s_upto[warp0 + l + o - 1] <= item) l += o;
      l = min(l, 31);
      const int face = __shfl_sync(0xffffffffu, f, l);
      if (item >= tests) continue;
      const int4 box = s_box[warp0 + l];
      const unsigned k = box.w + item - (l ? s_upto[warp0 + l - 1] : 0), w = box.z, dy = k / w;
      const int x = box.x + (int)(k - dy * w), y = box.y + (int)dy;
      test_pixel(m, rows, cols, face, s_quad[warp0 + l], triangles >> l & 1 ? 3 : 4, x, y, px(x), py(y), owner, stale);
    }
    __syncwarp();
  }
}

// One thread per pixel: the owner's PerFace value, or for PerVertex
// the float interpolation of rasterize_face's loop, which scales vertex 0's value by
// each weight (rasterizer.cpp:123-130, 174-181) and sums in float. A kernel each: with the
// weights' registers the PerFace pass took 18.9 us at 1024^2, 12.1 without.
template <bool VERTEX>
__global__ __launch_bounds__(256) void k_raster_resolve(MeshRef m, int rows, int cols, const double* value,
                                                        const int* owner, const float* vval, double* img) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= cols || y >= rows) return;
  const int f = owner[(size_t)y * cols + x];
  double out = 0.0;
  if (f >= 0) {
    if constexpr (VERTEX) {
      double w[4];
      int vid[4];
      const int c = pixel_weights(m, rows, cols, f, x, y, w, vid);
      const float v0 = vval[vid[0]];
      float acc = 0.0f;
      for (int q = 0; q < c; ++q) acc = acc + v0 * (float)w[q];
      out = (double)acc;
    } else {
      out = value[f];
    }
  }
  img[(size_t)y * cols + x] = out;
}

// PerVertex values (rasterizer.cpp:240-271) on the grid mesh: each vertex sums, in
// float and in face order, 1/|area| over its faces, then takes float(scale) * value /
// (number of faces) with the reference's float and double steps.
__global__ void k_vertex_values_grid(const double* xy, int n, float scale, float* value) {
  const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long V = (long)(n + 1) * (n + 1);
  if (v >= V) return;
  const int vi = (int)(v / (n + 1)), vj = (int)(v % (n + 1));
  float acc = 0.0f;
  double div = 0.0;
  // faces around vertex (vi, vj) in increasing index j + i*n
  const int ci[4] = {vi - 1, vi - 1, vi, vi}, cj[4] = {vj - 1, vj, vj - 1, vj};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (ci[k] < 0 || cj[k] < 0 || ci[k] >= n || cj[k] >= n) continue;
    Quad p;
    int vid[4];
    load_quad(xy, n, cj[k] + ci[k] * n, p, vid);
    acc = (float)((double)acc + 1. / face_abs_area(p, 4));
    div += 1.;
  }
  value[v] = (float)((double)(scale * acc) / div);
}

// Indexed meshes: vertex -> face lists (count, scan, scatter, then each list sorted by
// face index so the float sums run in the reference's face order).
__global__ void k_vf_count(MeshRef m, int* counts) {
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  for (int k = m.start[f]; k < m.start[f + 1]; ++k) atomicAdd(&counts[m.idx[k]], 1);
}

__global__ void k_vf_fill(MeshRef m, const int* vstart, int* cursor, int* vfaces, double* inv_area) {
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  Quad p;
  int vid[4];
  const int c = load_face(m, f, p, vid);
  inv_area[f] = 1. / face_abs_area(p, c);
  for (int k = m.start[f]; k < m.start[f + 1]; ++k) {
    const int v = m.idx[k];
    vfaces[vstart[v] + atomicAdd(&cursor[v], 1)] = f;
  }
}

__global__ void k_vertex_values_mesh(int nv, const int* vstart, int* vfaces, const double* inv_area, float scale,
                                     float* value) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const int s = vstart[v], e = vstart[v + 1];
  for (int a = s + 1; a < e; ++a) {  // insertion sort: lists are short
    int f = vfaces[a], b = a;
    while (b > s && vfaces[b - 1] > f) {
      vfaces[b] = vfaces[b - 1];
      --b;
    }
    vfaces[b] = f;
  }
  float acc = 0.0f;
  double div = 0.0;
  for (int a = s; a < e; ++a) {
    acc = (float)((double)acc + inv_area[vfaces[a]]);
    div += 1.;
  }
  value[v] = (float)((double)(scale * acc) / div);
}

// ---- backward of the grid raster and of the grid inversion (differentiable barycenters) ----

// dL/dA_f per face of a grid mesh from the pixels it owns in the last raster: an owned
// pixel's PerFace value is scale / |A_f| with A_f the signed fan area of face_abs_area,
// so d value / d A_f = -value / A_f.
__global__ void k_raster_area_grad(MeshRef m, int rows, int cols, const double* value, const int* owner,
                                   const double* dL_dpix, double* dL_dA) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  Quad p;
  int vid[4];
  load_face(m, f, p, vid);
  const FaceBox b = face_box(p, rows, cols);
  double acc = 0.0;
  for (int y = b.y0; y < b.y1; ++y)
    for (int x = b.x0; x < b.x1; ++x) {
      const size_t q = (size_t)y * cols + x;
      if (owner[q] == f) acc += dL_dpix[q];
    }
  const double A = signed_area3(p.x[0], p.y[0], p.x[1], p.y[1], p.x[2], p.y[2]) +
                   signed_area3(p.x[0], p.y[0], p.x[2], p.y[2], p.x[3], p.y[3]);
  dL_dA[f] = (acc != 0.0 && A != 0.0) ? -acc * value[f] / A : 0.0;
}

// Per vertex (i, j) of the grid mesh, in a fixed order over the faces around it (face
// (i,j) corner 0, (i-1,j) corner 1, (i-1,j-1) corner 2, (i,j-1) corner 3): with dL_dA,
// sum_f dL/dA_f times the shoelace gradient dA/dx_c = (y_{c+1} - y_{c-1}) / 2,
// dA/dy_c = (x_{c-1} - x_{c+1}) / 2; with cs, the per-face corner sums cs[f][c] as they are.
__global__ void k_grid_vertex_gather(const double* xy, int n, const double* dL_dA, const double2* cs, double* out) {
  const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long V = (long)(n + 1) * (n + 1);
  if (v >= V) return;
  const int i = (int)(v / (n + 1)), j = (int)(v % (n + 1));
  double gx = 0.0, gy = 0.0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int a = i - ((c == 1 || c == 2) ? 1 : 0), b = j - ((c == 2 || c == 3) ? 1 : 0);
    if (a < 0 || b < 0 || a >= n || b >= n) continue;
    const int f = b + a * n;
    if (cs) {
      const double2 t = cs[4 * (size_t)f + c];
      gx += t.x;
      gy += t.y;
    } else {
      const double g = dL_dA[f];
      if (g == 0.0) continue;
      Quad p;
      int vid[4];
      load_quad(xy, n, f, p, vid);
      const int nx = (c + 1) & 3, pv = (c + 3) & 3;
      gx += g * (0.5 * (p.y[nx] - p.y[pv]));
      gy += g * (0.5 * (p.x[pv] - p.x[nx]));
    }
  }
  out[2 * v] = gx;
  out[2 * v + 1] = gy;
}

struct InvGrad {  // per located origin vertex: q = -e J^-T dL/dI and the weights of its first hit
  double qx, qy, w[4];
};

// Origin vertex v = (i * (1/n), j * (1/n)) (mesh_utils.cpp:100-108) located in face
// h = hit0[v] of the forward mesh with weights w of the bilinear coordinates
// (u, v) = (w1 + w2, w2 + w3): its inverse position is I = sum_c w_c O_c with O the
// origin corners (a square of side e, so dI/d(u,v) = e Id), and x = sum_c w_c P_c with P
// the forward corners. Holding x fixed, d(u,v) = -J^-1 sum_c w_c dP_c with
// J = [dx/du | dx/dv], hence dL/dP_c = -e w_c J^-T dL/dI.
__global__ void k_inv_point_grad(const double* fwd, int n, const int* hit0, const double* dL_dI, InvGrad* pg,
                                 int* count) {
  const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long V = (long)(n + 1) * (n + 1);
  if (v >= V) return;
  InvGrad g;
  g.qx = g.qy = 0.0;
  g.w[0] = g.w[1] = g.w[2] = g.w[3] = 0.0;
  const int h = hit0[v];
  if (h >= 0) {
    const double dx = 1.0 / (double)n;
    const double qx = (double)(v / (n + 1)) * dx, qy = (double)(v % (n + 1)) * dx;
    Quad P;
    int vid[4];
    load_quad(fwd, n, h, P, vid);
    double w[4];
    if (bilinear_weights(qx, qy, P, w)) {
      const double u = w[1] + w[2], t = w[2] + w[3];
      const double jux = (1.0 - t) * (P.x[1] - P.x[0]) + t * (P.x[2] - P.x[3]);
      const double juy = (1.0 - t) * (P.y[1] - P.y[0]) + t * (P.y[2] - P.y[3]);
      const double jvx = (1.0 - u) * (P.x[3] - P.x[0]) + u * (P.x[2] - P.x[1]);
      const double jvy = (1.0 - u) * (P.y[3] - P.y[0]) + u * (P.y[2] - P.y[1]);
      const double det = jux * jvy - juy * jvx;
      if (det != 0.0 && isfinite(det)) {
        const double gx = dL_dI[2 * v], gy = dL_dI[2 * v + 1];
        const double s = -dx / det;
        g.qx = s * (jvy * gx - juy * gy);
        g.qy = s * (-jvx * gx + jux * gy);
#pragma unroll
        for (int c = 0; c < 4; ++c) g.w[c] = w[c];
      }
    }
    atomicAdd(&count[h], 1);
  }
  pg[v] = g;
}

__global__ void k_inv_fill(long V, const int* hit0, const int* start, int* cursor, int* list) {
  const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  const int h = hit0[v];
  if (h >= 0) list[start[h] + atomicAdd(&cursor[h], 1)] = (int)v;
}

// Per face: its points in increasing index order (the fill order is arbitrary), then the
// corner sums cs[f][c] = sum_points w_c q in that order.
__global__ void k_inv_face_sums(int N, const int* start, int* list, const InvGrad* pg, double2* cs) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= N) return;
  const int b = start[f], e = start[f + 1];
  for (int a = b + 1; a < e; ++a) {  // insertion sort: lists hold a few points
    const int key = list[a];
    int k = a - 1;
    while (k >= b && list[k] > key) {
      list[k + 1] = list[k];
      --k;
    }
    list[k + 1] = key;
  }
  double2 acc[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) acc[c] = make_double2(0.0, 0.0);
  for (int a = b; a < e; ++a) {
    const InvGrad g = pg[list[a]];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      acc[c].x += g.w[c] * g.qx;
      acc[c].y += g.w[c] * g.qy;
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) cs[4 * (size_t)f + c] = acc[c];
}

// ---- host ----

// The bins are built on the side stream while the BVH order, a chain of small launches that
// leaves most of the GPU idle, runs on the context's (one after the other under the profiler).
static void build_locator(otm_map* m) {
  otm_context* ctx = m->ctx;
  cudaStream_t st = ctx->stream;
  const int n = m->n, N = n * n;
  m->bin_start.reserve(sizeof(int) * (N + 1), st, ctx->pool);
  m->face_box.reserve(sizeof(double4) * N, st, ctx->pool);
  m->bvh_rank.reserve(sizeof(int) * N, st, ctx->pool);
  m->leaf_box.reserve(sizeof(double4) * N, st, ctx->pool);
  // bin counts, scan sums and the lists' length in the context's grow-only scratch
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t b_counts = al(sizeof(int) * N), b_sums = al(sizeof(int) * ((N + SCAN_B - 1) / SCAN_B + 1));
  ctx->locate_scratch.reserve(b_counts + b_sums + sizeof(unsigned long long));
  int* counts = ctx->locate_scratch.as<int>();
  int* sums = reinterpret_cast<int*>(ctx->locate_scratch.as<char>() + b_counts);
  unsigned long long* length = reinterpret_cast<unsigned long long*>(ctx->locate_scratch.as<char>() + b_counts + b_sums);
  const double* xy = m->fwd.as<double>();
  const bool beside = !ctx->prof.on;
  cudaStream_t bs = st;
  if (beside) {
    side_stream(ctx);
    bs = ctx->side;
    OTM_CUDA(cudaEventRecord(ctx->side_ready, st));  // the mesh and the buffers above
    OTM_CUDA(cudaStreamWaitEvent(bs, ctx->side_ready, 0));
  }
  build_bvh_order(ctx, xy, n, m->bvh_rank.as<int>(), m->leaf_box.as<double4>());
  try {
    auto bin = [&](const char* name, auto kernel, auto... args) {
      if (!beside) return launch(ctx, name, kernel, (N + BIN_T - 1) / BIN_T, BIN_T, args...);
      ctx->launches++;
      kernel<<<(N + BIN_T - 1) / BIN_T, BIN_T, 0, bs>>>(args...);
    };
    // n x n bins; fewer while the lists' length is beyond an int (a 512^2 mesh whose faces each cover a
    // sixth of the square has 10^10 entries). The bins only narrow a query's faces down.
    int B = n;
    unsigned long long total = 0;
    for (;; B = (B + 1) / 2) {
      OTM_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * B * B, bs));
      OTM_CUDA(cudaMemsetAsync(length, 0, sizeof(*length), bs));
      bin("bin_count", k_bin_count, xy, n, B, counts, m->face_box.as<double4>(), length);
      exclusive_scan(bs, counts, m->bin_start.as<int>(), sums, B * B);
      OTM_CUDA(cudaMemcpyAsync(&total, length, sizeof(total), cudaMemcpyDeviceToHost, bs));
      OTM_CUDA(cudaStreamSynchronize(bs));
      if (total <= (unsigned long long)INT_MAX) break;
    }
    m->bins = B;
    // filled on bs, read and freed on the context's stream (the two are joined below)
    m->bin_faces.reserve(sizeof(int) * (size_t)(total > 0 ? total : 1), bs, ctx->pool, st);
    OTM_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * B * B, bs));
    bin("bin_fill", k_bin_fill, xy, n, B, (const int*)m->bin_start.as<int>(), counts, m->bin_faces.as<int>());
    OTM_CUDA(cudaGetLastError());
    if (beside) {
      OTM_CUDA(cudaEventRecord(ctx->side_ready, bs));
      OTM_CUDA(cudaStreamWaitEvent(st, ctx->side_ready, 0));
    }
  } catch (...) {
    cudaStreamSynchronize(bs);  // the map's buffers go back on the context's stream
    throw;
  }
  m->located = true;
}

}  // namespace otm

namespace otm {

// Inversion of `count` points (device buffers) through map m, in place; face / hit0 (the
// first hit in the reference's order) / nhits may be null; missing is added to.
void map_inverse_dev(otm_map* m, double* pts, long count, int mode, int* face, int* hit0, int* nhits,
                     unsigned long long* missing) {
  otm_context* ctx = m->ctx;
  if (!m->located) build_locator(m);
  if (count <= 0) return;
  const Locator L{m->fwd.as<double>(),      m->density.as<double>(),   m->n, m->bins, m->bin_start.as<int>(),
                  m->bin_faces.as<int>(),   m->face_box.as<double4>(), m->bvh_rank.as<int>(), m->leaf_box.as<double4>()};
  launch(ctx, "inverse", k_inverse, (unsigned)((count + INV_T - 1) / INV_T), INV_T, L, pts, count, mode == OTM_INV_FIRST ? 1 : 0, face, hit0, nhits,
         missing);
  OTM_CUDA(cudaGetLastError());
}

void raster_grid_backward(otm_context* ctx, int n, const double* xy, int rows, int cols, const double* dL_dpix,
                          double* dL_dxy) {
  const int N = n * n;
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  // the layout raster_mesh leaves in the scratch: face values, then pixel owners
  const char* base = ctx->raster_scratch.as<char>();
  const double* value = reinterpret_cast<const double*>(base);
  const int* owner = reinterpret_cast<const int*>(base + al(sizeof(double) * (size_t)(N > 0 ? N : 1)));
  AsyncBuf dA;
  dA.reserve(sizeof(double) * N, ctx->stream, temp_pool(ctx));
  MeshRef m{xy, n, N, (n + 1) * (n + 1), nullptr, nullptr};
  launch(ctx, "raster_area_grad", k_raster_area_grad, (N + 255) / 256, 256, m, rows, cols, value, owner, dL_dpix,
         dA.as<double>());
  const long V = (long)(n + 1) * (n + 1);
  launch(ctx, "area_vertex_grad", k_grid_vertex_gather, (unsigned)((V + 255) / 256), 256, xy, n,
         (const double*)dA.as<double>(), (const double2*)nullptr, dL_dxy);
  OTM_CUDA(cudaGetLastError());
}

void inverse_grid_backward(otm_context* ctx, int n, const double* fwd, const int* hit0, const double* dL_dI,
                           double* dL_dfwd) {
  cudaStream_t st = ctx->stream;
  const int N = n * n;
  const long V = (long)(n + 1) * (n + 1);
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t b_pg = al(sizeof(InvGrad) * V), b_cnt = al(sizeof(int) * (N + 1)), b_list = al(sizeof(int) * V);
  const size_t b_cs = al(sizeof(double2) * 4 * (size_t)N), b_sums = al(sizeof(int) * ((N + SCAN_B - 1) / SCAN_B + 1));
  AsyncBuf buf;
  buf.reserve(b_pg + 3 * b_cnt + b_list + b_cs + b_sums, st, temp_pool(ctx));
  char* q = buf.as<char>();
  InvGrad* pg = reinterpret_cast<InvGrad*>(q);
  int* count = reinterpret_cast<int*>(q + b_pg);
  int* start = reinterpret_cast<int*>(q + b_pg + b_cnt);
  int* cursor = reinterpret_cast<int*>(q + b_pg + 2 * b_cnt);
  int* list = reinterpret_cast<int*>(q + b_pg + 3 * b_cnt);
  double2* cs = reinterpret_cast<double2*>(q + b_pg + 3 * b_cnt + b_list);
  int* sums = reinterpret_cast<int*>(q + b_pg + 3 * b_cnt + b_list + b_cs);
  OTM_CUDA(cudaMemsetAsync(count, 0, sizeof(int) * N, st));
  OTM_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int) * N, st));
  const unsigned gv = (unsigned)((V + 255) / 256), gf = (unsigned)((N + 255) / 256);
  launch(ctx, "inv_point_grad", k_inv_point_grad, gv, 256, fwd, n, hit0, dL_dI, pg, count);
  exclusive_scan(st, count, start, sums, N);
  launch(ctx, "inv_fill", k_inv_fill, gv, 256, V, hit0, (const int*)start, cursor, list);
  launch(ctx, "inv_face_sums", k_inv_face_sums, gf, 256, N, (const int*)start, list, (const InvGrad*)pg, cs);
  launch(ctx, "inv_vertex_grad", k_grid_vertex_gather, gv, 256, fwd, n, (const double*)nullptr, (const double2*)cs,
         dL_dfwd);
  OTM_CUDA(cudaGetLastError());
}

}  // namespace otm

using namespace otm;

extern "C" int otm_map_create(otm_context* ctx, int n, const double* fwd_xy, const double* density, otm_map** out) {
  return guarded([&] {
    if (!ctx || !fwd_xy || !density || !out) throw BadArg{"otm_map_create: null argument"};
    if (n < 1 || n > 16384) throw BadArg{"otm_map_create: grid size out of range"};
    make_current(ctx);
    auto* m = new otm_map;
    m->ctx = ctx;
    m->n = n;
    try {
      size_t V = (size_t)(n + 1) * (n + 1), N = (size_t)n * n;
      m->fwd.reserve(sizeof(double) * 2 * V, ctx->stream, ctx->pool);
      m->density.reserve(sizeof(double) * N, ctx->stream, ctx->pool);
      copy_in(ctx, m->fwd.p, fwd_xy, sizeof(double) * 2 * V);
      copy_in(ctx, m->density.p, density, sizeof(double) * N);
      OTM_CUDA(cudaStreamSynchronize(ctx->stream));
    } catch (...) {
      delete m;
      throw;
    }
    *out = m;
    return (int)OTM_OK;
  });
}

extern "C" int otm_map_destroy(otm_map* m) {
  if (!m) return OTM_OK;
  cudaSetDevice(m->ctx->device);
  delete m;  // the buffers are freed in stream order, after the work queued on them
  return OTM_OK;
}

extern "C" int otm_map_init_inverse(otm_map* m) {
  return guarded([&] {
    if (!m) throw BadArg{"otm_map_init_inverse: null map"};
    make_current(m->ctx);
    if (!m->located) build_locator(m);
    return (int)OTM_OK;
  });
}

extern "C" int otm_map_inverse_mode(otm_map* m, double* points, long count, int mode, int* face, int* nhits,
                                   long* missing) {
  return guarded([&] {
    if (!m) throw BadArg{"otm_map_inverse: null map"};
    if (mode != OTM_INV_DENSEST && mode != OTM_INV_FIRST) throw BadArg{"otm_map_inverse: unknown mode"};
    if (count < 0 || (count > 0 && !points)) throw BadArg{"otm_map_inverse: bad points"};
    otm_context* ctx = m->ctx;
    make_current(ctx);
    if (!m->located) build_locator(m);
    cudaStream_t st = ctx->stream;
    if (count == 0) {
      if (missing) *missing = 0;
      return (int)OTM_OK;
    }
    // device staging: points (2P doubles), faces, nhits, missing counter
    bool pdev = is_device_ptr(points), fdev = face && is_device_ptr(face), hdev = nhits && is_device_ptr(nhits);
    size_t bp = pdev ? 0 : sizeof(double) * 2 * (size_t)count;
    size_t bf = (face && !fdev) ? sizeof(int) * (size_t)count : 0;
    size_t bh = (nhits && !hdev) ? sizeof(int) * (size_t)count : 0;
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    m->scratch.reserve(al(bp) + al(bf) + al(bh) + 256, ctx->stream, ctx->pool);
    char* base = m->scratch.as<char>();
    double* dp = pdev ? points : reinterpret_cast<double*>(base);
    int* df = face ? (fdev ? face : reinterpret_cast<int*>(base + al(bp))) : nullptr;
    int* dh = nhits ? (hdev ? nhits : reinterpret_cast<int*>(base + al(bp) + al(bf))) : nullptr;
    unsigned long long* dm = reinterpret_cast<unsigned long long*>(base + al(bp) + al(bf) + al(bh));
    if (!pdev) copy_in(ctx, dp, points, bp);
    OTM_CUDA(cudaMemsetAsync(dm, 0, sizeof(unsigned long long), st));
    map_inverse_dev(m, dp, (long)count, mode, df, nullptr, dh, dm);
    if (!pdev) copy_out(ctx, points, dp, bp);
    if (face && !fdev) copy_out(ctx, face, df, bf);
    if (nhits && !hdev) copy_out(ctx, nhits, dh, bh);
    unsigned long long miss = 0;
    OTM_CUDA(cudaMemcpyAsync(&miss, dm, sizeof(miss), cudaMemcpyDeviceToHost, st));
    OTM_CUDA(cudaStreamSynchronize(st));
    ctx->prof.flush();
    if (missing) *missing = (long)miss;
    return (int)OTM_OK;
  });
}

extern "C" int otm_map_inverse(otm_map* m, double* points, long count, int* face, int* nhits, long* missing) {
  return otm_map_inverse_mode(m, points, count, OTM_INV_DENSEST, face, nhits, missing);
}

// ---- stochastic splatting (utils/stochastic_rasterizer.cpp:19-88) ----

// Counter-based uniform doubles in [0, 1): the splitmix64 output function (Steele, Lea
// and Flood, "Fast splittable pseudorandom number generators", OOPSLA 2014) applied to
// a key made of (seed, face, sample, draw), so any sample can be drawn independently.
__host__ __device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

__device__ __forceinline__ double splat_uniform(unsigned long long face_key, long sample, int draw) {
  const unsigned long long x = mix64(face_key + (unsigned long long)(2 * sample + draw + 1) * 0x9e3779b97f4a7c15ULL);
  return (double)(x >> 11) * 0x1.0p-53;
}

// One warp per face: each of the face's samples is a random point of the face (uniform
// bilinear coordinates for a quad, uniform barycentric ones for a triangle), counted in
// the pixel that contains it. Counts are integers, so the atomic additions are exact and
// the image does not depend on their order.
__global__ void k_splat(MeshRef m, const int* spf, unsigned long long seed, int rows, int cols, double* img) {
  const int lane = threadIdx.x & 31;
  const long f = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (f >= m.nf) return;
  const int ns = spf[f];
  if (ns <= 0) return;
  Quad p;
  int vid[4];
  const int c = load_face(m, (int)f, p, vid);
  const unsigned long long key = mix64(seed ^ mix64((unsigned long long)(f + 1) * 0xd1b54a32d192ed03ULL));
  const double dx = 1. / double(cols), dy = 1. / double(rows);
  for (long s = lane; s < ns; s += 32) {
    double px, py;
    if (c == 3) {
      const double r1 = sqrt(splat_uniform(key, s, 0)), r2 = splat_uniform(key, s, 1);
      const double b0 = 1. - r1, b1 = r1 * (1. - r2), b2 = r1 * r2;
      px = b0 * p.x[0] + b1 * p.x[1] + b2 * p.x[2];
      py = b0 * p.y[0] + b1 * p.y[1] + b2 * p.y[2];
    } else {
      const double u = splat_uniform(key, s, 0), v = splat_uniform(key, s, 1);
      const double w0 = (1. - u) * (1 - v), w1 = (u) * (1 - v), w2 = (u) * (v), w3 = (1. - u) * (v);
      px = w0 * p.x[0] + w1 * p.x[1] + w2 * p.x[2] + w3 * p.x[3];
      py = w0 * p.y[0] + w1 * p.y[1] + w2 * p.y[2] + w3 * p.y[3];
    }
    // stochastic_rasterizer.cpp:71-83: points off the unit square (or not finite) are dropped
    if (!(px >= 0 && py >= 0 && px <= 1 && py <= 1)) continue;
    const int pi = (int)(py / dy), pj = (int)(px / dx);
    if (pi < rows && pj < cols) atomicAdd(&img[(size_t)pi * cols + pj], 1.0);
  }
}

namespace otm {

// Rasterizes mesh m (all pointers on the device) into img (device, rows*cols).
static void raster_mesh(otm_context* ctx, const MeshRef& m, const double* density, int cells, int rows, int cols,
                        int mode, double* img) {
  cudaStream_t st = ctx->stream;
  const int nf = m.nf;
  const size_t pix = (size_t)rows * cols;
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t b_val = al(sizeof(double) * (size_t)(nf > 0 ? nf : 1)), b_own = al(sizeof(int) * (pix + 6));
  const size_t b_vv = al(sizeof(float) * (size_t)(m.nv > 0 ? m.nv : 1));
  const size_t b_list = al(sizeof(int) * (size_t)(nf + 1));
  const size_t b_start = al(sizeof(long long) * (size_t)(nf + 1));
  const size_t b_stale = al(sizeof(uint2) * (size_t)(nf + 1));
  ctx->raster_scratch.reserve(b_val + b_own + b_vv + 2 * b_list + b_start + b_stale);  // grows, kept for the next call
  char* next = ctx->raster_scratch.as<char>();
  auto take = [&](size_t b) {
    char* r = next;
    next += b;
    return r;
  };
  double* value = reinterpret_cast<double*>(take(b_val));
  int* owner = reinterpret_cast<int*>(take(b_own));  // then the counters of the two lists
  float* vval = reinterpret_cast<float*>(take(b_vv));
  int* counters = owner + (pix + 1) / 2 * 2;  // 8-byte aligned
  FaceLists lists{counters, counters + 1, reinterpret_cast<int*>(take(b_list)), reinterpret_cast<int*>(take(b_list))};
  long long* big_start = reinterpret_cast<long long*>(take(b_start));
  StaleList stale{reinterpret_cast<PlaceCount*>(counters + 2), reinterpret_cast<uint2*>(take(b_stale)), nf};
  OTM_CUDA(cudaMemsetAsync(owner, 0xff, sizeof(int) * (pix + 6), st));  // -1: no face, empty lists
  // rasterizer.cpp:193 keeps 1/density.size() in a float
  const float scale = (float)(1. / (double)(density ? cells : nf));
  const int fblocks = nf > 0 ? (nf + 255) / 256 : 1;
  if (nf > 0) {
    auto faces = [&](auto kernel, int per_warp) {
      const int slots = RF_T / 32 * per_warp;
      launch(ctx, "raster_faces", kernel, (nf + slots - 1) / slots, RF_T, m, density, scale, rows, cols, value, owner,
             lists, stale);
    };
    // 32 faces a warp where that gives an SM 16 warps, else fewer: a mesh of few faces has its tests on
    // few warps. Calls with 32, 8, 4 and 1 faces a warp: 40^2 faces folded at 64^2 79, 53, 50 and 47 us,
    // 96^2 smooth at 288^2 47, 36, 34 and 39, 128^2 at 128^2 35, 33, 34 and 42; with 32, 8 and 2 200^2
    // at 600^2 52, 46 and 57, 512^2 at 512^2 49, 66 and 133.
    if (nf >= 512 * ctx->num_sms)
      faces(k_raster_faces<32>, 32);
    else if (nf >= 64 * ctx->num_sms)
      faces(k_raster_faces<8>, 8);
    else if (nf >= 16 * ctx->num_sms)
      faces(k_raster_faces<4>, 4);
    else
      faces(k_raster_faces<1>, 1);
    launch(ctx, "big_scan", k_big_scan, 1, 1024, (const int*)lists.big_count, (const int*)lists.big_chunks, big_start);
    launch(ctx, "raster_listed", k_raster_listed, ctx->num_sms * RL_BLOCKS, RL_T, m, rows, cols, lists,
           (const long long*)big_start, owner, stale);
    launch(ctx, "raster_stale", k_raster_stale, ctx->num_sms * STALE_BLOCKS, 128, m, rows, cols, owner, stale);
  }
  const float* pv = nullptr;
  AsyncBuf vcount, vstart, vsums, vfaces, inv_area;  // indexed PerVertex temporaries
  if (mode == OTM_RIO_PER_VERTEX) {
    const unsigned vb = (unsigned)((m.nv + 255) / 256);
    if (!m.start) {
      launch(ctx, "vertex_values", k_vertex_values_grid, vb, 256, m.xy, m.n, scale, vval);
    } else {
      int nref = 0;
      OTM_CUDA(cudaMemcpyAsync(&nref, m.start + nf, sizeof(int), cudaMemcpyDeviceToHost, st));
      vcount.reserve(sizeof(int) * m.nv, st, temp_pool(ctx));
      vstart.reserve(sizeof(int) * (m.nv + 1), st, temp_pool(ctx));
      vsums.reserve(sizeof(int) * ((m.nv + SCAN_B - 1) / SCAN_B + 1), st, temp_pool(ctx));
      inv_area.reserve(sizeof(double) * (size_t)(nf > 0 ? nf : 1), st, temp_pool(ctx));
      OTM_CUDA(cudaMemsetAsync(vcount.p, 0, sizeof(int) * m.nv, st));
      launch(ctx, "vf_count", k_vf_count, fblocks, 256, m, vcount.as<int>());
      exclusive_scan(st, vcount.as<int>(), vstart.as<int>(), vsums.as<int>(), m.nv);
      OTM_CUDA(cudaStreamSynchronize(st));
      vfaces.reserve(sizeof(int) * (size_t)(nref > 0 ? nref : 1), st, temp_pool(ctx));
      OTM_CUDA(cudaMemsetAsync(vcount.p, 0, sizeof(int) * m.nv, st));
      launch(ctx, "vf_fill", k_vf_fill, fblocks, 256, m, (const int*)vstart.as<int>(), vcount.as<int>(),
             vfaces.as<int>(), inv_area.as<double>());
      launch(ctx, "vertex_values", k_vertex_values_mesh, vb, 256, m.nv, (const int*)vstart.as<int>(),
             vfaces.as<int>(), (const double*)inv_area.as<double>(), scale, vval);
    }
    pv = vval;
  }
  dim3 blk(32, 8), grd((cols + 31) / 32, (rows + 7) / 8);
  launch(ctx, "raster_resolve", pv ? k_raster_resolve<true> : k_raster_resolve<false>, grd, blk, m, rows, cols,
         (const double*)value, (const int*)owner, pv, img);
  OTM_CUDA(cudaGetLastError());
}

void raster_grid(otm_context* ctx, int n, const double* xy, const double* density, int rows, int cols, int mode,
                 double* img) {
  MeshRef m{xy, n, n * n, (n + 1) * (n + 1), nullptr, nullptr};
  raster_mesh(ctx, m, density, n * n, rows, cols, mode, img);
}

// Host-side check of an indexed face set (the kernels index with it unchecked).
static void check_faces(int nv, int nf, const int* start, const int* idx) {
  if (start[0] != 0) throw BadArg{"otm_rasterize_mesh: face_start[0] must be 0"};
  for (int f = 0; f < nf; ++f) {
    const int c = start[f + 1] - start[f];
    if (c != 3 && c != 4) throw BadArg{"otm_rasterize_mesh: faces must be triangles or quads"};
  }
  const int total = start[nf];
  for (int k = 0; k < total; ++k)
    if (idx[k] < 0 || idx[k] >= nv) throw BadArg{"otm_rasterize_mesh: vertex index out of range"};
}

}  // namespace otm

extern "C" int otm_rasterize_mode(otm_context* ctx, int n, const double* xy, const double* density, int rows,
                                  int cols, int mode, double* img) {
  return guarded([&] {
    if (!ctx || !xy || !img) throw BadArg{"otm_rasterize: null argument"};
    if (n < 1 || n > 16384 || rows < 1 || cols < 1 || rows > 65536 || cols > 65536)
      throw BadArg{"otm_rasterize: size out of range"};
    if (mode != OTM_RIO_PER_VERTEX && mode != OTM_RIO_PER_FACE) throw BadArg{"otm_rasterize: unknown mode"};
    make_current(ctx);
    cudaStream_t st = ctx->stream;
    const int N = n * n;
    size_t V = (size_t)(n + 1) * (n + 1);
    size_t pix = (size_t)rows * cols;
    AsyncBuf dxy, dden, dimg;
    const double* pxy = xy;
    if (!is_device_ptr(xy)) {
      dxy.reserve(sizeof(double) * 2 * V, st, temp_pool(ctx));
      copy_in(ctx, dxy.p, xy, sizeof(double) * 2 * V);
      pxy = dxy.as<double>();
    }
    const double* pden = density;
    if (density && !is_device_ptr(density)) {
      dden.reserve(sizeof(double) * N, st, temp_pool(ctx));
      copy_in(ctx, dden.p, density, sizeof(double) * N);
      pden = dden.as<double>();
    }
    bool idev = is_device_ptr(img);
    double* pimg = img;
    if (!idev) {
      dimg.reserve(sizeof(double) * pix, st, temp_pool(ctx));
      pimg = dimg.as<double>();
    }
    raster_grid(ctx, n, pxy, pden, rows, cols, mode, pimg);
    if (!idev) copy_out(ctx, img, pimg, sizeof(double) * pix);
    OTM_CUDA(cudaStreamSynchronize(st));
    ctx->prof.flush();
    return (int)OTM_OK;
  });
}

extern "C" int otm_rasterize_faces(otm_context* ctx, int n, const double* xy, int rows, int cols, int* face) {
  return guarded([&] {
    if (!ctx || !xy || !face) throw BadArg{"otm_rasterize_faces: null argument"};
    if (n < 1 || n > 16384 || rows < 1 || cols < 1 || rows > 65536 || cols > 65536)
      throw BadArg{"otm_rasterize_faces: size out of range"};
    make_current(ctx);
    cudaStream_t st = ctx->stream;
    const size_t V2 = 2 * (size_t)(n + 1) * (n + 1), pix = (size_t)rows * cols;
    AsyncBuf buf;
    buf.reserve(sizeof(double) * (V2 + pix) + 256, st, temp_pool(ctx));
    const double* pxy = xy;
    if (!is_device_ptr(xy)) {
      copy_in(ctx, buf.p, xy, sizeof(double) * V2);
      pxy = buf.as<double>();
    }
    double* img = buf.as<double>() + V2;
    raster_grid(ctx, n, pxy, nullptr, rows, cols, OTM_RIO_PER_FACE, img);
    const int N = n * n;
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    const int* owner =
        reinterpret_cast<const int*>(ctx->raster_scratch.as<char>() + al(sizeof(double) * (size_t)N));
    copy_out(ctx, face, owner, sizeof(int) * pix);
    OTM_CUDA(cudaStreamSynchronize(st));
    ctx->prof.flush();
    return (int)OTM_OK;
  });
}

extern "C" int otm_rasterize(otm_context* ctx, int n, const double* xy, const double* density, int rows, int cols,
                             double* img) {
  return otm_rasterize_mode(ctx, n, xy, density, rows, cols, OTM_RIO_PER_FACE, img);
}

extern "C" int otm_rasterize_mesh(otm_context* ctx, int nv, const double* xy, int nf, const int* face_start,
                                  const int* face_vertices, const double* density, int cells, int rows, int cols,
                                  int mode, double* img) {
  return guarded([&] {
    if (!ctx || !img || nv < 0 || nf < 0 || (nv > 0 && !xy) || (nf > 0 && (!face_start || !face_vertices)))
      throw BadArg{"otm_rasterize_mesh: null argument"};
    if (rows < 1 || cols < 1 || rows > 65536 || cols > 65536) throw BadArg{"otm_rasterize_mesh: size out of range"};
    if (mode != OTM_RIO_PER_VERTEX && mode != OTM_RIO_PER_FACE) throw BadArg{"otm_rasterize_mesh: unknown mode"};
    if (density && cells < nf) throw BadArg{"otm_rasterize_mesh: density shorter than the face count"};
    make_current(ctx);
    cudaStream_t st = ctx->stream;
    // host copies of the topology (from host or device memory), validated before any
    // kernel indexes with it
    auto to_host = [&](int* dst, const int* src, size_t count) {
      if (is_device_ptr(src)) {
        OTM_CUDA(cudaMemcpyAsync(dst, src, sizeof(int) * count, cudaMemcpyDeviceToHost, st));
        OTM_CUDA(cudaStreamSynchronize(st));
      } else {
        std::memcpy(dst, src, sizeof(int) * count);
      }
    };
    std::vector<int> hstart((size_t)nf + 1, 0);
    if (nf > 0) to_host(hstart.data(), face_start, (size_t)nf + 1);
    const int total = nf > 0 ? hstart[nf] : 0;
    if (total < 0 || total > 4 * nf) throw BadArg{"otm_rasterize_mesh: bad face_start"};
    std::vector<int> hidx((size_t)(total > 0 ? total : 1));
    if (total > 0) to_host(hidx.data(), face_vertices, (size_t)total);
    if (nf > 0) check_faces(nv, nf, hstart.data(), hidx.data());
    const size_t pix = (size_t)rows * cols;
    AsyncBuf dxy, dden, dimg, dstart, didx;
    const double* pxy = xy;
    if (nv > 0 && !is_device_ptr(xy)) {
      dxy.reserve(sizeof(double) * 2 * (size_t)nv, st, temp_pool(ctx));
      copy_in(ctx, dxy.p, xy, sizeof(double) * 2 * (size_t)nv);
      pxy = dxy.as<double>();
    }
    const double* pden = density;
    if (density && !is_device_ptr(density)) {
      dden.reserve(sizeof(double) * (size_t)cells, st, temp_pool(ctx));
      copy_in(ctx, dden.p, density, sizeof(double) * (size_t)cells);
      pden = dden.as<double>();
    }
    bool idev = is_device_ptr(img);
    double* pimg = img;
    if (!idev) {
      dimg.reserve(sizeof(double) * pix, st, temp_pool(ctx));
      pimg = dimg.as<double>();
    }
    if (nf == 0) {
      OTM_CUDA(cudaMemsetAsync(pimg, 0, sizeof(double) * pix, st));
    } else {
      dstart.reserve(sizeof(int) * ((size_t)nf + 1), st, temp_pool(ctx));
      didx.reserve(sizeof(int) * (size_t)total, st, temp_pool(ctx));
      copy_in(ctx, dstart.p, hstart.data(), sizeof(int) * ((size_t)nf + 1));
      copy_in(ctx, didx.p, hidx.data(), sizeof(int) * (size_t)total);
      MeshRef m{pxy, 0, nf, nv, dstart.as<int>(), didx.as<int>()};
      raster_mesh(ctx, m, pden, cells, rows, cols, mode, pimg);
    }
    if (!idev) copy_out(ctx, img, pimg, sizeof(double) * pix);
    OTM_CUDA(cudaStreamSynchronize(st));
    ctx->prof.flush();
    return (int)OTM_OK;
  });
}

namespace otm {
static void splat(otm_context* ctx, const MeshRef& m, const int* spf_dev, unsigned long long seed, int rows, int cols,
                  double* img_dev) {
  OTM_CUDA(cudaMemsetAsync(img_dev, 0, sizeof(double) * (size_t)rows * cols, ctx->stream));
  if (m.nf == 0) return;
  const unsigned blocks = (unsigned)(((long)m.nf * 32 + 255) / 256);
  launch(ctx, "splat", k_splat, blocks, 256, m, spf_dev, seed, rows, cols, img_dev);
  OTM_CUDA(cudaGetLastError());
}
}  // namespace otm

extern "C" int otm_sample_image(otm_context* ctx, int nv, const double* xy, int nf, const int* face_start,
                                const int* face_vertices, int grid_n, const int* samples_per_face,
                                unsigned long long seed, int rows, int cols, double* img) {
  return guarded([&] {
    if (!ctx || !img || !samples_per_face || nf < 0 || nv < 0 || (nv > 0 && !xy))
      throw BadArg{"otm_sample_image: null argument"};
    if (rows < 1 || cols < 1 || rows > 65536 || cols > 65536) throw BadArg{"otm_sample_image: size out of range"};
    const bool grid = grid_n > 0;
    if (grid && (grid_n > 16384 || nf != grid_n * grid_n || nv != (grid_n + 1) * (grid_n + 1)))
      throw BadArg{"otm_sample_image: grid_n does not match nv and nf"};
    if (!grid && nf > 0 && (!face_start || !face_vertices)) throw BadArg{"otm_sample_image: null face arrays"};
    make_current(ctx);
    cudaStream_t st = ctx->stream;
    std::vector<int> hstart, hidx;
    if (!grid && nf > 0) {
      auto to_host = [&](std::vector<int>& dst, const int* src, size_t count) {
        dst.resize(count);
        if (is_device_ptr(src)) {
          OTM_CUDA(cudaMemcpyAsync(dst.data(), src, sizeof(int) * count, cudaMemcpyDeviceToHost, st));
          OTM_CUDA(cudaStreamSynchronize(st));
        } else {
          std::memcpy(dst.data(), src, sizeof(int) * count);
        }
      };
      to_host(hstart, face_start, (size_t)nf + 1);
      if (hstart[nf] < 0 || hstart[nf] > 4 * nf) throw BadArg{"otm_sample_image: bad face_start"};
      to_host(hidx, face_vertices, (size_t)(hstart[nf] > 0 ? hstart[nf] : 1));
      check_faces(nv, nf, hstart.data(), hidx.data());
    }
    const size_t pix = (size_t)rows * cols;
    AsyncBuf dxy, dspf, dimg, dstart, didx;
    const double* pxy = xy;
    if (nv > 0 && !is_device_ptr(xy)) {
      dxy.reserve(sizeof(double) * 2 * (size_t)nv, st, temp_pool(ctx));
      copy_in(ctx, dxy.p, xy, sizeof(double) * 2 * (size_t)nv);
      pxy = dxy.as<double>();
    }
    const int* pspf = samples_per_face;
    if (nf > 0 && !is_device_ptr(samples_per_face)) {
      dspf.reserve(sizeof(int) * (size_t)nf, st, temp_pool(ctx));
      copy_in(ctx, dspf.p, samples_per_face, sizeof(int) * (size_t)nf);
      pspf = dspf.as<int>();
    }
    const bool idev = is_device_ptr(img);
    double* pimg = img;
    if (!idev) {
      dimg.reserve(sizeof(double) * pix, st, temp_pool(ctx));
      pimg = dimg.as<double>();
    }
    MeshRef m{pxy, grid ? grid_n : 0, nf, nv, nullptr, nullptr};
    if (!grid && nf > 0) {
      dstart.reserve(sizeof(int) * ((size_t)nf + 1), st, temp_pool(ctx));
      didx.reserve(sizeof(int) * hidx.size(), st, temp_pool(ctx));
      copy_in(ctx, dstart.p, hstart.data(), sizeof(int) * hstart.size());
      copy_in(ctx, didx.p, hidx.data(), sizeof(int) * hidx.size());
      m.start = dstart.as<int>();
      m.idx = didx.as<int>();
    }
    splat(ctx, m, pspf, seed, rows, cols, pimg);
    if (!idev) copy_out(ctx, img, pimg, sizeof(double) * pix);
    OTM_CUDA(cudaStreamSynchronize(st));
    ctx->prof.flush();
    return (int)OTM_OK;
  });
}
