// Drop-in transfers on the reference's own array layouts (sm_103a).
//
//   gbg_interpolate             interpolate!            Interpolation.jl:1181-1198, 1007-1052
//   gbg_anterpolate             anterpolate!            Interpolation.jl:1299-1323, 1063-1106
//   gbg_point_traversal_order   point_traversal_order   Interpolation.jl:816-833, 636-684
//   gbg_validate_traversal      PointTraversalOrder     Interpolation.jl:560-589
//
// The gather is one thread per work item, as in the reference, contracting the x
// direction first for every component of the chunk.  The scatter is not the reference's
// atomic push: points are grouped by brick and cell (a counting placement), and a thread per node
// of a brick sums the node's contributions as integers on a scale local to the brick (or, for a
// stencil wider than the grid, in floating point in a fixed order).  No float atomics are used, so
// the scatter is bitwise reproducible and independent of any traversal order, and each node keeps
// the accuracy of an FP64 sum of its own contributions.
#include <algorithm>
#include <string>
#include <type_traits>

#include "gbg_common.cuh"

namespace gbg {
namespace {

constexpr int kThreads = 256;

template <typename T>
struct GridT {
  int64_t nx, ny, nz, npf;
  T ox, oy, oz;  // T.(grid.origin)
  T dx, dy, dz;  // T.(grid.grid_spacing)
  T rx, ry, rz;  // their reciprocals, rounded once
  bool recip;    // locate_recip's quotients are the divisions' (reciprocal_locates)
};

// Spacings whose reciprocal, and the products and residuals of locate_recip with it, stay in the normal range.
// (2^-900 and 2^900: a quotient that matters, between 2^-53 and 2^63, has a residual above 2^-1022 there.)
bool reciprocal_locates(const gbg_grid &g) {
  for (int d = 0; d < 3; ++d)
    if (!(g.spacing[d] >= std::ldexp(1.0, -900) && g.spacing[d] <= std::ldexp(1.0, 900))) return false;
  return true;
}

template <typename T>
GridT<T> make_grid(const gbg_grid &g) {
  GridT<T> r;
  r.nx = g.n[0];
  r.ny = g.n[1];
  r.nz = g.n[2];
  r.npf = g.n[0] * g.n[1] * g.n[2];
  r.ox = T(g.origin[0]);
  r.oy = T(g.origin[1]);
  r.oz = T(g.origin[2]);
  r.dx = T(g.spacing[0]);
  r.dy = T(g.spacing[1]);
  r.dz = T(g.spacing[2]);
  r.rx = T(1) / r.dx;
  r.ry = T(1) / r.dy;
  r.rz = T(1) / r.dz;
  r.recip = reciprocal_locates(g);
  return r;
}

template <typename T>
__device__ __forceinline__ T quiet_nan();
template <>
__device__ __forceinline__ double quiet_nan<double>() { return __longlong_as_double(0x7ff8000000000000LL); }
template <>
__device__ __forceinline__ float quiet_nan<float>() { return __int_as_float(0x7fc00000); }

// mod(c, n), the remainder taken only outside the grid.
__device__ __forceinline__ int64_t wrap_cell(int64_t c, int64_t n) {
  return (uint64_t)c < (uint64_t)n ? c : imod(c, n);
}

// The wrapped node offsets visited along one axis: the reference's wrapped start
// mod(base - n, N) followed by its step rule (Interpolation.jl:1000, 1025-1027).
template <int N2>
__device__ __forceinline__ void walk_offsets(int64_t base, int64_t extent, int64_t stride,
                                             int64_t (&off)[N2]) {
  // (the remainder, not wrap_cell's branch around it: the FP32 gather, waiting for its loads either way,
  // takes 1.61 ms with the branch and 1.48 without, 193 x 160 x 127 x 9, 3e6 points; FP64 the same)
  int64_t node = imod(base - (N2 - 2) / 2, extent);
#pragma unroll
  for (int i = 0; i < N2; ++i) {
    off[i] = node * stride;
    node = (node + 1 == extent) ? 0 : node + 1;
  }
}

__device__ __forceinline__ int64_t step_up(int64_t node, int64_t extent) {
  return (node + 1 == extent) ? 0 : node + 1;
}
__device__ __forceinline__ int64_t step_down(int64_t node, int64_t extent) {
  return node == 0 ? extent - 1 : node - 1;
}

// Locates a point on the three axes; false if any coordinate is non-finite.
template <typename T>
__device__ __forceinline__ bool locate3(const GridT<T> &g, const T *__restrict__ pos, int64_t p,
                                        int64_t m, int64_t (&b)[3], T (&t)[3]) {
  bool ok = locate(__ldg(pos + p), g.ox, g.dx, b[0], t[0]);
  ok &= locate(__ldg(pos + p + m), g.oy, g.dy, b[1], t[1]);
  ok &= locate(__ldg(pos + p + 2 * m), g.oz, g.dz, b[2], t[2]);
  return ok;
}

// _visit (Interpolation.jl:618-619), bounds-checked instead of trusted.
__device__ __forceinline__ bool visit(const int32_t *__restrict__ trav, int64_t w, int64_t m,
                                      int64_t &p, int32_t *status) {
  p = w;
  if (!trav) return true;
  const int64_t v = (int64_t)__ldg(trav + w) - 1;
  if (v < 0 || v >= m) {
    if (status) atomicOr(status, GBG_DEV_TRAVERSAL);
    return false;
  }
  p = v;
  return true;
}

// The reference's _locate with the quotient from the reciprocal of the spacing, r = RN(1/d): q =
// RN(a r), then q + r (a - q d) with the residual exact by a fused multiply-add (Markstein's
// correction).  Before its rounding the corrected quotient is within 2^-104 of a/d, so it is the
// correctly rounded one of _locate unless a/d lies that close to a midpoint.  The floor is taken on
// the bits: GB300 starts an FP64 operation of a warp every 76 clocks per scheduler and these points
// need five instead of about seventeen.  False where floor(Int, q) throws in the reference.
__device__ __forceinline__ bool locate_recip(double x, double o, double d, double r, int64_t &base, double &t) {
  const double a = x - o;
  const double q0 = a * r;
  const double q = fma(fma(-q0, d, a), r, q0);
  const unsigned long long bits = (unsigned long long)__double_as_longlong(q);
  const unsigned long long mag = bits & 0x7fffffffffffffffull;
  const bool ok = mag < 0x43df399b1438a100ull;  // the bits of 9.0e18; NaN and infinities order above
  const int ex = (int)(mag >> 52) - 1023;
  unsigned long long whole = 0ull, cut = 0ull;  // |trunc q|, and the fraction's bits
  unsigned long long tb = bits & 0x8000000000000000ull;
  if (ex >= 0 && ok) {
    const unsigned long long man = (mag & 0xfffffffffffffull) | 0x10000000000000ull;
    const unsigned long long low = ex < 52 ? (1ull << (52 - ex)) - 1ull : 0ull;
    cut = bits & low;
    tb = bits & ~low;
    whole = ex <= 52 ? man >> (52 - ex) : man << (ex - 52);
  } else if (ok) {
    cut = mag;
  }
  double fl = __longlong_as_double((long long)tb);
  base = (long long)whole;
  if (bits >> 63) {
    base = -base;
    if (cut) {
      base -= 1;
      fl -= 1.0;
    }
  }
  if (!ok) base = 0;
  t = q - fl;
  return ok;
}
__device__ __forceinline__ bool locate_recip(float x, float o, float d, float, int64_t &base, float &t) {
  return locate(x, o, d, base, t);  // FP32 divides at full rate
}

template <typename T>
__device__ __forceinline__ bool locate3_recip(const GridT<T> &g, const T *__restrict__ pos, int64_t p, int64_t m,
                                              int64_t (&b)[3], T (&t)[3]) {
  bool ok = locate_recip(__ldg(pos + p), g.ox, g.dx, g.rx, b[0], t[0]);
  ok &= locate_recip(__ldg(pos + p + m), g.oy, g.dy, g.ry, b[1], t[1]);
  ok &= locate_recip(__ldg(pos + p + 2 * m), g.oz, g.dz, g.rz, b[2], t[2]);
  return ok;
}

// ---------------------------------------------------------------- gather

// Horner with fused multiply-adds (one rounding per step instead of the reference's two;
// the weights differ by at most an ulp or so, far inside the transfer's 1e-13 bar).
// M2 > 0: that many powers at compile time; M2 == 0: the scheme's own count.
template <typename T, int N2, int M2>
__device__ __forceinline__ void axis_weights_fma(const SchemeT<T, N2> &s, T t, T (&w)[N2]) {
  if constexpr (M2 > 0) {
#pragma unroll
    for (int q = 0; q < N2; ++q) w[q] = s.c[q + N2 * (M2 - 1)];
#pragma unroll
    for (int p = M2 - 2; p >= 0; --p)
#pragma unroll
      for (int q = 0; q < N2; ++q) w[q] = fma_rn(w[q], t, s.c[q + N2 * p]);
  } else {
#pragma unroll
    for (int q = 0; q < N2; ++q) w[q] = T(0);
#pragma unroll
    for (int p = GBG_MAX_POWERS - 1; p >= 0; --p) {
      if (p < s.m2) {
#pragma unroll
        for (int q = 0; q < N2; ++q) w[q] = fma_rn(w[q], t, s.c[q + N2 * p]);
      }
    }
  }
}

// Compile-time width N2: the (j, i) stencil plane is unrolled, z advances by the reference's running
// walk.  In FP64 this kernel is bound by the FP64 pipe (an operation of a warp every 76 clocks of a
// scheduler), so it counts operations: x is contracted first, then y over the plane, then z -- N2^3 +
// N2^2 + N2 a component and no weight products, 774 at width 6 and 3 components beside 90 for the
// weights and 15 for the locate; the product form (w2[j] w3[k] once per plane row) with a division to
// locate takes 792 + 90 + 50.  256^3 x 3, 1e7 points, width 6: 14.98 ms, 15.75 that way.
template <typename T, int N2, int M2, int CC>
__global__ void __launch_bounds__(kThreads)
    k_gather_plain(GridT<T> g, SchemeT<T, N2> s, int ncomp, const T *__restrict__ field,
                   const T *__restrict__ pos, int64_t m, const int32_t *__restrict__ trav,
                   T *__restrict__ out, int32_t *status) {
  // FP32 (whose bound is its loads) and nine components keep the product form: fewer sums to hold
  constexpr bool kPlane = sizeof(T) == 8 && CC < 9;
  const int64_t nxny = g.nx * g.ny;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < m;
       w += (int64_t)gridDim.x * blockDim.x) {
    int64_t p;
    if (!visit(trav, w, m, p, status)) continue;
    int64_t b[3];
    T t[3];
    const bool ok = locate3_recip(g, pos, p, m, b, t);
    if (!ok && status) atomicOr(status, GBG_DEV_NONFINITE);
    T w1[N2], w2[N2], w3[N2];
    axis_weights_fma<T, N2, M2>(s, t[0], w1);
    axis_weights_fma<T, N2, M2>(s, t[1], w2);
    axis_weights_fma<T, N2, M2>(s, t[2], w3);
    int64_t ix[N2], iy[N2];
    walk_offsets<N2>(b[0], g.nx, 1, ix);
    walk_offsets<N2>(b[1], g.ny, g.nx, iy);
    const int64_t z0 = imod(b[2] - (N2 - 2) / 2, g.nz);
    for (int c0 = 0; c0 < ncomp; c0 += CC) {
      T acc[CC];
#pragma unroll
      for (int c = 0; c < CC; ++c) acc[c] = T(0);
      const T *fc = field + g.npf * c0;
      int64_t node_z = z0;
#pragma unroll 1
      for (int k = 0; k < N2; ++k) {
        T w3k = w3[0];
#pragma unroll
        for (int q = 1; q < N2; ++q)
          if (q == k) w3k = w3[q];
        const T *plane = fc + node_z * nxny;
        [[maybe_unused]] T sy[CC];
#pragma unroll
        for (int j = 0; j < N2; ++j) {
          [[maybe_unused]] const T wyz = kPlane ? T(0) : mul_rn(w2[j], w3k);
          const T *row = plane + iy[j];
          T sx[CC];
#pragma unroll
          for (int c = 0; c < CC; ++c) sx[c] = mul_rn(w1[0], __ldg(row + ix[0] + g.npf * c));
#pragma unroll
          for (int i = 1; i < N2; ++i) {
            const T *f = row + ix[i];
#pragma unroll
            for (int c = 0; c < CC; ++c) sx[c] = fma_rn(w1[i], __ldg(f + g.npf * c), sx[c]);
          }
          if constexpr (kPlane) {
#pragma unroll
            for (int c = 0; c < CC; ++c) sy[c] = j ? fma_rn(w2[j], sx[c], sy[c]) : mul_rn(w2[0], sx[c]);
          } else {
#pragma unroll
            for (int c = 0; c < CC; ++c) acc[c] = fma_rn(wyz, sx[c], acc[c]);
          }
        }
        if constexpr (kPlane) {
#pragma unroll
          for (int c = 0; c < CC; ++c) acc[c] = fma_rn(w3k, sy[c], acc[c]);
        }
        node_z = step_up(node_z, g.nz);
      }
#pragma unroll
      for (int c = 0; c < CC; ++c) out[p + m * (c0 + c)] = ok ? acc[c] : quiet_nan<T>();
    }
  }
}

// Single precision, widths 6 and 8, vectors and tensors: eight lanes per point, a lane per x node of the
// stencil.  A row's nodes are then one contiguous read, where a thread per point has 32 lanes in 32
// places of the cache for every node and component.  Every lane forms its own node's three weights
// and takes the others' y and z weights by shuffles; y is contracted first, then z, and the lane's x
// weight comes last.  96^3, 1.5e6 points, width 6, a thread per point and this, points in no order: 3
// components 1.49 and 0.68 ms, 9 components 9.96 and 2.18; in traversal order 0.79 and 0.62, 2.73 and 1.88.  FP64 keeps a thread per
// point: it is bound by the FP64 pipe, and the weights and sums that the lanes form more than once
// would cost it a third more operations.
template <int N2, int CC>
__global__ void __launch_bounds__(kThreads)
    k_gather_rows(GridT<float> g, SchemeT<float, N2> s, int ncomp, const float *__restrict__ field,
                  const float *__restrict__ pos, int64_t m, const int32_t *__restrict__ trav, float *__restrict__ out,
                  int32_t *status) {
  constexpr int G = 8;
  __shared__ float cs[N2 * GBG_MAX_POWERS];
  stage_coeffs(s, cs);
  const int sub = threadIdx.x & (G - 1), node = min(sub, N2 - 1);
  const unsigned mask = ((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1));
  const int64_t nxny = g.nx * g.ny;
  auto weight = [&](float t) {
    float w = cs[node + N2 * (s.m2 - 1)];
    for (int p = s.m2 - 2; p >= 0; --p) w = fmaf(w, t, cs[node + N2 * p]);
    return w;
  };
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; w < m;
       w += (int64_t)gridDim.x * blockDim.x / G) {
    int64_t p;
    if (!visit(trav, w, m, p, status)) continue;  // the group's lanes visit one point
    int64_t b[3];
    float t[3];
    const bool ok = locate3(g, pos, p, m, b, t);
    if (!ok && status && sub == 0) atomicOr(status, GBG_DEV_NONFINITE);
    const float w1 = weight(t[0]), w2 = weight(t[1]), w3 = weight(t[2]);
    const int64_t x = wrap_cell(b[0] - (N2 - 2) / 2 + node, g.nx);
    int64_t yo[N2];
    int64_t y = wrap_cell(b[1] - (N2 - 2) / 2, g.ny);
    float wy[N2];
#pragma unroll
    for (int j = 0; j < N2; ++j) {
      yo[j] = x + g.nx * y;
      y = step_up(y, g.ny);
      wy[j] = __shfl_sync(mask, w2, j, G);
    }
    const int64_t z0 = wrap_cell(b[2] - (N2 - 2) / 2, g.nz);
    for (int c0 = 0; c0 < ncomp; c0 += CC) {
      float acc[CC];
#pragma unroll
      for (int c = 0; c < CC; ++c) acc[c] = 0.0f;
      int64_t z = z0;
#pragma unroll 1
      for (int k = 0; k < N2; ++k) {
        const float wz = __shfl_sync(mask, w3, k, G);
        const float *plane = field + g.npf * c0 + nxny * z;
        float sy[CC];
#pragma unroll
        for (int j = 0; j < N2; ++j) {
          const float *f = plane + yo[j];
#pragma unroll
          for (int c = 0; c < CC; ++c) {
            const float v = __ldg(f + g.npf * c);
            sy[c] = j ? fmaf(wy[j], v, sy[c]) : wy[0] * v;
          }
        }
#pragma unroll
        for (int c = 0; c < CC; ++c) acc[c] = fmaf(wz, sy[c], acc[c]);
        z = step_up(z, g.nz);
      }
#pragma unroll
      for (int c = 0; c < CC; ++c) {
        float v = sub < N2 ? w1 * acc[c] : 0.0f;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(mask, v, o, G);
        if (c % G == sub) out[p + m * (c0 + c)] = ok ? v : quiet_nan<float>();
      }
    }
  }
}

// The largest |w| of a scheme as a kernel in T evaluates it: the Bernstein bound, and the evaluation's
// roundings (about two a power, each of sum |c| at most).
template <typename T>
double evaluated_weight_bound(const gbg_scheme &sch) {
  return weight_bound(sch, sizeof(T) == 8 ? std::ldexp(1.0, -40) : std::ldexp((double)sch.num_powers, -23));
}

// Fixed-point exponent P of the scatter's weights, w * 2^P: |w| <= L (evaluated_weight_bound)
// <= 1.5 * 2^lb, P = 61 - lb.  Then |w * 2^P| < 1.5 * 2^61 (its high digit of 31 bits fits an int32), a
// product of two less its low 62 bits stays below 2.25 * 2^60 and of three below 3.375 * 2^59.
int fixed_weight_exp(double L) {
  int lb = 0;
  while (1.5 * std::ldexp(1.0, lb) < L && lb < 60) ++lb;
  return 61 - lb;
}

// Run-time width (stencils of 10..16 nodes): nothing unrolled.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    k_gather_plain_dyn(GridT<T> g, SchemeT<T, GBG_MAX_NODES> s, int ncomp,
                       const T *__restrict__ field, const T *__restrict__ pos, int64_t m,
                       const int32_t *__restrict__ trav, T *__restrict__ out, int32_t *status) {
  __shared__ T cs[GBG_MAX_NODES * GBG_MAX_POWERS];
  stage_coeffs(s, cs);
  const int n2 = s.n2, nb = (n2 - 2) / 2;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < m;
       w += (int64_t)gridDim.x * blockDim.x) {
    int64_t p;
    if (!visit(trav, w, m, p, status)) continue;
    int64_t b[3];
    T t[3];
    const bool ok = locate3(g, pos, p, m, b, t);
    if (!ok && status) atomicOr(status, GBG_DEV_NONFINITE);
    T w1[GBG_MAX_NODES], w2[GBG_MAX_NODES], w3[GBG_MAX_NODES];
    axis_weights_dyn(cs, n2, s.m2, t[0], w1);
    axis_weights_dyn(cs, n2, s.m2, t[1], w2);
    axis_weights_dyn(cs, n2, s.m2, t[2], w3);
    const int64_t x0 = imod(b[0] - nb, g.nx), y0 = imod(b[1] - nb, g.ny), z0 = imod(b[2] - nb, g.nz);
#pragma unroll 1
    for (int c = 0; c < ncomp; ++c) {
      T acc = T(0);
      int64_t node_z = z0;
#pragma unroll 1
      for (int k = 0; k < n2; ++k) {
        int64_t node_y = y0;
#pragma unroll 1
        for (int j = 0; j < n2; ++j) {
          const T wyz = mul_rn(w2[j], w3[k]);
          const T *row = field + g.npf * c + g.nx * node_y + g.nx * g.ny * node_z;
          int64_t node_x = x0;
#pragma unroll 1
          for (int i = 0; i < n2; ++i) {
            acc = fma_rn(mul_rn(wyz, w1[i]), __ldg(row + node_x), acc);
            node_x = step_up(node_x, g.nx);
          }
          node_y = step_up(node_y, g.ny);
        }
        node_z = step_up(node_z, g.nz);
      }
      out[p + m * c] = ok ? acc : quiet_nan<T>();
    }
  }
}

// --------------------------------------------------------------- scatter

// The cell (of the base node) each point falls in, and the per-cell point count.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    k_cell_keys(GridT<T> g, const T *__restrict__ pos, int64_t m, uint32_t *__restrict__ keys,
                uint32_t *__restrict__ counts, uint32_t *__restrict__ rank, int32_t *status) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < m;
       p += (int64_t)gridDim.x * blockDim.x) {
    int64_t b[3];
    T t[3];
    const bool ok = locate3(g, pos, p, m, b, t);
    if (!ok && status) atomicOr(status, GBG_DEV_NONFINITE);
    const uint32_t key =
        (uint32_t)(imod(b[0], g.nx) + g.nx * (imod(b[1], g.ny) + g.ny * imod(b[2], g.nz)));
    keys[p] = key;
    rank[p] = atomicAdd(counts + key, 1u);  // the point's rank within its cell, in no order
  }
}

// Per sorted slot: the point's three weight vectors and its alpha-scaled quantities
// (quantity = T(alpha) * q, Interpolation.jl:1085), laid out slot-major for the pull.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    k_scatter_prep(GridT<T> g, SchemeT<T, GBG_MAX_NODES> s, int ncomp, const T *__restrict__ pos,
                   const T *__restrict__ q, int64_t m, const uint32_t *__restrict__ perm, T alpha,
                   T *__restrict__ rec, T *__restrict__ qs) {
  __shared__ T cs[GBG_MAX_NODES * GBG_MAX_POWERS];
  stage_coeffs(s, cs);
  const int n2 = s.n2;
  for (int64_t sl = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; sl < m;
       sl += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = perm[sl];
    int64_t b[3];
    T t[3];
    const bool ok = locate3(g, pos, p, m, b, t);
    T *r = rec + sl * 3 * n2;
#pragma unroll 1
    for (int a = 0; a < 3; ++a) {
      T w[GBG_MAX_NODES];
      axis_weights_dyn(cs, n2, s.m2, t[a], w);
#pragma unroll 1
      for (int i = 0; i < n2; ++i) r[a * n2 + i] = ok ? w[i] : quiet_nan<T>();
    }
#pragma unroll 1
    for (int c = 0; c < ncomp; ++c) qs[sl * ncomp + c] = mul_rn(alpha, q[p + m * c]);
  }
}

// One thread per grid node: sum, in a fixed order, the contributions of the points in
// every cell whose stencil reaches this node, then write alpha*W^T q + beta*field.  Weight
// index i reaches node x from the cell (x + n - i) mod N; for a stencil wider than the
// grid a cell is reached through several weight indices and each contributes, exactly as
// the reference's wrapped walk deposits it several times.
template <typename T, int CC>
__global__ void __launch_bounds__(kThreads)
    k_scatter_pull(GridT<T> g, int n2, int ncomp, const uint32_t *__restrict__ cell_start,
                   const T *__restrict__ rec, const T *__restrict__ qs, T *__restrict__ field,
                   T beta, int beta_zero) {
  const int nb = (n2 - 2) / 2;
  const int64_t nxny = g.nx * g.ny;
  for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < g.npf;
       n += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = n % g.nx;
    const int64_t yz = n / g.nx;
    const int64_t y = yz % g.ny;
    const int64_t z = yz / g.ny;
    const int64_t cx0 = imod(x + nb, g.nx), cy0 = imod(y + nb, g.ny), cz0 = imod(z + nb, g.nz);
    for (int c0 = 0; c0 < ncomp; c0 += CC) {
      T acc[CC];
#pragma unroll
      for (int c = 0; c < CC; ++c) acc[c] = T(0);
      int64_t cz = cz0;
#pragma unroll 1
      for (int k = 0; k < n2; ++k) {
        int64_t cy = cy0;
#pragma unroll 1
        for (int j = 0; j < n2; ++j) {
          const int64_t rowoff = g.nx * cy + nxny * cz;
          int64_t cx = cx0;
#pragma unroll 1
          for (int i = 0; i < n2; ++i) {
            const int64_t cell = cx + rowoff;
            const uint32_t s0 = __ldg(cell_start + cell), s1 = __ldg(cell_start + cell + 1);
#pragma unroll 1
            for (uint32_t sl = s0; sl < s1; ++sl) {
              const T *r = rec + (int64_t)sl * 3 * n2;
              const T wv = mul_rn(mul_rn(__ldg(r + n2 + j), __ldg(r + 2 * n2 + k)), __ldg(r + i));
              const T *qv = qs + (int64_t)sl * ncomp + c0;
#pragma unroll
              for (int c = 0; c < CC; ++c) acc[c] = fma_rn(wv, __ldg(qv + c), acc[c]);
            }
            cx = step_down(cx, g.nx);
          }
          cy = step_down(cy, g.ny);
        }
        cz = step_down(cz, g.nz);
      }
#pragma unroll
      for (int c = 0; c < CC; ++c) {
        T *f = field + n + g.npf * (c0 + c);
        *f = beta_zero ? acc[c] : add_rn(mul_rn(beta, *f), acc[c]);
      }
    }
  }
}

// The same pull for a compile-time width: the cells of a node's x walk are computed once,
// the x loop is unrolled; the order of every sum is the one above (z, y, x cells, then each
// cell's points in slot order), so the results are the same bits.
template <typename T, int N2, int CC>
__global__ void __launch_bounds__(kThreads)
    k_scatter_pull_n(GridT<T> g, int ncomp, const uint32_t *__restrict__ cell_start, const T *__restrict__ rec,
                     const T *__restrict__ qs, T *__restrict__ field, T beta, int beta_zero) {
  constexpr int nb = (N2 - 2) / 2;
  const int64_t nxny = g.nx * g.ny;
  for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < g.npf;
       n += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = n % g.nx;
    const int64_t yz = n / g.nx;
    const int64_t y = yz % g.ny;
    const int64_t z = yz / g.ny;
    int64_t cxs[N2];
    {
      int64_t cx = imod(x + nb, g.nx);
#pragma unroll
      for (int i = 0; i < N2; ++i) {
        cxs[i] = cx;
        cx = step_down(cx, g.nx);
      }
    }
    const int64_t cy0 = imod(y + nb, g.ny), cz0 = imod(z + nb, g.nz);
    for (int c0 = 0; c0 < ncomp; c0 += CC) {
      T acc[CC];
#pragma unroll
      for (int c = 0; c < CC; ++c) acc[c] = T(0);
      int64_t cz = cz0;
#pragma unroll 1
      for (int k = 0; k < N2; ++k) {
        int64_t cy = cy0;
#pragma unroll 1
        for (int j = 0; j < N2; ++j) {
          const int64_t rowoff = g.nx * cy + nxny * cz;
#pragma unroll
          for (int i = 0; i < N2; ++i) {
            const int64_t cell = cxs[i] + rowoff;
            const uint32_t s0 = __ldg(cell_start + cell), s1 = __ldg(cell_start + cell + 1);
#pragma unroll 1
            for (uint32_t sl = s0; sl < s1; ++sl) {
              const T *r = rec + (int64_t)sl * (3 * N2);
              const T wv = mul_rn(mul_rn(__ldg(r + N2 + j), __ldg(r + 2 * N2 + k)), __ldg(r + i));
              const T *qv = qs + (int64_t)sl * ncomp + c0;
#pragma unroll
              for (int c = 0; c < CC; ++c) acc[c] = fma_rn(wv, __ldg(qv + c), acc[c]);
            }
          }
          cy = step_down(cy, g.ny);
        }
        cz = step_down(cz, g.nz);
      }
#pragma unroll
      for (int c = 0; c < CC; ++c) {
        T *f = field + n + g.npf * (c0 + c);
        *f = beta_zero ? acc[c] : add_rn(mul_rn(beta, *f), acc[c]);
      }
    }
  }
}

// ------------------------------------------------------ brick scatter
//
// The default scatter.  Points are grouped by brick and by cell within the brick (a counting
// placement; the order within a cell does not matter, every sum being an integer).  A CTA owns one
// brick of nodes and a thread one of its nodes; the thread visits the points whose stencils reach
// its node and sums their contributions in registers as integers, so the sum does not depend on
// the order.  Each node is written to HBM once, and no atomic touches a node.

struct BrickGeo {
  int32_t b[3];   // nodes (and cells) of a brick
  int64_t nb[3];
  int64_t bvol;
  int32_t eb[3];  // the bricks that the largest quantity exponents are kept for
  int64_t enb[3];
};

// A cell's key: the cells brick by brick, each brick's own x fastest, with no room for what a last brick
// lacks (so that the counts of a grid take its cells' number of words, however thin it is).  Along an axis
// cell c is cell l = c % b of its brick, the first of which is c - l, in an extent of v = min(b, n - c + l)
// cells: the cells before the brick are v2 (v1 (c0 - l0) + (c1 - l1) n0) + (c2 - l2) n0 n1.
__device__ __forceinline__ uint32_t cell_key(uint32_t n0, uint32_t n01, uint32_t f0, uint32_t f1, uint32_t f2, uint32_t l0,
                                             uint32_t l1, uint32_t l2, uint32_t v0, uint32_t v1, uint32_t v2) {
  return f2 * n01 + v2 * (f1 * n0 + v1 * f0) + (l2 * v1 + l1) * v0 + l0;
}

// A quantity as an exact integer mantissa and a binary exponent, from its bits: v = mq 2^(e - 62)
// with 2^61 <= |mq| < 2^62.  The exponent is kept biased so that 0 means zero and kENonFinite (above
// every finite one) a NaN or an infinity.
constexpr int kEBias = 2048;
constexpr int kENonFinite = 4095;

__device__ __forceinline__ int split_quantity(double v, long long &mq) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  const int be = (int)((bits >> 52) & 0x7ffu);
  unsigned long long man = bits & 0xfffffffffffffull;
  mq = 0;
  if (be == 0x7ff) return kENonFinite;
  if (be == 0 && man == 0ull) return 0;
  int e = be - 1022;
  if (be) {
    man = (man | 0x10000000000000ull) << 9;
  } else {  // subnormal: man 2^-1074
    const int up = __clzll((long long)man) - 2;
    man <<= up;
    e = 62 - 1074 - up;
  }
  mq = (bits >> 63) ? -(long long)man : (long long)man;
  return e + kEBias;
}
__device__ __forceinline__ int split_quantity(float v, long long &mq) {
  const uint32_t bits = __float_as_uint(v);
  const int be = (int)((bits >> 23) & 0xffu);
  unsigned long long man = bits & 0x7fffffu;
  mq = 0;
  if (be == 0xff) return kENonFinite;
  if (be == 0 && man == 0ull) return 0;
  int e = be - 126;
  if (be) {
    man = (man | 0x800000ull) << 38;
  } else {  // subnormal: man 2^-149
    const int up = __clzll((long long)man) - 2;
    man <<= up;
    e = 62 - 149 - up;
  }
  mq = (bits >> 31) ? -(long long)man : (long long)man;
  return e + kEBias;
}

// One pass over the points in their own order: the locate, the brick-major key, the cell
// count (the atomic's value is the point's rank in its cell, for the placement), and
// per exponent brick and component the largest exponent of the finite non-zero alpha*q.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    k_brick_keys(GridT<T> g, BrickGeo bg, const T *__restrict__ pos, int64_t m, uint32_t *__restrict__ keys,
                 uint32_t *__restrict__ counts, uint32_t *__restrict__ rank, const T *__restrict__ q, int ncomp,
                 T alpha, uint32_t *__restrict__ ebrick, int32_t *status) {
  const int64_t n[3] = {g.nx, g.ny, g.nz};
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < m;
       p += (int64_t)gridDim.x * blockDim.x) {
    int64_t b[3];
    T t[3];
    const bool ok = g.recip ? locate3_recip(g, pos, p, m, b, t) : locate3(g, pos, p, m, b, t);
    if (!ok) report(status, GBG_DEV_NONFINITE);
    // cells, bricks and keys fit 32 bits (fewer than 2^32 keys)
    uint32_t f[3], l[3], v[3], eb = 0;
#pragma unroll
    for (int d = 2; d >= 0; --d) {
      const uint32_t c = (uint32_t)wrap_cell(b[d], n[d]), bd = (uint32_t)bg.b[d];
      f[d] = c / bd * bd;
      l[d] = c - f[d];
      v[d] = min(bd, (uint32_t)n[d] - f[d]);
      eb = eb * (uint32_t)bg.enb[d] + c / (uint32_t)bg.eb[d];
    }
    const uint32_t key = cell_key((uint32_t)n[0], (uint32_t)n[0] * (uint32_t)n[1], f[0], f[1], f[2], l[0], l[1], l[2],
                                  v[0], v[1], v[2]);
    keys[p] = key;
    rank[p] = atomicAdd(counts + key, 1u);
    for (int c = 0; c < ncomp; ++c) {
      long long mq;
      const int e = split_quantity(mul_rn(alpha, __ldg(q + p + m * c)), mq);  // quantity = T(alpha)*q
      if (e == kENonFinite) {
        report(status, GBG_DEV_NONFINITE);
      } else if (e) {
        // most points find their brick's exponent at least as large already
        uint32_t *at = ebrick + (size_t)eb * ncomp + c;
        if (__ldcg(at) < (uint32_t)e) atomicMax(at, (uint32_t)e);
      }
    }
  }
}

__device__ __forceinline__ long long weight_digits(long long w) {
  return (long long)((unsigned long long)(w >> 31) << 32 | ((unsigned long long)w & 0x7fffffffull));
}

// The point of every slot: a point goes to its cell's first slot plus its rank there.
__global__ void __launch_bounds__(kThreads)
    k_brick_place(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ rank,
                  const uint32_t *__restrict__ starts, int64_t m, uint32_t *__restrict__ perm) {
  // four points a trip: keys and ranks, then the keys' starts, then the stores
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < m; p += 4 * stride) {
    uint32_t k[4], r[4], a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = p + u * stride < m;
      k[u] = in ? __ldg(keys + p + u * stride) : 0u;
      r[u] = in ? __ldg(rank + p + u * stride) : 0u;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = __ldg(starts + k[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (p + u * stride < m) perm[a[u] + r[u]] = (uint32_t)(p + u * stride);
  }
}

// Slot by slot: the point's three axes' stencil weights (the reference's Horner with fused
// multiply-adds, once per point) as fixed point W = w * 2^wexp in two digits, the signed W >> 31 in the
// high half of a word and the 31 bits below it in the low half, and each alpha*q as its mantissa and
// exponent.  Reading the points through the permutation and writing in slot order moves a third less
// than writing the points' own order to its slots (1e7 points at width 4: 2.5 ms so).
template <typename T, int N2, int M2>
__global__ void __launch_bounds__(kThreads)
    k_brick_order(GridT<T> g, SchemeT<T, N2> sch, const T *__restrict__ pos, const uint32_t *__restrict__ perm,
                  int64_t m, int wexp, long long *__restrict__ wts, const T *__restrict__ q, int ncomp, T alpha,
                  long long *__restrict__ qi, int16_t *__restrict__ qe) {
  for (int64_t sl = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; sl < m;
       sl += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = __ldg(perm + sl);
    for (int c = 0; c < ncomp; ++c) {
      long long mq;
      const int e = split_quantity(mul_rn(alpha, __ldg(q + p + m * c)), mq);
      qi[sl * ncomp + c] = mq;
      qe[sl * ncomp + c] = (int16_t)e;
    }
    int64_t b[3];
    T t[3];
    const bool ok = g.recip ? locate3_recip(g, pos, p, m, b, t) : locate3(g, pos, p, m, b, t);
    longlong2 *dst = reinterpret_cast<longlong2 *>(wts + sl * (3 * N2));  // 48, 96, 144 or 192 bytes a point
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      T w[N2];
      axis_weights_fma<T, N2, M2>(sch, ok ? t[d] : T(0), w);
#pragma unroll
      for (int k = 0; k < N2; k += 2)
        dst[(d * N2 + k) / 2] = make_longlong2(ok ? weight_digits(fixed_rn((double)w[k], wexp)) : 0ll,
                                               ok ? weight_digits(fixed_rn((double)w[k + 1], wexp)) : 0ll);
    }
  }
}

// A 192-bit two's-complement integer (s2 its signed top): s += v << sh.
struct Int192 {
  unsigned long long s0, s1, s2;
};
template <int SH>
__device__ __forceinline__ void add_shifted(Int192 &s, long long v) {
  constexpr int b = SH & 63;
  const unsigned long long ext = (unsigned long long)(v >> 63);
  const unsigned long long lo = (unsigned long long)v << b;
  const unsigned long long hi = b ? (unsigned long long)(v >> ((64 - b) & 63)) : ext;
  if constexpr (SH < 64) {
    s.s0 += lo;
    unsigned long long c = s.s0 < lo;
    const unsigned long long h = hi + c;
    c = h < c;
    s.s1 += h;
    c += s.s1 < h;
    s.s2 += ext + c;
  } else {
    s.s1 += lo;
    const unsigned long long c = s.s1 < lo;
    s.s2 += hi + c;
  }
}

// s * 2^e rounded once to a double (ties to even); the rare results outside the normal range are
// left to ldexp.
__device__ __forceinline__ double to_double(Int192 s, int e) {
  const bool neg = (long long)s.s2 < 0;
  if (neg) {
    s.s0 = ~s.s0 + 1ull;
    const unsigned long long c0 = s.s0 == 0ull;
    s.s1 = ~s.s1 + c0;
    s.s2 = ~s.s2 + (unsigned long long)(c0 && s.s1 == 0ull);
  }
  if ((s.s0 | s.s1 | s.s2) == 0ull) return 0.0;
  // the leading bit to bit 191
  if (s.s2 == 0ull) {
    s.s2 = s.s1;
    s.s1 = s.s0;
    s.s0 = 0ull;
    e -= 64;
    if (s.s2 == 0ull) {
      s.s2 = s.s1;
      s.s1 = 0ull;
      e -= 64;
    }
  }
  const int up = __clzll((long long)s.s2);
  if (up) {
    s.s2 = (s.s2 << up) | (s.s1 >> (64 - up));
    s.s1 = (s.s1 << up) | (s.s0 >> (64 - up));
    s.s0 <<= up;
  }
  e += 191 - up;  // what the leading bit weighs
  const unsigned long long top = s.s2 >> 11, rem = s.s2 & 0x7ffull;
  const bool sticky = (s.s1 | s.s0) != 0ull;
  const unsigned long long man =
      top + (unsigned long long)(rem > 0x400ull || (rem == 0x400ull && (sticky || (top & 1ull))));
  const int biased = e + 1023;
  if (biased >= 1 && biased <= 2045) {
    const unsigned long long bits = ((unsigned long long)biased << 52) + (man - 0x10000000000000ull);
    return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
  }
  const double v = ldexp((double)man, e - 52);
  return neg ? -v : v;
}

__device__ __forceinline__ void mad_wide(long long &acc, int a, int b) {
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}

// The product of two fixed-point numbers of two 31-bit digits, h 2^31 + l, less its low 62 bits (to
// two units: the lowest partial product is left out).
__device__ __forceinline__ long long mul_high62(int ah, int al, int bh, int bl) {
  long long mid = 0, top;
  mad_wide(mid, ah, bl);
  mad_wide(mid, al, bh);
  top = mid >> 31;
  mad_wide(top, ah, bh);
  return top;
}

__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ int2 lds64(uint32_t a) {
  int2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}

// Digits of a quantity on its region's scale, ND of kDigit bits to a window.  With 2^e_r above every
// quantity of the region, window 0 holds q / 2^(e_r + 1 - 24 ND) down to its whole part (a signed top
// digit, the others unsigned), window k the next 24 ND k bits below it.  Three digits keep a double
// whole unless it is below 2^-18 of the region's largest, two a float below 2^-23: what is left
// then makes further windows, that are summed apart.  The last bit kept of any quantity is 2^(e_r + 1 - D),
// to which it is rounded first (sum_depth): a region's sums are exact whole numbers of one unit.
constexpr int kDigit = 24, kDepth = 144;

// D for a region of count points: a node's sum of products of node weights (below 2^61) and quantities
// (at most 2^(D - 1) units) has to fit 224 bits.
__device__ __forceinline__ int sum_depth(uint32_t count) { return min(kDepth, 163 - (32 - __clz((int)count))); }

// mq rounded to a multiple of 2^rc (ties up).
__device__ __forceinline__ long long round_quantity(long long mq, int rc) {
  if (rc <= 0) return mq;
  return rc > 62 ? 0ll : ((mq + (1ll << (rc - 1))) >> rc) << rc;
}

template <typename T>
constexpr int kDigits = sizeof(T) == 8 ? 3 : 2;

// The default scatter (deterministic, at least FP64-grade per node).  A CTA takes a brick of nodes (up
// to 8x8x4) and each thread one node.  The brick's region (its cells widened by N2 - 1) is listed with
// per-cell offsets; its points are staged in shared memory (three axes' weights, the quantities'
// digits for CC components), and a thread walks the N2 x N2 rows of cells that feed its node, one
// trip a point: no lane works for a node that the point does not reach.
//
// The arithmetic is integer: an FP64 operation of a warp takes 76 clocks of a scheduler, a 32 x 32 ->
// 64-bit multiply-add 2.  A node's weight is the product of three fixed-point weights w * 2^P (P = 61 -
// lb, |w| <= 1.5 * 2^lb from the scheme's Bernstein bound), each product less its low 62 bits: w1 w2 w3
// * 2^(3P - 124), to a few units of 2^-59 and below 2^61.  Cut in two digits, of 30 bits and the signed
// rest, it meets the quantity's digits in
// 2 ND products, each added by one multiply-add to an accumulator of its own: no shifts
// and no carries per contribution, and no accumulator can overflow over the points of one staging
// (owner_points).  The accumulators
// are folded at their weights into a 192-bit sum; where a region goes in several stagings, these are added, in
// 192 bits a node while no quantity has bits below window 0, then shifted to the unit of the last bit kept, in
// 224 (in 224 from the first staging on, 256^3 x 3 with 1e7 points takes 1% longer, width 8 at a point a cell 3%).
// No bit is dropped between
// the products and the final conversion, so the results depend neither on the order of the points nor on
// how a region is cut.  The only roundings of a node are those of its weights, the quantities' last bit
// (2^-143 of the region's largest, and a bit more for each doubling of a region past half a million points)
// and the final conversion.  A non-finite quantity marks
// every node its stencil reaches, which is written as NaN (the reference's 0 * NaN included).
//
// Bound by issue and by the latency of a brick's phases (at 256^3 x 3 and 6e6 uniform points half of its
// time is the listing and staging, half the trips, at 23 of 32 lanes).  256^3 x 3, 1e7 points with 30% in
// blobs, cubic: 10.5 ms; a warp to a point, which adds to 128-bit sums in shared memory by four dependent
// atomics per contribution, takes 21.4, and three CTAs per SM (80 registers, which spill) 12.0.
constexpr int kOwnerPoints = 508;  // staged points, at most

// The points that one staging may hold for weights up to L in P bits: a node adds each of them once to an
// accumulator between folds.  The node weight, below L^3 2^(3P - 124), has a low digit below 2^30 and a high
// one below h = L^3 2^(3P - 154) + 1, and meets digits below 2^24: no accumulator passes 2^63 in 2^39 / h
// points.  508 for L <= 1.25 * 2^lb (the Lalescu and Lagrange splines, whose weights are at most one or a
// little above), 300 for the largest weights of a caller's own scheme (and never below 256: weights past
// 1.5 * 2^60, which no P holds, must not leave a staging without points).
int owner_points(double L, int wexp) {
  const double h = 1.001 * L * L * L * std::ldexp(1.0, 3 * wexp - 154) + 2.0;
  return (int)std::max(256.0, std::min<double>(kOwnerPoints, std::ldexp(1.0, 39) / h)) & ~3;
}

// Shared words of a staged point: the digits of CC components and the meta word, in 16-byte units of
// an odd count, so that lanes reading neighbouring points meet different banks.
template <int CC, int ND>
constexpr int kDigitWords = 4 * (((CC * ND + 4) / 4) | 1);
template <int N2>
constexpr int kWeightWords = 3 * N2 + 1;  // 64-bit words, odd

// The trips of one lane's node over the points [lo, hi) of the region, staged where point p's digits and weights
// are at digits and weights plus p of their strides: `rows` marks (bit kk * 8 + jj) the rows of cells
// (lx..lx+N2-1, ly+jj, lz+kk) to take.  The loop is the warp's, held together by its vote: a trip takes
// one point of every lane that has one left, and a lane whose row is done moves to its next row within
// the trip.  (Left to itself the compiler makes this a loop over rows around a loop over their points,
// where the lanes wait for the fullest of 32 rows at every row.)  Returns the points' meta words, or-ed.
template <int N2, int CC, int ND>
__device__ __forceinline__ uint32_t owner_walk(unsigned long long rows, const uint32_t *po, int ebase, int E0, int E1,
                                               int xk, uint32_t lo, uint32_t hi, uint32_t digits, uint32_t weights,
                                               long long (&A)[CC][2 * ND]) {
  constexpr int DW = kDigitWords<CC, ND>, WW = kWeightWords<N2>;
  int todo = 0;
  uint32_t marks = 0u, dp = 0, wp = 0, wy = 0, wz = 0;  // the point's digits and weights
  auto next_row = [&]() {
    const int s = __ffsll((long long)rows) - 1;
    rows &= rows - 1ull;
    const int kk = s >> 3, jj = s & 7;
    const int e0 = ebase + (kk * E1 + jj) * E0;
    const uint32_t p0 = max(po[e0], lo);
    todo = (int)(min(po[e0 + N2], hi) - p0);
    dp = digits + p0 * (DW * 4);
    wp = weights + p0 * (WW * 8);
    wy = wp + 8 * (2 * N2 - 1 - jj);
    wz = wp + 8 * (3 * N2 - 1 - kk);
    wp += 8 * xk;
  };
  if (rows) next_row();
#pragma unroll
  for (int c = 0; c < CC; ++c)
#pragma unroll
    for (int j = 0; j < 2 * ND; ++j) A[c][j] = 0ll;
  while (__any_sync(0xffffffffu, todo > 0)) {
    if (todo > 0) {
      uint32_t d[(CC * ND + 4) / 4 * 4];
#pragma unroll
      for (int j = 0; j < (CC * ND + 4) / 4; ++j) {
        const uint4 v = lds128(dp + 16 * j);
        d[4 * j] = v.x;
        d[4 * j + 1] = v.y;
        d[4 * j + 2] = v.z;
        d[4 * j + 3] = v.w;
      }
      const uint32_t meta = d[CC * ND];
      const int2 b = lds64(wy), c = lds64(wz), a = lds64(wp - 8 * (meta & 0xffu));
      const long long u = mul_high62(b.y, b.x, c.y, c.x);
      const long long w = mul_high62((int)(u >> 31), (int)((uint32_t)u & 0x7fffffffu), a.y, a.x);
      marks |= meta;
      const int w0 = (int)((uint32_t)w & 0x3fffffffu), w1 = (int)(w >> 30);
#pragma unroll
      for (int c = 0; c < CC; ++c)
#pragma unroll
        for (int j = 0; j < ND; ++j) {
          mad_wide(A[c][j], w0, (int)d[c * ND + j]);
          mad_wide(A[c][ND + j], w1, (int)d[c * ND + j]);
        }
      dp += DW * 4;
      wp += WW * 8;
      wy += WW * 8;
      wz += WW * 8;
      if (--todo == 0 && rows) next_row();
    }
  }
  return marks;
}

// The accumulators folded at their weights.
template <int ND>
__device__ __forceinline__ Int192 owner_fold(const long long (&A)[2 * ND]) {
  Int192 s{0ull, 0ull, 0ull};
  add_shifted<0>(s, A[0]);
  add_shifted<24>(s, A[1]);
  if constexpr (ND == 3) add_shifted<48>(s, A[2]);
  add_shifted<30>(s, A[ND]);
  add_shifted<54>(s, A[ND + 1]);
  if constexpr (ND == 3) add_shifted<78>(s, A[ND + 2]);
  return s;
}

// v * 2^shift (shift >= 0), its signed top returned.
__device__ __forceinline__ unsigned long long shift_up(Int192 &v, int shift) {
  unsigned long long s3 = (unsigned long long)((long long)v.s2 >> 63);
  if (shift >= 64) {
    s3 = v.s2;
    v.s2 = v.s1;
    v.s1 = v.s0;
    v.s0 = 0ull;
    shift -= 64;
  }
  if (shift > 0) {
    s3 = (s3 << shift) | (v.s2 >> (64 - shift));
    v.s2 = (v.s2 << shift) | (v.s1 >> (64 - shift));
    v.s1 = (v.s1 << shift) | (v.s0 >> (64 - shift));
    v.s0 <<= shift;
  }
  return s3;
}

// A node's 192-bit sum (words at[0], at[plane] and at[2 plane]) += v, and what leaves its top.
__device__ __forceinline__ uint32_t add_sum(unsigned long long *at, int plane, const Int192 &v) {
  const unsigned long long a0 = at[0] + v.s0, c0 = a0 < v.s0;
  const unsigned long long h1 = v.s1 + c0, a1 = at[plane] + h1, c1 = (unsigned long long)(h1 < c0) + (a1 < h1);
  const unsigned long long h2 = v.s2 + c1, a2 = at[2 * plane] + h2;
  at[0] = a0;
  at[plane] = a1;
  at[2 * plane] = a2;
  return (uint32_t)(h2 < c1) + (uint32_t)(a2 < h2);
}

// A 224-bit sum (with the signed top) += v * 2^shift; with shift < 0 the bits that leave are zeros, the
// quantities having been rounded above them.
__device__ __forceinline__ void add_sum(unsigned long long *at, int plane, uint32_t *top, Int192 v, int shift) {
  unsigned long long s3 = (unsigned long long)((long long)v.s2 >> 63);
  if (shift >= 0) {
    s3 = shift_up(v, shift);
  } else {
    const int d = -shift;
    v.s0 = (v.s0 >> d) | (v.s1 << (64 - d));
    v.s1 = (v.s1 >> d) | (v.s2 << (64 - d));
    v.s2 = (v.s2 >> d) | (s3 << (64 - d));
  }
  *top += (uint32_t)s3 + add_sum(at, plane, v);
}

// A 192-bit sum to 224 bits, times 2^shift.
__device__ __forceinline__ void widen_sum(unsigned long long *at, int plane, uint32_t *top, int shift) {
  Int192 v{at[0], at[plane], at[2 * plane]};
  *top = (uint32_t)shift_up(v, shift);
  at[0] = v.s0;
  at[plane] = v.s1;
  at[2 * plane] = v.s2;
}

// Such a sum as 192 bits: whole where it fits, else without its lowest 64 bits (bits -= 64), their
// being there kept in the lowest one for the rounding.
__device__ __forceinline__ Int192 leading_bits(const unsigned long long *at, int plane, uint32_t top, int &bits) {
  Int192 s{at[0], at[plane], at[2 * plane]};
  const long long s3 = (long long)(int)top;
  if (s3 != ((long long)s.s2 >> 63)) {
    s = Int192{s.s1 | (unsigned long long)(s.s0 != 0ull), s.s2, (unsigned long long)s3};
    bits -= 64;
  }
  return s;
}

// Whether a pass's first slots take the place of the cells' own, each moved on by what the pass lists, so that
// the staging has the room of a second table: from width 6, whose regions go in several passes (150 x 111 x 97
// x 3, 0.6 points a cell, width 6, FP32: 3.29 ms, 3.54 with the second table).  Up to width 4 the staging holds
// its most points either way, and the kernel is 3% slower without the table.
template <int N2>
constexpr bool kSlotsMove = N2 >= 6;

// The components from cfrom up to cto, CMAX at a time and the last REST of them by themselves.
template <typename T, int N2, int CMAX, int REST>
__global__ void __launch_bounds__(kThreads, 2)
    k_scatter_owner(GridT<T> g, BrickGeo bg, int ncomp, int cfrom, int cto, int chunk, int chunk1, int sums_bytes,
                    const uint32_t *__restrict__ cell_start, const long long *__restrict__ wts,
                    const long long *__restrict__ qi, const int16_t *__restrict__ qe,
                    const uint32_t *__restrict__ ebrick, int wexp, T *__restrict__ field, T beta, int beta_zero,
                    uint32_t *__restrict__ ticket) {
  constexpr int ND = kDigits<T>, WW = kWeightWords<N2>, half = N2 / 2;
  extern __shared__ __align__(16) unsigned char smem_owner[];
  __shared__ uint32_t warp_tot[32];
  __shared__ uint32_t s_brick[2], s_unit, s_lump;
  const int B0 = bg.b[0], B1 = bg.b[1], B2 = bg.b[2];
  const int E0 = B0 + N2 - 1, E1 = B1 + N2 - 1, E2 = B2 + N2 - 1, ecount = E0 * E1 * E2;
  const int bvol = (int)bg.bvol;
  const size_t per = kDigitWords<(REST > CMAX ? REST : CMAX), ND> * 4 + WW * 8 + 4;
  const size_t staging = max((size_t)sums_bytes + (size_t)chunk * per, (size_t)chunk1 * per);
  uint32_t *off = reinterpret_cast<uint32_t *>(smem_owner + staging);  // ecount + 1 offsets
  uint32_t *r0s = off + ecount + 1;                                    // the cells' first slots
  uint32_t *poff = r0s + ecount;                                       // the same of one pass's share
  uint32_t *pr0 = kSlotsMove<N2> ? r0s : poff + ecount + 1;
  uint32_t *fx = poff + ecount + 1 + (kSlotsMove<N2> ? 0 : ecount);    // per axis the first cell of a cell's brick
  uint32_t *fy = fx + E0, *fz = fy + E1;
  uint32_t *vx = fz + E2, *vy = vx + E0, *vz = vy + E1;                // its place in it, and the brick's extent
  uint32_t *xe = vz + E2, *ye = xe + E0, *ze = ye + E1;                // per-axis exponent brick tables
  uint32_t *marked = ze + E2;                                          // bvol nodes' non-finite marks
  uint32_t *ereg = marked + bvol;                                      // ncomp region scales
  // the nodes' sums of 224 bits: three planes of 64 a component, then the signed tops
  unsigned long long *sums = reinterpret_cast<unsigned long long *>(smem_owner);
  const uint32_t nbricks = (uint32_t)(bg.nb[0] * bg.nb[1] * bg.nb[2]);
  const int n[3] = {(int)g.nx, (int)g.ny, (int)g.nz};
  const uint32_t n0 = (uint32_t)n[0], n01 = n0 * (uint32_t)n[1];
  const int tid = (int)threadIdx.x;
  // a thread's node; a warp's are a block of 4x4x2 in a full brick, so that its lanes' stencils overlap
  // and their point counts differ little
  int nx0 = tid % B0, ny0 = (tid / B0) % B1, nz0 = tid / (B0 * B1);
  if (B0 == 8 && B1 == 8 && B2 == 4) {
    const int warp = tid >> 5, lane = tid & 31;
    nx0 = (lane & 3) + 4 * (warp & 1);
    ny0 = ((lane >> 2) & 3) + 4 * ((warp >> 1) & 1);
    nz0 = (lane >> 4) + 2 * (warp >> 2);
  }
  // a thread's first region cell and the step to its next, as coordinates
  const int ex0 = tid % E0, ey0 = (tid / E0) % E1, ez0 = tid / (E0 * E1);
  const int esx = (int)blockDim.x % E0, esy = ((int)blockDim.x / E0) % E1, esz = (int)blockDim.x / (E0 * E1);
  if (tid == 0) {
    s_brick[0] = atomicAdd(ticket, 1u);
    s_lump = 0u;
  }
  uint32_t passed = 0u;  // passes so far; s_lump: the last one of a region with such cells in one row
  for (int it = 0;; ++it) {
    __syncthreads();
    const uint32_t brick = s_brick[it & 1];
    if (brick >= nbricks) break;
    // the next brick's number arrives while this one is summed
    if (tid == 0) s_brick[(it & 1) ^ 1] = atomicAdd(ticket, 1u);
    const int bc[3] = {(int)(brick % (uint32_t)bg.nb[0]), (int)((brick / (uint32_t)bg.nb[0]) % (uint32_t)bg.nb[1]),
                       (int)(brick / (uint32_t)(bg.nb[0] * bg.nb[1]))};
    for (int t = tid; t < E0 + E1 + E2 + ncomp; t += blockDim.x) {
      if (t >= E0 + E1 + E2) {
        ereg[t - (E0 + E1 + E2)] = 0u;
        continue;
      }
      const int d = t < E0 ? 0 : (t < E0 + E1 ? 1 : 2);
      const int e = t - (d == 0 ? 0 : (d == 1 ? E0 : E0 + E1));
      int c = (bc[d] * bg.b[d] - half + e) % n[d];
      if (c < 0) c += n[d];
      const uint32_t cl = (uint32_t)c % (uint32_t)bg.b[d];
      fx[t] = (uint32_t)c - cl;
      vx[t] = cl | (uint32_t)min(bg.b[d], n[d] - c + (int)cl) << 8;
      // the exponent brick of the cell, marked where the axis enters one
      const uint32_t eb = (uint32_t)c / (uint32_t)bg.eb[d], before = (uint32_t)(c ? c - 1 : n[d] - 1) / (uint32_t)bg.eb[d];
      const uint32_t step = d == 0 ? 1u : (uint32_t)(d == 1 ? bg.enb[0] : bg.enb[0] * bg.enb[1]);
      xe[t] = eb * step | (e == 0 || eb != before ? 0x80000000u : 0u);
    }
    __syncthreads();
    // the cells, and each component's scale: the largest exponent of the exponent bricks that hold a
    // cell of the region
    for (int e = tid, ex = ex0, ey = ey0, ez = ez0; e < ecount; e += blockDim.x) {
      const uint32_t lx = vx[ex], ly = vy[ey], lz = vz[ez];
      const uint32_t key = cell_key(n0, n01, fx[ex], fy[ey], fz[ez], lx & 0xffu, ly & 0xffu, lz & 0xffu, lx >> 8, ly >> 8, lz >> 8);
      const uint32_t a = __ldg(cell_start + key);
      r0s[e] = a;
      off[e] = __ldg(cell_start + key + 1) - a;
      if (xe[ex] & ye[ey] & ze[ez] & 0x80000000u) {
        const size_t eb = (size_t)(xe[ex] & 0x7fffffffu) + (ye[ey] & 0x7fffffffu) + (ze[ez] & 0x7fffffffu);
        for (int c = 0; c < ncomp; ++c) atomicMax(ereg + c, __ldg(ebrick + eb * ncomp + c));
      }
      ex += esx;
      ey += esy;
      ez += esz;
      if (ex >= E0) { ex -= E0; ++ey; }
      if (ey >= E1) { ey -= E1; ++ez; }
    }
    __syncthreads();
    const uint32_t count = block_scan_counts(off, ecount, warp_tot);
    if (tid == 0) off[ecount] = count;
    const int depth = sum_depth(count);
    auto components = [&](auto some, int cc0) {  // `some` components from cc0 on
      constexpr int CC = decltype(some)::value, DW = kDigitWords<CC, ND>;
      uint32_t *tops = reinterpret_cast<uint32_t *>(sums + (size_t)3 * CC * bvol);
      long long A[CC][2 * ND] = {};  // the products' accumulators, [weight digit * ND + quantity digit]
      auto inside = [&](int lx, int ly, int lz) -> bool {
        return bc[0] * B0 + lx < n[0] && bc[1] * B1 + ly < n[1] && bc[2] * B2 + lz < n[2];
      };
      // a node's sum, in units of 2^(e_r + 1 - bits) times the node weight's
      auto write = [&](int c, int lx, int ly, int lz, const Int192 &s, int bits, uint32_t marks) {
        const int e = (int)ereg[cc0 + c];
        T v = e ? (T)to_double(s, (e - kEBias) + 1 - bits + 124 - 3 * wexp) : T(0);
        if ((marks >> c) & 1u) v = quiet_nan<T>();
        T *f = field + (bc[0] * B0 + lx) + g.nx * ((bc[1] * B1 + ly) + g.ny * (bc[2] * B2 + lz)) + g.npf * (cc0 + c);
        *f = beta_zero ? v : add_rn(mul_rn(beta, *f), v);
      };
      // staging room for the whole region at once, or pieces beside the nodes' sums
      bool multi = count > (uint32_t)chunk1, again;
      bool wide = false;  // the sums are in the unit of the last bit kept, not of window 0
      do {
        again = false;
        if (multi) {
          for (int i = tid; i < 3 * CC * bvol; i += blockDim.x) sums[i] = 0ull;
          for (int i = tid; i < bvol; i += blockDim.x) marked[i] = 0u;
        }
        const int P = multi ? chunk : chunk1;
        unsigned char *st = smem_owner + (multi ? sums_bytes : 0);
        uint4 *dig = reinterpret_cast<uint4 *>(st);
        long long *wgt = reinterpret_cast<long long *>(st + (size_t)P * DW * 4);
        uint32_t *pslot = reinterpret_cast<uint32_t *>(wgt + (size_t)P * WW);
        const uint32_t digits = (uint32_t)__cvta_generic_to_shared(dig),
                       weights = (uint32_t)__cvta_generic_to_shared(wgt);
        // A crowded region goes in passes that each take an even share of every cell (the cells'
        // remainders falling in passes of their own), so that every pass has work for every node;
        // a pass above the staging's size goes in pieces.
        const uint32_t even = (uint32_t)(P * 7 / 8), passes = multi ? (count + even - 1) / even : 1u;
        const uint32_t third = count / 3u;
        for (uint32_t pass = 0; pass < passes && !again; ++pass) {
          const uint32_t *po = off, *pr = r0s;
          uint32_t total = count;
          if (multi) {
            __syncthreads();  // the previous pass is listed no longer
            ++passed;
            for (int e = tid; e < ecount; e += blockDim.x) {
              const unsigned long long cells = off[e + 1] - off[e], phase = (uint32_t)e * 2654435761u % passes;
              const unsigned long long at0 = cells * pass + phase, at1 = at0 + cells;
              const bool big = (at1 >> 32) != 0ull;
              const uint32_t a = big ? (uint32_t)(at0 / passes) : (uint32_t)at0 / passes;
              const uint32_t b = big ? (uint32_t)(at1 / passes) : (uint32_t)at1 / passes;
              if constexpr (!kSlotsMove<N2>) pr0[e] = r0s[e] + a;
              poff[e] = b - a;
              // a node's cells in one row hold a third of the points (seen anew in every pass: found once a brick
              // or a region, the trips came out 0.5 to 1% slower at width 4)
              if (off[min(e + N2, ecount)] - off[e] > third) s_lump = passed;
            }
            __syncthreads();
            total = block_scan_counts(poff, ecount, warp_tot);
            if (tid == 0) poff[ecount] = total;
            po = poff;
            pr = pr0;
          }
          // (an empty region takes one empty piece, which writes its nodes)
          for (uint32_t c0 = 0; (c0 < total || (c0 == 0 && !multi)) && !again; c0 += (uint32_t)P) {
            const uint32_t c1 = min(total, c0 + (uint32_t)P);
            const int np = (int)(c1 - c0);
            for (int win = 0; win < kDepth / (kDigit * ND); ++win) {
              __syncthreads();  // the previous points are summed (and the offsets' end is set)
              if (win == 0) {
                for (int e = tid, ex = ex0; e < ecount; e += blockDim.x) {
                  const uint32_t o0 = po[e], lo = max(o0, c0), hi = min(po[e + 1], c1);
                  for (uint32_t t = lo; t < hi; ++t) {
                    pslot[t - c0] = pr[e] + (t - o0);
                    reinterpret_cast<uint32_t *>(dig)[(t - c0) * DW + CC * ND] = (uint32_t)ex;
                  }
                  ex += esx;
                  if (ex >= E0) ex -= E0;
                }
                if (kSlotsMove<N2> && multi && c1 == total)  // (a cell is the same thread's in every loop over them)
                  for (int e = tid; e < ecount; e += blockDim.x) r0s[e] += po[e + 1] - po[e];
                __syncthreads();
              }
              int left = 0;  // some quantity has bits below this window
              for (int t = tid; t < np; t += blockDim.x) {
                const uint32_t slot = pslot[t];
                longlong2 v[3 * N2 / 2];
                if (win == 0) {
#pragma unroll
                  for (int k = 0; k < 3 * N2 / 2; ++k)
                    v[k] = __ldg(reinterpret_cast<const longlong2 *>(wts + (int64_t)slot * (3 * N2)) + k);
                }
                uint32_t w[DW];
                const int64_t q0 = (int64_t)slot * ncomp + cc0;
                uint32_t meta = reinterpret_cast<uint32_t *>(dig)[t * DW + CC * ND] & 0xffu;
#pragma unroll
                for (int k = 0; k < DW; ++k) w[k] = 0u;
#pragma unroll
                for (int c = 0; c < CC; ++c) {
                  const int e = __ldg(qe + q0 + c);
                  if (e == kENonFinite) meta |= 256u << c;
                  const int drop = 63 + (e ? max((int)ereg[cc0 + c] - e, 0) : 0);  // bits of q below 2^(e_r + 1) in mq
                  const int r0 = drop - kDigit * ND * (win + 1);
                  // 0 for a zero or non-finite quantity
                  const long long mq = round_quantity(__ldg(qi + q0 + c), drop - depth);
                  if (win == 0) {
                    // the mantissa's bits from r0 up: 24 (ND - 1) of them, and the signed rest above
                    const int rt = r0 + kDigit * (ND - 1);  // >= 39
                    w[c * ND + ND - 1] = (uint32_t)(mq >> min(rt, 63));
                    const unsigned long long low =
                        r0 >= 0 ? (unsigned long long)(mq >> min(r0, 63)) : (unsigned long long)mq << -r0;
                    w[c * ND] = (uint32_t)low & 0xffffffu;
                    if constexpr (ND == 3) w[c * ND + 1] = (uint32_t)(low >> kDigit) & 0xffffffu;
                  } else {
#pragma unroll
                    for (int j = 0; j < ND; ++j) {
                      const int r = r0 + kDigit * j;
                      w[c * ND + j] =
                          (r >= 0 ? (uint32_t)(mq >> min(r, 63)) : r > -kDigit ? (uint32_t)mq << -r : 0u) & 0xffffffu;
                    }
                  }
                  if (r0 > 0 && (mq & ((1ll << min(r0, 63)) - 1ll)) != 0) left = 1;
                }
                w[CC * ND] = meta;
#pragma unroll
                for (int k = 0; k < DW / 4; ++k)
                  dig[t * (DW / 4) + k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
                if (win == 0) {
#pragma unroll
                  for (int k = 0; k < 3 * N2 / 2; ++k) {
                    wgt[t * WW + 2 * k] = v[k].x;
                    wgt[t * WW + 2 * k + 1] = v[k].y;
                  }
                }
              }
              if (tid == 0) s_unit = 0u;
              left = __syncthreads_or(left);
              if (left && !multi) {  // several windows fold into the sums: start over with room for them
                again = true;
                break;
              }
              if (left && !wide) {
                for (int i = tid; i < CC * bvol; i += blockDim.x)
                  widen_sum(sums + (size_t)3 * (i / bvol) * bvol + i % bvol, bvol, tops + i, depth - kDigit * ND);
                wide = true;
                __syncthreads();
              }
              if (!multi) {
                const bool node = tid < bvol && inside(nx0, ny0, nz0);
                const int ebase = (nz0 * E1 + ny0) * E0 + nx0;
                unsigned long long rows = 0ull;
                if (node) {
#pragma unroll
                  for (int kk = 0; kk < N2; ++kk)
#pragma unroll
                    for (int jj = 0; jj < N2; ++jj) {
                      const int e0 = ebase + (kk * E1 + jj) * E0;
                      if (po[e0] < po[e0 + N2]) rows |= 1ull << (kk * 8 + jj);
                    }
                }
                const uint32_t marks = owner_walk<N2, CC, ND>(rows, po, ebase, E0, E1, nx0 + N2 - 1, c0, c1, digits, weights, A);
                if (node)
#pragma unroll
                  for (int c = 0; c < CC; ++c) write(c, nx0, ny0, nz0, owner_fold<ND>(A[c]), kDigit * ND, marks >> 8);
                break;  // no window is left
              }
              // A crowded region's nodes differ much in their points (at a blob's edge tenfold within a
              // brick), so a node has four lanes, each with a quarter of its rows, and the warps take the
              // 2x2x2 blocks of nodes as they get free.  (A thread a node there kept a fifth of the lanes
              // busy.)  Where one row holds a third of the points, a lane has all rows and a quarter of the
              // staging instead: 64^3 x 1, 1e6 points in one cell, 83 ms, by rows 184; in six along x, 105 and 205.
              const int nu0 = (B0 + 1) / 2, nu1 = (B1 + 1) / 2, units = nu0 * nu1 * ((B2 + 1) / 2);
              const int lane = tid & 31, part = lane & 3;
              while (true) {
                int u = lane == 0 ? (int)atomicAdd(&s_unit, 1u) : 0;
                u = __shfl_sync(0xffffffffu, u, 0);
                if (u >= units) break;
                const int lx = 2 * (u % nu0) + ((lane >> 2) & 1), ly = 2 * ((u / nu0) % nu1) + ((lane >> 3) & 1),
                          lz = 2 * (u / (nu0 * nu1)) + (lane >> 4);
                const bool node = lx < B0 && ly < B1 && lz < B2 && inside(lx, ly, lz);
                const int ebase = (lz * E1 + ly) * E0 + lx;
                unsigned long long rows = 0ull;
                uint32_t lo = c0, hi = c1;
                if (s_lump == passed) {
                  lo += (uint32_t)(np * part / 4);
                  hi = c0 + (uint32_t)(np * (part + 1) / 4);
#pragma unroll 1
                  for (int r = 0; node && r < N2 * N2; ++r) {
                    const int kk = r / N2, jj = r % N2, e0 = ebase + (kk * E1 + jj) * E0;
                    if (max(po[e0], lo) < min(po[e0 + N2], hi)) rows |= 1ull << (kk * 8 + jj);
                  }
                } else if (node) {
#pragma unroll
                  for (int i = 0; i < (N2 * N2 + 3) / 4; ++i) {
                    const int r = 4 * i + part;  // rows r of this lane's quarter, turned so that each has every y
                    const int kk = r / N2, jj = (r + kk) % N2;
                    if (kk < N2) {
                      const int e0 = ebase + (kk * E1 + jj) * E0;
                      if (max(po[e0], c0) < min(po[e0 + N2], c1)) rows |= 1ull << (kk * 8 + jj);
                    }
                  }
                }
                uint32_t marks = owner_walk<N2, CC, ND>(rows, po, ebase, E0, E1, lx + N2 - 1, lo, hi, digits - c0 * (DW * 4), weights - c0 * (WW * 8), A);
                // the four lanes' sums, then a component a lane
                long long mine[2 * ND];
#pragma unroll
                for (int j = 0; j < 2 * ND; ++j) {
#pragma unroll
                  for (int c = 0; c < CC; ++c) {
                    A[c][j] += __shfl_xor_sync(0xffffffffu, A[c][j], 1);
                    A[c][j] += __shfl_xor_sync(0xffffffffu, A[c][j], 2);
                  }
                  mine[j] = A[0][j];
#pragma unroll
                  for (int c = 1; c < CC; ++c)
                    if (part == c) mine[j] = A[c][j];
                }
                marks |= __shfl_xor_sync(0xffffffffu, marks, 1);
                marks |= __shfl_xor_sync(0xffffffffu, marks, 2);
                if (node && part < CC) {
                  const int nl = (lz * B1 + ly) * B0 + lx;
                  if (part == 0 && (marks >> 8)) marked[nl] |= marks >> 8;
                  const Int192 s = owner_fold<ND>(mine);
                  unsigned long long *at = sums + (size_t)3 * part * bvol + nl;
                  if (wide) add_sum(at, bvol, tops + part * bvol + nl, s, depth - kDigit * ND * (win + 1));
                  else add_sum(at, bvol, s);
                }
              }
              if (!left) break;
            }
          }
        }
        if (again) multi = true;
      } while (again);
      if (multi) {
        if constexpr (kSlotsMove<N2>)
          for (int e = tid; e < ecount; e += blockDim.x) r0s[e] -= off[e + 1] - off[e];
        __syncthreads();
        if (tid < bvol && inside(nx0, ny0, nz0)) {
          const int nl = (nz0 * B1 + ny0) * B0 + nx0;
#pragma unroll
          for (int c = 0; c < CC; ++c) {
            const unsigned long long *at = sums + (size_t)3 * c * bvol + nl;
            int bits = wide ? depth : kDigit * ND;
            const Int192 sum = wide ? leading_bits(at, bvol, tops[c * bvol + nl], bits) : Int192{at[0], at[bvol], at[2 * bvol]};
            write(c, nx0, ny0, nz0, sum, bits, marked[nl]);
          }
        }
      }
      __syncthreads();  // the sums and the staging are free for the next components
    };
    int cc0 = cfrom;
    for (; cc0 + CMAX + REST <= cto; cc0 += CMAX) components(std::integral_constant<int, CMAX>{}, cc0);
    if constexpr (REST > 0) components(std::integral_constant<int, REST>{}, cc0);
  }
}

// ------------------------------------------------------- traversal order

// Interpolation.jl:636-642: the comparisons happen in floating point, before any
// conversion, so non-finite and far-away coordinates saturate into a real tile.
template <typename T>
__device__ __forceinline__ int64_t tile_index(T c, T o, T inv, int64_t tiles) {
  const T u = (c - o) * inv;
  if (isnan(u)) return 0;
  if (u <= T(0)) return 0;
  if (u >= T(tiles)) return tiles - 1;
  return (int64_t)u;
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    k_tile_keys(const T *__restrict__ pos, int64_t m, T o0, T o1, T o2, T i0, T i1, T i2,
                int64_t t0, int64_t t1, int64_t t2, uint32_t *__restrict__ keys) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < m;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = tile_index(pos[p], o0, i0, t0);
    const int64_t b = tile_index(pos[p + m], o1, i1, t1);
    const int64_t c = tile_index(pos[p + 2 * m], o2, i2, t2);
    keys[p] = (uint32_t)(a + t0 * (b + t1 * c));  // the reference's key less its 2 offset
  }
}

__global__ void k_to_one_based(const uint32_t *__restrict__ perm, int32_t *__restrict__ order,
                               int64_t m) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x)
    order[i] = (int32_t)perm[i] + 1;
}

// Bound by the bitmap's L2 atomics, one per entry: a bit per point (an eighth of a byte to clear
// and touch instead of a word), while the span and the number of points seen first are kept per
// thread and reach the one global triple by three atomics a block.  Three atomics per entry, all on that
// triple, take 3.9 ms for 3e6 entries; with these the order's whole rebuild, this check and a 9-component
// gather at its points take 1.80 ms.
__global__ void __launch_bounds__(kThreads)
    k_validate(const int32_t *__restrict__ order, int64_t m, uint32_t *__restrict__ seen, unsigned long long *stats) {
  __shared__ int32_t s_lo[kThreads / 32], s_hi[kThreads / 32];
  __shared__ uint32_t s_new[kThreads / 32];
  int32_t lo = INT32_MAX, hi = INT32_MIN;
  uint32_t fresh = 0u;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = __ldg(order + i);
    lo = min(lo, v);
    hi = max(hi, v);
    if (v >= 1 && v <= m) {
      const uint32_t k = (uint32_t)v - 1u, bit = 1u << (k & 31u);
      fresh += (atomicOr(seen + (k >> 5), bit) & bit) ? 0u : 1u;
    }
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  fresh = __reduce_add_sync(0xffffffffu, fresh);
  if ((threadIdx.x & 31) == 0) {
    s_lo[threadIdx.x >> 5] = lo;
    s_hi[threadIdx.x >> 5] = hi;
    s_new[threadIdx.x >> 5] = fresh;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kThreads / 32; ++w) {
      lo = min(lo, s_lo[w]);
      hi = max(hi, s_hi[w]);
      fresh += s_new[w];
    }
    if (lo <= hi) {  // a block without entries has nothing to say
      atomicMin(reinterpret_cast<long long *>(stats), (long long)lo);
      atomicMax(reinterpret_cast<long long *>(stats + 1), (long long)hi);
      atomicAdd(stats + 2, (unsigned long long)fresh);
    }
  }
}

__global__ void k_validate_init(unsigned long long *stats) {
  reinterpret_cast<long long *>(stats)[0] = 0x7fffffffffffffffLL;
  reinterpret_cast<long long *>(stats)[1] = (-0x7fffffffffffffffLL - 1);
  stats[2] = 0ull;
}

__global__ void k_fill_or_scale(void *data, int64_t count, int is_f64, double beta) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (is_f64) {
      double *d = static_cast<double *>(data);
      d[i] = beta == 0.0 ? 0.0 : __dmul_rn(d[i], beta);
    } else {
      float *f = static_cast<float *>(data);
      f[i] = beta == 0.0 ? 0.0f : __fmul_rn(f[i], (float)beta);
    }
  }
}

// ------------------------------------------------------------- dispatch

int chunk_for(int ncomp) { return ncomp % 9 == 0 ? 9 : (ncomp % 3 == 0 ? 3 : 1); }

template <typename T, int N2>
gbg_status launch_gather(const gbg_grid &grid, const gbg_scheme &sch, int ncomp, const void *field,
                         const void *pos, int64_t m, const int32_t *trav, void *out,
                         int32_t *status, cudaStream_t st) {
  const GridT<T> g = make_grid<T>(grid);
  const SchemeT<T, N2> s = make_scheme<T, N2>(sch);
  const int blocks = launch_blocks(m, kThreads);
  const T *f = static_cast<const T *>(field);
  const T *x = static_cast<const T *>(pos);
  T *o = static_cast<T *>(out);
  mark_main_start(st);
  const int chunk = chunk_for(ncomp);
  auto plain = [&](auto cc) {
    constexpr int CC = decltype(cc)::value;
    if (sch.num_powers == N2)  // num_powers == width: compile-time Horner
      k_gather_plain<T, N2, N2, CC><<<blocks, kThreads, 0, st>>>(g, s, ncomp, f, x, m, trav, o, status);
    else
      k_gather_plain<T, N2, 0, CC><<<blocks, kThreads, 0, st>>>(g, s, ncomp, f, x, m, trav, o, status);
  };
  if constexpr (sizeof(T) == 4 && N2 >= 6) {
    // by rows for vectors and tensors; a scalar's row is too little to share (96^3, 1.5e6 points, width 6,
    // in traversal order: 321 us by rows, 280 by a thread per point), nor does width 4 gain in that order
    // (193 x 160 x 127 x 9, 3e6 points: 1.92 ms by rows, 1.47)
    const int groups = launch_blocks(m * 8, kThreads);
    if (chunk == 9)
      k_gather_rows<N2, 9><<<groups, kThreads, 0, st>>>(g, s, ncomp, f, x, m, trav, o, status);
    else if (chunk == 3)
      k_gather_rows<N2, 3><<<groups, kThreads, 0, st>>>(g, s, ncomp, f, x, m, trav, o, status);
    else
      plain(std::integral_constant<int, 1>{});
  } else if (chunk == 9) {
    plain(std::integral_constant<int, 9>{});
  } else if (chunk == 3) {
    plain(std::integral_constant<int, 3>{});
  } else {
    plain(std::integral_constant<int, 1>{});
  }
  note_launch();
  mark_main_stop(st);
  GBG_CUDA_TRY(cudaGetLastError());
  return GBG_OK;
}

template <typename T>
gbg_status dispatch_gather(const gbg_grid &grid, const gbg_scheme &sch, int ncomp, const void *field,
                           const void *pos, int64_t m, const int32_t *trav, void *out,
                           int32_t *status, cudaStream_t st) {
  // the compiled widths' FP64 locate multiplies by the spacing's reciprocal; the run-time width's divides
  switch (sizeof(T) == 4 || reciprocal_locates(grid) ? sch.stencil_width : 0) {
    case 2: return launch_gather<T, 2>(grid, sch, ncomp, field, pos, m, trav, out, status, st);
    case 4: return launch_gather<T, 4>(grid, sch, ncomp, field, pos, m, trav, out, status, st);
    case 6: return launch_gather<T, 6>(grid, sch, ncomp, field, pos, m, trav, out, status, st);
    case 8: return launch_gather<T, 8>(grid, sch, ncomp, field, pos, m, trav, out, status, st);
    default: {
      const GridT<T> g = make_grid<T>(grid);
      const SchemeT<T, GBG_MAX_NODES> s = make_scheme<T, GBG_MAX_NODES>(sch);
      k_gather_plain_dyn<T><<<launch_blocks(m, kThreads), kThreads, 0, st>>>(
          g, s, ncomp, static_cast<const T *>(field), static_cast<const T *>(pos), m, trav,
          static_cast<T *>(out), status);
      note_launch();
      GBG_CUDA_TRY(cudaGetLastError());
      return GBG_OK;
    }
  }
}

// Whether the brick scatter takes so many components.  Its quantities' mantissas and exponents need up to
// twice the workspace of the pull's own copy of them, so the line is a part of the call's contract: a set
// below it has integer sums whatever its type, a set above it the pull's workspace.  It is where the nodes
// of an 8x8x8 brick, clipped to the grid, with 16 bytes a component and the tables of their region fill
// 200 KB: 21 or 22 components on a grid of full bricks, 46 where an axis has 4 nodes.
bool brick_takes(const gbg_grid &g, int ncomp, int n2) {
  if (ncomp <= 20) return true;
  size_t b[3], e[3];
  for (int d = 0; d < 3; ++d) {
    b[d] = (size_t)std::min<int64_t>(8, g.n[d]);
    e[d] = b[d] + n2 - 1;
  }
  // the most stretches of consecutive cells along x in a row of any brick's region (only the first and the
  // last two bricks' regions reach over the grid's end; the others are alike)
  size_t most = 1;
  const int64_t bricks = (g.n[0] + (int64_t)b[0] - 1) / (int64_t)b[0];
  for (int64_t k = 0; k < bricks; k = (k == 3 ? std::max<int64_t>(4, bricks - 3) : k + 1)) {
    size_t stretches = 0;
    for (size_t i = 0; i < e[0]; ++i)
      stretches += i == 0 || imod(k * (int64_t)b[0] - n2 / 2 + (int64_t)i, g.n[0]) % (int64_t)b[0] == 0;
    most = std::max(most, stretches);
  }
  const size_t nodes = b[0] * b[1] * b[2], words = e[0] * e[1] * e[2] + e[1] * e[2] * most + 2 * 1024 + 2 * e[0] + e[1] +
                                                   e[2] + nodes + 1 + most + (size_t)ncomp;
  return nodes * ((size_t)ncomp * 16 + 4) + 4 * words <= 200 * 1024;
}

// Which scatter runs, and its bricks: a thread per node of a brick whenever every axis is at least
// a stencil wide and the components are not too many (brick_takes), else the node pull (which also handles
// a stencil wider than the grid, reached several times per node).
struct ScatterPlan {
  bool bricked = false;
  BrickGeo bg{};
  int64_t nkeys = 0;
};

ScatterPlan plan_scatter(const gbg_grid &g, int ncomp, size_t esize, int n2) {
  ScatterPlan p;
  // 256 nodes, one a thread: at width 4 a region of 847 cells (3.3 a node), which one staging holds up
  // to 0.6 points a cell.  8x8x8 bricks with two nodes a thread (2.6 cells a node, half the bricks) took
  // 14.5 ms where these took 12.8 (256^3 x 3, 1e7 points, 30% in blobs): more regions go in passes.
  const int base[3] = {8, 8, 4};
  const int ebase[3] = {(size_t)ncomp * esize > 24 ? 8 : 16, 8, 8};
  p.nkeys = g.n[0] * g.n[1] * g.n[2];
  p.bricked = n2 <= 8 && p.nkeys < (int64_t(1) << 32) - 1 && brick_takes(g, ncomp, n2);
  for (int d = 0; d < 3; ++d) {
    p.bg.b[d] = (int32_t)std::min<int64_t>(base[d], g.n[d]);
    p.bg.nb[d] = (g.n[d] + p.bg.b[d] - 1) / p.bg.b[d];
    p.bg.eb[d] = (int32_t)std::min<int64_t>(ebase[d], g.n[d]);
    p.bg.enb[d] = (g.n[d] + p.bg.eb[d] - 1) / p.bg.eb[d];
    if (g.n[d] < n2 || g.n[d] >= (int64_t(1) << 31)) p.bricked = false;
  }
  p.bg.bvol = (int64_t)p.bg.b[0] * p.bg.b[1] * p.bg.b[2];
  return p;
}

// The scatter's workspace: keys, per-cell counts (then slot starts), ranks within a cell, the
// permutation, the scan's scratch, per slot the three axes' weights (64-bit fixed point for the
// brick scatter) and the quantities (for the brick scatter as mantissas and exponents, with per
// exponent brick the largest exponent of every component); for the pull also the stable sort's
// scratch.  flag: the sort's count of long runs, or the brick scatter's ticket.
struct ScatterLayout {
  uint32_t *keys, *counts, *rank, *perm, *flag;
  uint32_t *sort_tmp, *scan_tmp;
  void *rec, *qs;
  long long *qi;
  int16_t *qe;
  uint32_t *ebrick;
};

ScatterLayout scatter_layout(Arena &a, int64_t m, const ScatterPlan &P, int ncomp, int n2, size_t esize) {
  ScatterLayout L;
  // the words that start at zero stand together (scatter_clear)
  const size_t nexp = P.bricked ? (size_t)(P.bg.enb[0] * P.bg.enb[1] * P.bg.enb[2]) : 0;
  L.flag = a.take<uint32_t>(8);
  L.ebrick = P.bricked ? a.take<uint32_t>(nexp * ncomp) : nullptr;
  L.counts = a.take<uint32_t>((size_t)P.nkeys + 1);
  L.keys = a.take<uint32_t>((size_t)m);
  L.rank = a.take<uint32_t>((size_t)m);
  L.perm = a.take<uint32_t>((size_t)m);
  L.sort_tmp = P.bricked ? nullptr : a.take<uint32_t>((size_t)m);
  L.scan_tmp = a.take<uint32_t>(scan_temp_elems(P.nkeys + 1));
  const size_t rec_bytes = 3 * (size_t)n2 * (P.bricked ? sizeof(long long) : esize);
  L.rec = a.take<char>((size_t)m * rec_bytes);
  L.qs = P.bricked ? nullptr : a.take<char>((size_t)m * ncomp * esize);
  L.qi = P.bricked ? a.take<long long>((size_t)m * ncomp) : nullptr;
  L.qe = P.bricked ? a.take<int16_t>((size_t)m * ncomp) : nullptr;
  return L;
}

// Clears the flag, the exponent bricks and the counts.
gbg_status scatter_clear(const ScatterLayout &L, const ScatterPlan &P, cudaStream_t st) {
  const char *from = reinterpret_cast<const char *>(L.flag), *to = reinterpret_cast<const char *>(L.counts + P.nkeys + 1);
  GBG_CUDA_TRY(cudaMemsetAsync(L.flag, 0, (size_t)(to - from), st));
  return GBG_OK;
}

int bits_for(uint64_t max_value) {
  int b = 0;
  while (b < 32 && (max_value >> b) != 0) ++b;
  return b;
}

template <typename T, int N2, int CMAX, int REST = 0>
gbg_status launch_owner(const GridT<T> &g, const ScatterPlan &P, int ncomp, int cfrom, int cto, int wexp, int points,
                        const ScatterLayout &L, T *field, double beta, cudaStream_t st) {
  constexpr int CC = REST > CMAX ? REST : CMAX;
  constexpr size_t per = kDigitWords<CC, kDigits<T>> * 4 + kWeightWords<N2> * 8 + 4;
  const BrickGeo &bg = P.bg;
  const size_t e[3] = {(size_t)bg.b[0] + N2 - 1, (size_t)bg.b[1] + N2 - 1, (size_t)bg.b[2] + N2 - 1};
  const size_t tables = sizeof(uint32_t) * ((kSlotsMove<N2> ? 3 : 4) * e[0] * e[1] * e[2] + 2 + 3 * (e[0] + e[1] + e[2]) + (size_t)bg.bvol + (size_t)ncomp);
  const size_t sums = ((size_t)bg.bvol * CC * 28 + 15) & ~size_t(15);
  // an SM's 228 KB over the CTAs that the launch bounds ask for, less 1 KB reserved and the static part
  const size_t budget = 228 * 1024 / 2 - 1024 - 512;
  const int chunk = (int)(std::min<size_t>(points, (budget - tables - sums) / per) & ~size_t(3));
  const int chunk1 = (int)(std::min<size_t>(points, (budget - tables) / per) & ~size_t(3));
  const size_t smem = std::max(sums + chunk * per, chunk1 * per) + tables;
  auto kernel = k_scatter_owner<T, N2, CMAX, REST>;
  GBG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GBG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  // two CTAs per SM, by the launch bounds and the shared memory's share (more would find no ticket left)
  const int64_t nbricks = bg.nb[0] * bg.nb[1] * bg.nb[2];
  const int blocks = launch_blocks(nbricks, 1, 2);
  kernel<<<blocks, kThreads, smem, st>>>(g, bg, ncomp, cfrom, cto, chunk, chunk1, (int)sums, L.counts,
                                         static_cast<const long long *>(L.rec), L.qi, L.qe, L.ebrick, wexp, field,
                                         T(beta), beta == 0.0, L.flag + (cfrom > 0));
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  return GBG_OK;
}

// The owner kernel over all components, three to a trip and the last one, two or four by themselves: in the
// same launch up to width 4, whose bricks' listing costs more than the registers that a kernel of two
// sizes spills, in a second one from width 6.  96^3, 885k points, FP64, for 3, 4 and 5 components: width
// 4, 1.21, 1.64 and 2.18 ms (one at a time 2.82 and 3.47 for the last two), width 8, 8.4, 10.7 and 14.7 (18.7 and
// 23.1).
template <typename T, int N2>
gbg_status launch_owners(const GridT<T> &g, const ScatterPlan &P, int ncomp, int wexp, int points, const ScatterLayout &L,
                         T *field, double beta, cudaStream_t st) {
  auto go = [&](auto cmax, auto rest, int cfrom, int cto) {
    return launch_owner<T, N2, decltype(cmax)::value, decltype(rest)::value>(g, P, ncomp, cfrom, cto, wexp, points, L,
                                                                             field, beta, st);
  };
  constexpr std::integral_constant<int, 0> none{};
  constexpr std::integral_constant<int, 1> one{};
  constexpr std::integral_constant<int, 2> two{};
  constexpr std::integral_constant<int, 3> three{};
  constexpr std::integral_constant<int, 4> four{};
  if (ncomp == 1) return go(one, none, 0, 1);
  if (ncomp == 2) return go(two, none, 0, 2);
  if (ncomp == 4) return go(four, none, 0, 4);
  if (ncomp % 3 == 0) return go(three, none, 0, ncomp);
  if constexpr (N2 <= 4) return ncomp % 3 == 1 ? go(three, four, 0, ncomp) : go(three, two, 0, ncomp);
  const int main = ncomp % 3 == 1 ? ncomp - 4 : ncomp - 2;
  GBG_TRY(go(three, none, 0, main));
  return ncomp % 3 == 1 ? go(four, none, main, ncomp) : go(two, none, main, ncomp);
}

template <typename T, int N2, bool FIXED>
gbg_status launch_bricked(const GridT<T> &g, const ScatterPlan &P, const gbg_scheme &sch, int ncomp,
                          const T *x, const T *q, int64_t m, double alpha, const ScatterLayout &L, T *field,
                          double beta, int32_t *status, cudaStream_t st) {
  const SchemeT<T, N2> s = make_scheme<T, N2>(sch);
  const double bound = evaluated_weight_bound<T>(sch);
  const int wexp = fixed_weight_exp(bound), points = owner_points(bound, wexp);
  const int blocks_m = launch_blocks(m, kThreads);
  k_brick_keys<T><<<blocks_m, kThreads, 0, st>>>(g, P.bg, x, m, L.keys, L.counts, L.rank, q, ncomp, T(alpha),
                                                 L.ebrick, status);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  GBG_TRY(exclusive_scan_u32(L.counts, L.counts, P.nkeys + 1, L.scan_tmp, st));
  k_brick_place<<<blocks_m, kThreads, 0, st>>>(L.keys, L.rank, L.counts, m, L.perm);
  note_launch();
  k_brick_order<T, N2, FIXED ? N2 : 0><<<blocks_m, kThreads, 0, st>>>(
      g, s, x, L.perm, m, wexp, static_cast<long long *>(L.rec), q, ncomp, T(alpha), L.qi, L.qe);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  mark_main_start(st);
  GBG_TRY((launch_owners<T, N2>(g, P, ncomp, wexp, points, L, field, beta, st)));
  mark_main_stop(st);
  return GBG_OK;
}

// The deterministic scatter.  The brick scatter (integer sums, FP64-grade per node)
// whenever every axis is at least a stencil wide; otherwise the node pull (points sorted by
// cell, one thread per node summing its contributions in T in a fixed order), which also takes
// a stencil wider than the grid.
template <typename T>
gbg_status dispatch_scatter(const gbg_grid &grid, const gbg_scheme &sch, int ncomp, void *field,
                            const void *pos, int64_t m, const void *q, double alpha, double beta,
                            const ScatterPlan &P, const ScatterLayout &L, int32_t *status, cudaStream_t st) {
  const GridT<T> g = make_grid<T>(grid);
  const T *x = static_cast<const T *>(pos);
  T *f = static_cast<T *>(field);
  GBG_TRY(scatter_clear(L, P, st));
  if (P.bricked) {
    const T *qq = static_cast<const T *>(q);
    const int w = sch.stencil_width;
    const bool fixed = sch.num_powers == w;
#define GBG_BRICKED(W)                                                                               \
  return fixed ? launch_bricked<T, W, true>(g, P, sch, ncomp, x, qq, m, alpha, L, f, beta, status, st) \
               : launch_bricked<T, W, false>(g, P, sch, ncomp, x, qq, m, alpha, L, f, beta, status, st)
    if (w == 2) GBG_BRICKED(2);
    if (w == 4) GBG_BRICKED(4);
    if (w == 6) GBG_BRICKED(6);
    GBG_BRICKED(8);
#undef GBG_BRICKED
  }
  const int64_t ncells = g.npf;
  const SchemeT<T, GBG_MAX_NODES> s = make_scheme<T, GBG_MAX_NODES>(sch);
  k_cell_keys<T><<<launch_blocks(m, kThreads), kThreads, 0, st>>>(g, x, m, L.keys, L.counts, L.rank, status);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  GBG_TRY(exclusive_scan_u32(L.counts, L.counts, ncells + 1, L.scan_tmp, st));
  GBG_TRY(stable_counting_sort(L.keys, L.rank, L.counts, m, L.perm, L.flag, L.sort_tmp, st));
  T *rec = static_cast<T *>(L.rec);
  T *qs = static_cast<T *>(L.qs);
  k_scatter_prep<T><<<launch_blocks(m, kThreads), kThreads, 0, st>>>(
      g, s, ncomp, x, static_cast<const T *>(q), m, L.perm, T(alpha), rec, qs);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  const int blocks = launch_blocks(ncells, kThreads);
  const int bz = beta == 0.0;
  const int n2 = sch.stencil_width;
  const int cc = chunk_for(ncomp);
  mark_main_start(st);
#define GBG_PULL_N(W)                                                                                                  \
  if (n2 == W) {                                                                                                       \
    if (cc == 9) k_scatter_pull_n<T, W, 9><<<blocks, kThreads, 0, st>>>(g, ncomp, L.counts, rec, qs, f, T(beta), bz);  \
    else if (cc == 3) k_scatter_pull_n<T, W, 3><<<blocks, kThreads, 0, st>>>(g, ncomp, L.counts, rec, qs, f, T(beta), bz); \
    else k_scatter_pull_n<T, W, 1><<<blocks, kThreads, 0, st>>>(g, ncomp, L.counts, rec, qs, f, T(beta), bz);          \
  } else
  GBG_PULL_N(2) GBG_PULL_N(4) GBG_PULL_N(6) GBG_PULL_N(8) {
    switch (cc) {
      case 9: k_scatter_pull<T, 9><<<blocks, kThreads, 0, st>>>(g, n2, ncomp, L.counts, rec, qs, f, T(beta), bz); break;
      case 3: k_scatter_pull<T, 3><<<blocks, kThreads, 0, st>>>(g, n2, ncomp, L.counts, rec, qs, f, T(beta), bz); break;
      default: k_scatter_pull<T, 1><<<blocks, kThreads, 0, st>>>(g, n2, ncomp, L.counts, rec, qs, f, T(beta), bz); break;
    }
  }
#undef GBG_PULL_N
  mark_main_stop(st);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  return GBG_OK;
}

// ------------------------------------------------------- argument checks

gbg_status check_grid(const gbg_grid *g) {
  if (!g) return set_error(GBG_EARG, "null grid");
  for (int d = 0; d < 3; ++d) {
    if (g->n[d] <= 0) return set_error(GBG_EARG, "grid_size must be positive along every axis");
    if (!(std::isfinite(g->domain[d]) && g->domain[d] > 0))
      return set_error(GBG_EARG, "domain_size must be finite and positive along every axis");
    if (!(std::isfinite(g->spacing[d]) && g->spacing[d] > 0))
      return set_error(GBG_EARG, "grid_spacing must be finite and positive along every axis");
    if (!std::isfinite(g->origin[d])) return set_error(GBG_EARG, "origin must be finite along every axis");
  }
  if (g->n[0] > (int64_t(1) << 31) || g->n[1] > (int64_t(1) << 31) || g->n[2] > (int64_t(1) << 31))
    return set_error(GBG_EUNSUPPORTED, "grid axis longer than 2^31");
  return GBG_OK;
}

gbg_status check_scheme(const gbg_scheme *s) {
  if (!s) return set_error(GBG_EARG, "null scheme");
  if (s->stencil_width < 2 || s->stencil_width % 2 || s->stencil_width > GBG_MAX_NODES)
    return set_error(GBG_EARG, "scheme stencil_width must be even, 2..GBG_MAX_NODES");
  if (s->num_powers < 1 || s->num_powers > GBG_MAX_POWERS)
    return set_error(GBG_EARG, "scheme num_powers must be 1..GBG_MAX_POWERS");
  return GBG_OK;
}

gbg_status check_common(const gbg_grid *grid, gbg_dtype dtype, int32_t ncomp, int64_t m,
                        const gbg_scheme *scheme) {
  GBG_TRY(check_grid(grid));
  GBG_TRY(check_scheme(scheme));
  if (dtype != GBG_F32 && dtype != GBG_F64) return set_error(GBG_EARG, "dtype must be GBG_F32 or GBG_F64");
  if (ncomp < 1) return set_error(GBG_EARG, "ncomp must be at least 1");
  if (m < 0) return set_error(GBG_EDIM, "negative point count");
  if (m > 0x7fffffffLL) return set_error(GBG_EUNSUPPORTED, "more than 2^31-1 points");
  return GBG_OK;
}

}  // namespace
}  // namespace gbg

using namespace gbg;

extern "C" {

gbg_status gbg_interpolate(const gbg_grid *grid, gbg_dtype dtype, int32_t ncomp, const void *field,
                           const void *positions, int64_t npoints, const int32_t *traversal,
                           const gbg_scheme *scheme, void *out, int32_t *device_status,
                           void *stream) {
  clear_error();
  try {
    GBG_TRY(check_common(grid, dtype, ncomp, npoints, scheme));
    if (npoints == 0) return GBG_OK;
    if (!field || !positions || !out) return set_error(GBG_EARG, "interpolate: null array");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == GBG_F64)
      return dispatch_gather<double>(*grid, *scheme, ncomp, field, positions, npoints, traversal,
                                     out, device_status, st);
    return dispatch_gather<float>(*grid, *scheme, ncomp, field, positions, npoints, traversal, out,
                                  device_status, st);
  } catch (...) {
    return set_error(GBG_ENOMEM, "interpolate: host exception");
  }
}

gbg_status gbg_anterpolate_workspace_size(const gbg_grid *grid, gbg_dtype dtype, int32_t ncomp,
                                          int64_t npoints, const gbg_scheme *scheme, size_t *bytes) {
  clear_error();
  GBG_TRY(check_common(grid, dtype, ncomp, npoints, scheme));
  if (!bytes) return set_error(GBG_EARG, "null bytes");
  const int64_t ncells = grid->n[0] * grid->n[1] * grid->n[2];
  if (ncells >= (int64_t(1) << 32) - 1)
    return set_error(GBG_EUNSUPPORTED, "anterpolate: grids of 2^32 or more cells");
  const size_t es = dtype == GBG_F64 ? 8 : 4;
  const ScatterPlan P = plan_scatter(*grid, ncomp, es, scheme->stencil_width);
  Arena a;
  scatter_layout(a, npoints, P, ncomp, scheme->stencil_width, es);
  *bytes = npoints == 0 ? 0 : a.used + 256;
  return GBG_OK;
}

gbg_status gbg_anterpolate(const gbg_grid *grid, gbg_dtype dtype, int32_t ncomp, void *field,
                           const void *positions, int64_t npoints, const void *quantities,
                           const int32_t *traversal, const gbg_scheme *scheme, double alpha,
                           double beta, void *workspace, size_t workspace_bytes,
                           int32_t *device_status, void *stream) {
  clear_error();
  (void)traversal;  // the deterministic pull is independent of the visiting order
  try {
    size_t need = 0;
    GBG_TRY(gbg_anterpolate_workspace_size(grid, dtype, ncomp, npoints, scheme, &need));
    if (!field) return set_error(GBG_EARG, "anterpolate: null field");
    if (!std::isfinite(alpha) || !std::isfinite(beta)) {
      // allowed by the reference (T(alpha) of an Inf is Inf); passed through as given
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t total = grid->n[0] * grid->n[1] * grid->n[2] * (int64_t)ncomp;
    if (npoints == 0) {
      // Interpolation.jl:1309-1313: the prescale happens even with no points.
      k_fill_or_scale<<<launch_blocks(total, kThreads), kThreads, 0, st>>>(field, total,
                                                                           dtype == GBG_F64, beta);
      note_launch();
      GBG_CUDA_TRY(cudaGetLastError());
      return GBG_OK;
    }
    if (!positions || !quantities) return set_error(GBG_EARG, "anterpolate: null array");
    Scratch scratch;
    GBG_TRY(scratch.acquire(workspace, workspace_bytes, need, st));
    Arena a;
    a.base = static_cast<char *>(scratch.ptr);
    const size_t es = dtype == GBG_F64 ? 8 : 4;
    const ScatterPlan P = plan_scatter(*grid, ncomp, es, scheme->stencil_width);
    const ScatterLayout L = scatter_layout(a, npoints, P, ncomp, scheme->stencil_width, es);
    if (dtype == GBG_F64)
      return dispatch_scatter<double>(*grid, *scheme, ncomp, field, positions, npoints, quantities,
                                      alpha, beta, P, L, device_status, st);
    return dispatch_scatter<float>(*grid, *scheme, ncomp, field, positions, npoints, quantities,
                                   alpha, beta, P, L, device_status, st);
  } catch (...) {
    return set_error(GBG_ENOMEM, "anterpolate: host exception");
  }
}

// ------------------------------------------------ allocation-free scatter
//
// The scratch of gbg_anterpolate_noalloc: one fixed array per device, part of this
// library's device image, so the entry point never allocates.  Host code must not pass
// the array's name to a kernel (on the host it names a host-side stand-in).  Its device
// address is looked up on every call, in the context current at the call: an address
// kept from an earlier call would be stale after a device reset or in another context.
static __device__ __align__(256) unsigned char g_noalloc_scratch[GBG_NOALLOC_SCRATCH_BYTES];

static gbg_status noalloc_scratch(void **out) {
  void *p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess || !p)
    return set_error(GBG_ECUDA, std::string("cudaGetSymbolAddress of the static scratch failed: ") +
                                    cudaGetErrorString(e));
  *out = p;
  return GBG_OK;
}

gbg_status gbg_anterpolate_noalloc(const gbg_grid *grid, gbg_dtype dtype, int32_t ncomp, void *field,
                                   const void *positions, int64_t npoints, const void *quantities,
                                   const gbg_scheme *scheme, double alpha, double beta,
                                   int32_t *device_status, void *stream) {
  clear_error();
  try {
    size_t need = 0;
    GBG_TRY(gbg_anterpolate_workspace_size(grid, dtype, ncomp, npoints, scheme, &need));
    if (need > GBG_NOALLOC_SCRATCH_BYTES)
      return set_error(GBG_EUNSUPPORTED, "anterpolate (no-alloc): this problem needs " + std::to_string(need) +
                                             " bytes of scratch; the static scratch holds " +
                                             std::to_string((size_t)GBG_NOALLOC_SCRATCH_BYTES));
    void *scratch = nullptr;
    if (need > 0) GBG_TRY(noalloc_scratch(&scratch));
    // The shared path: with a caller workspace it allocates nothing, and it clears the
    // per-cell counts and the sort's flag (the only words that must start at zero) before
    // every use.
    const gbg_status st = gbg_anterpolate(grid, dtype, ncomp, field, positions, npoints, quantities, nullptr,
                                          scheme, alpha, beta, scratch, GBG_NOALLOC_SCRATCH_BYTES,
                                          device_status, stream);
    return st;
  } catch (...) {
    return set_error(GBG_ENOMEM, "anterpolate (no-alloc): host exception");
  }
}

static gbg_status traversal_tiles(const gbg_grid *grid, int64_t tile_size, int64_t tiles[3]) {
  if (tile_size < 1) return set_error(GBG_EARG, "tile_size must be at least 1, got " + std::to_string(tile_size));
  for (int d = 0; d < 3; ++d) {
    const int64_t t = (grid->n[d] + tile_size - 1) / tile_size;
    tiles[d] = t > 1 ? t : 1;
  }
  const double total = (double)tiles[0] * (double)tiles[1] * (double)tiles[2];
  if (total >= 4294967296.0) return set_error(GBG_EUNSUPPORTED, "traversal order: 2^32 or more tiles");
  return GBG_OK;
}

gbg_status gbg_point_traversal_order_workspace_size(const gbg_grid *grid, int64_t npoints,
                                                    int64_t tile_size, size_t *bytes) {
  clear_error();
  GBG_TRY(check_grid(grid));
  int64_t tiles[3];
  GBG_TRY(traversal_tiles(grid, tile_size, tiles));
  if (!bytes) return set_error(GBG_EARG, "null bytes");
  if (npoints < 0 || npoints > 0x7fffffffLL) return set_error(GBG_EUNSUPPORTED, "point count outside 0..2^31-1");
  Arena a;
  a.take<uint32_t>((size_t)npoints);
  a.take<uint32_t>((size_t)npoints);
  a.take<uint32_t>((size_t)npoints);
  a.take<char>(radix_sort_temp_bytes(npoints));
  *bytes = npoints == 0 ? 0 : a.used + 256;
  return GBG_OK;
}

gbg_status gbg_point_traversal_order(const gbg_grid *grid, gbg_dtype dtype, const void *positions,
                                     int64_t npoints, int64_t tile_size, int32_t *order,
                                     void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  try {
    size_t need = 0;
    GBG_TRY(gbg_point_traversal_order_workspace_size(grid, npoints, tile_size, &need));
    if (dtype != GBG_F32 && dtype != GBG_F64) return set_error(GBG_EARG, "dtype must be GBG_F32 or GBG_F64");
    if (npoints == 0) return GBG_OK;
    if (!positions || !order) return set_error(GBG_EARG, "traversal order: null array");
    int64_t tiles[3];
    GBG_TRY(traversal_tiles(grid, tile_size, tiles));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Scratch scratch;
    GBG_TRY(scratch.acquire(workspace, workspace_bytes, need, st));
    Arena a;
    a.base = static_cast<char *>(scratch.ptr);
    uint32_t *keys = a.take<uint32_t>((size_t)npoints);
    uint32_t *skeys = a.take<uint32_t>((size_t)npoints);
    uint32_t *perm = a.take<uint32_t>((size_t)npoints);
    void *tmp = a.take<char>(radix_sort_temp_bytes(npoints));
    const int blocks = launch_blocks(npoints, kThreads);
    if (dtype == GBG_F64) {
      // inverse_tile = T(tiles) / T(domain), origin = T(origin)  (Interpolation.jl:773-774)
      k_tile_keys<double><<<blocks, kThreads, 0, st>>>(
          static_cast<const double *>(positions), npoints, grid->origin[0], grid->origin[1],
          grid->origin[2], (double)tiles[0] / grid->domain[0], (double)tiles[1] / grid->domain[1],
          (double)tiles[2] / grid->domain[2], tiles[0], tiles[1], tiles[2], keys);
      note_launch();
    } else {
      k_tile_keys<float><<<blocks, kThreads, 0, st>>>(
          static_cast<const float *>(positions), npoints, (float)grid->origin[0],
          (float)grid->origin[1], (float)grid->origin[2], (float)tiles[0] / (float)grid->domain[0],
          (float)tiles[1] / (float)grid->domain[1], (float)tiles[2] / (float)grid->domain[2],
          tiles[0], tiles[1], tiles[2], keys);
      note_launch();
    }
    GBG_CUDA_TRY(cudaGetLastError());
    const uint64_t max_key = (uint64_t)tiles[0] * (uint64_t)tiles[1] * (uint64_t)tiles[2] - 1;
    GBG_TRY(radix_sort_pairs(keys, nullptr, skeys, perm, npoints, bits_for(max_key), tmp, st));
    k_to_one_based<<<blocks, kThreads, 0, st>>>(perm, order, npoints);
    note_launch();
    GBG_CUDA_TRY(cudaGetLastError());
    return GBG_OK;
  } catch (...) {
    return set_error(GBG_ENOMEM, "traversal order: host exception");
  }
}

gbg_status gbg_validate_traversal(const int32_t *order, int64_t npoints, int64_t *host_low,
                                  int64_t *host_high, int64_t *host_visited, void *stream) {
  clear_error();
  if (npoints < 0 || npoints > 0x7fffffffLL) return set_error(GBG_EUNSUPPORTED, "point count outside 0..2^31-1");
  if (npoints == 0) {
    if (host_visited) *host_visited = 0;
    return GBG_OK;
  }
  if (!order) return set_error(GBG_EARG, "validate traversal: null order");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Scratch scratch;
  const size_t words = ((size_t)npoints + 31) / 32;  // a bit per point
  const size_t need = 256 + sizeof(uint32_t) * words;
  GBG_TRY(scratch.acquire(nullptr, 0, need, st));
  unsigned long long *stats = static_cast<unsigned long long *>(scratch.ptr);
  uint32_t *seen = reinterpret_cast<uint32_t *>(static_cast<char *>(scratch.ptr) + 256);
  GBG_CUDA_TRY(cudaMemsetAsync(seen, 0, sizeof(uint32_t) * words, st));
  k_validate_init<<<1, 1, 0, st>>>(stats);
  note_launch();
  k_validate<<<launch_blocks(npoints, kThreads), kThreads, 0, st>>>(order, npoints, seen, stats);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  long long h[3];
  GBG_CUDA_TRY(cudaMemcpyAsync(h, stats, sizeof(h), cudaMemcpyDeviceToHost, st));
  GBG_CUDA_TRY(cudaStreamSynchronize(st));
  if (host_low) *host_low = h[0];
  if (host_high) *host_high = h[1];
  if (host_visited) *host_visited = h[2];
  if (h[0] < 1 || h[1] > npoints)
    return set_error(GBG_ETRAVERSAL, "a point traversal order must name points in 1:" + std::to_string(npoints) +
                                         ", but it spans " + std::to_string(h[0]) + ":" + std::to_string(h[1]));
  if (h[2] != npoints)
    return set_error(GBG_ETRAVERSAL, "a point traversal order must name every point exactly once, but it names " +
                                         std::to_string(h[2]) + " of " + std::to_string(npoints));
  return GBG_OK;
}

}  // extern "C"
