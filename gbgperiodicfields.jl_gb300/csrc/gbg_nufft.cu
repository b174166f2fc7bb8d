// NUFFT window transfers on the oversampled grid (sm_103a), and the host-side window
// transform used for the deconvolution.
//
// The reference's fast spectral transfer (src/Interpolation.jl:1611-2070, NUFFT) spreads
// point quantities onto an oversampled (sigma*N) physical grid with the exponential-of-
// semicircle (ES) window, or gathers from it, and does the rest -- the FFT of the
// oversampled grid, the exchange of modes with the reference grid, the division by the
// window's transform -- on whole arrays.  This file holds the two per-point kernels
// (_nufft_gather_kernel!, 1864-1914; _nufft_spread_kernel!, 1919-1950) and the window
// transform (_es_window_transform, 1652-1662); the array steps use cuFFT through the host
// facade.
//
// The FP32 gather bins the points by tile of the oversampled grid; a CTA per tile stages the
// tile's region in shared memory and a warp per point contracts its W^3 stencil there (the
// lanes over the W^2 rows, the x direction first), reduced across the warp.  The FP64 gather
// is a thread per point reading the oversampled field directly (FP64-pipe-bound either way).
//
// The spread is deterministic, unlike the reference's atomic float adds: the window
// weights (evaluated in T as the reference does) and the quantities are converted once per
// point to 64-bit fixed point, every contribution is formed from them with integer high
// products and added as an integer.  Integer addition is associative, so the sums -- and
// the field -- do not depend on the order in which threads add.  The scales leave no
// node's sum able to overflow and keep about M*max|q|*2^-62 of absolute resolution per
// contribution.  The points are binned by tile of the oversampled grid and each tile's sums
// are formed in shared memory before one global add per node: no FP64 arithmetic and no
// global atomic runs per node and point (GB300 runs FP64 at 1/58 of its FP32 rate, while
// 64-bit integer products run on the integer pipes).

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "gbg_common.cuh"

namespace gbg {
namespace {

constexpr int kNThreads = 256;
constexpr int kMaxWidth = 16;
constexpr int kTile = 8;  // points are binned by tiles of kTile^3 oversampled-grid nodes

template <typename T>
struct NGrid {
  int64_t n[3];
  T o[3], d[3];  // T.(origin), T.(grid_spacing) of the oversampled grid
};

template <typename T>
NGrid<T> make_ngrid(const gbg_grid &g) {
  NGrid<T> r;
  for (int a = 0; a < 3; ++a) {
    r.n[a] = g.n[a];
    r.o[a] = T(g.origin[a]);
    r.d[a] = T(g.spacing[a]);
  }
  return r;
}

template <typename T>
__device__ __forceinline__ T nan_t();
template <>
__device__ __forceinline__ double nan_t<double>() { return __longlong_as_double(0x7ff8000000000000LL); }
template <>
__device__ __forceinline__ float nan_t<float>() { return __int_as_float(0x7fc00000); }

__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }

// Interpolation.jl:1634-1635 -- _stencil_half: the stencil follows the nearer node for an
// odd width.
template <int W, typename T>
__device__ __forceinline__ int stencil_half(T t) {
  return (W % 2 == 1 && t < T(0.5)) ? (W + 1) / 2 : W / 2;
}

// Interpolation.jl:1638-1645 -- _es_weights: node i (1-based) at offset i - half, weight
// exp(beta*(sqrt(max(1 - z^2, 0)) - 1)) with z = 2*(t - (i - half))/W; in FP32 with the reference's
// separate roundings.
template <int W>
__device__ __forceinline__ float es_weight(float t, float beta, int off) {
  const float z = div_rn(mul_rn(2.0f, add_rn(t, -(float)off)), (float)W);
  const float r = add_rn(1.0f, -mul_rn(z, z));
  return expf(mul_rn(beta, add_rn(sqrtf(r > 0.0f ? r : 0.0f), -1.0f)));
}

// The FP64 window's own exponential, e^x for x <= 0, since its kernels are bound by the FP64 pipe: x = (32
// m + j) ln2/32 + r with |r| <= ln2/64, a table of 2^(j/32) and e^r - 1 by its Taylor polynomial to the
// sixth degree (what is left out, r^7/5040, is below 4e-18), as in Tang's table-driven exponential
// (ACM TOMS 15, 1989).  Ten FP64 operations, within 1.8 * 2^-53 of itself; below -700 it gives 0.
struct ExpTable {
  double v[32];
};
inline ExpTable make_exp_table() {
  ExpTable t;
  for (int j = 0; j < 32; ++j) t.v[j] = std::exp2(j / 32.0);
  return t;
}
__device__ __forceinline__ double window_exp(double x, const double *table) {
  const double big = 6755399441055744.0;  // 1.5 * 2^52: the low bits of a sum with it are a rounded integer
  const double kd = fma(x, 46.16624130844683, big);  // 32 / ln 2
  const int k = __double2loint(kd);
  const double kr = kd - big;
  double r = fma(kr, -0.02166084939249829, x);  // ln2/32, in two parts
  r = fma(kr, -7.247021293269686e-19, r);
  double p = fma(1.0 / 720.0, r, 1.0 / 120.0);
  p = fma(p, r, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  const double t = table[k & 31];
  const double v = fma(t * r, p, t);
  if ((uint32_t)__double2hiint(x) > 0xc085e000u) return 0.0;  // x < -700, by its high word
  return __hiloint2double(__double2hiint(v) + ((k >> 5) << 20), __double2loint(v));
}

// The window's W weights in FP64, fused: z = 2 (t - off) / W (one product for a power of two, else the
// product by the rounded reciprocal corrected by its residual), w = exp(beta sqrt(1 - z^2) - beta); 24
// operations a weight beside the root's instead of about 50.
template <int W>
__device__ __forceinline__ double es_weight_fused(double t, double beta, int off, const double *table) {
  const double a = t - (double)off;
  double z = a * (2.0 / W);
  if constexpr ((W & (W - 1)) != 0) z = fma(fma(-z, (double)W, a + a), 1.0 / W, z);
  const double r = fma(-z, z, 1.0);
  // past the window's end by a rounding: the root of zero
  return window_exp(__double2hiint(r) < 0 ? -beta : fma(beta, sqrt(r), -beta), table);
}

// _visit (Interpolation.jl:618-619), bounds-checked.
__device__ __forceinline__ bool nvisit(const int32_t *__restrict__ trav, int64_t w, int64_t m, int64_t &p,
                                       int32_t *status) {
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

// The FP64 gather, a thread per point straight from the oversampled field: the three axes'
// weights, the W^3 stencil with the periodic wrap, contracted x, then y, then z.  It is bound by the FP64
// pipe (a warp's operation every 76 clocks of a scheduler), so it counts operations: W^3 + W^2 + W a
// component and 3 W weights.  128^3 x 3, 2e6 points, W = 8: 9.1 ms, 11.3 with the plain weights and a
// weight product per row.  The tiled form's cross-lane FP64 reductions and per-lane weights cost more.
template <int W>
__global__ void __launch_bounds__(kNThreads)
    k_nufft_gather(NGrid<double> g, ExpTable exps, const double *__restrict__ f, const double *__restrict__ pos,
                   int64_t m, int ncomp, double beta, const int32_t *__restrict__ trav, double *__restrict__ out,
                   int32_t *status) {
  __shared__ double table[32];
  if (threadIdx.x < 32) table[threadIdx.x] = exps.v[threadIdx.x];
  __syncthreads();
  const int64_t nxy = g.n[0] * g.n[1], npf = nxy * g.n[2];
  for (int64_t wi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; wi < m; wi += (int64_t)gridDim.x * blockDim.x) {
    int64_t p;
    if (!nvisit(trav, wi, m, p, status)) continue;
    double w[3][W];
    int32_t first[3];
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      int64_t base;
      double t;
      ok &= locate(__ldg(pos + p + m * a), g.o[a], g.d[a], base, t);
      const int half = stencil_half<W>(t);
#pragma unroll
      for (int i = 0; i < W; ++i) w[a][i] = es_weight_fused<W>(t, beta, i + 1 - half, table);
      first[a] = (int32_t)imod(base + (1 - half), g.n[a]);
    }
    if (!ok) {
      if (status) atomicOr(status, GBG_DEV_NONFINITE);
      for (int c = 0; c < ncomp; ++c) out[p + m * c] = nan_t<double>();
      continue;
    }
    const int32_t n0 = (int32_t)g.n[0], n1 = (int32_t)g.n[1], n2 = (int32_t)g.n[2];
    int32_t ix[W], iy[W];
    ix[0] = first[0];
    iy[0] = first[1];
#pragma unroll
    for (int i = 1; i < W; ++i) {
      ix[i] = ix[i - 1] + 1 == n0 ? 0 : ix[i - 1] + 1;
      iy[i] = iy[i - 1] + 1 == n1 ? 0 : iy[i - 1] + 1;
    }
    for (int c = 0; c < ncomp; ++c) {
      const double *fc = f + npf * c;
      double acc = 0.0;
      int32_t z = first[2];
#pragma unroll 1
      for (int k = 0; k < W; ++k) {
        const double *plane = fc + nxy * z;
        double wz = w[2][0];
#pragma unroll
        for (int q = 1; q < W; ++q)
          if (q == k) wz = w[2][q];
        double sy = 0.0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
          const double *row = plane + g.n[0] * iy[j];
          double sx = w[0][0] * __ldg(row + ix[0]);
#pragma unroll
          for (int i = 1; i < W; ++i) sx = fma(w[0][i], __ldg(row + ix[i]), sx);
          sy = j ? fma(w[1][j], sx, sy) : w[1][0] * sx;
        }
        acc = k ? fma(wz, sy, acc) : wz * sy;
        z = z + 1 == n2 ? 0 : z + 1;
      }
      out[p + m * c] = acc;
    }
  }
}

// Tiled window gather: a CTA per tile stages the tile's region ((kTile + W - 1)^3 nodes of
// the oversampled field, for a group of components) in shared memory; a warp per point
// evaluates the point's 3W window weights across its lanes, its lanes take the W^2 rows of the
// stencil, contract x first, and the row sums are reduced across the warp.
template <typename T, int W>
__global__ void __launch_bounds__(kNThreads)
    k_nufft_gather_tiles(NGrid<T> g, const T *__restrict__ f, const T *__restrict__ pos, int64_t m, int ncomp,
                         int group, T beta, const int32_t *__restrict__ trav, int64_t nt0, int64_t nt1,
                         int64_t ntiles, const uint32_t *__restrict__ tstart, const uint32_t *__restrict__ order,
                         const int32_t *__restrict__ first, T *__restrict__ out) {
  constexpr int R = kTile + W - 1;
  constexpr int R3 = R * R * R;
  extern __shared__ __align__(16) unsigned char gsm[];
  T *reg = reinterpret_cast<T *>(gsm);  // group x R3 values
  __shared__ T swt[kNThreads / 32][3 * W];
  const int64_t nxy = g.n[0] * g.n[1], npf = nxy * g.n[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint32_t t0 = tstart[tile], t1 = tstart[tile + 1];
    if (t1 == t0) continue;  // uniform over the CTA
    const int64_t tx = (tile % nt0) * kTile, ty = ((tile / nt0) % nt1) * kTile, tz = (tile / (nt0 * nt1)) * kTile;
    for (int c0 = 0; c0 < ncomp; c0 += group) {
      const int cg = min(group, ncomp - c0);
      __syncthreads();  // the previous group's region is no longer read
      for (int e = threadIdx.x; e < cg * R3; e += blockDim.x) {
        const int cc = e / R3, r = e - cc * R3;
        const int rx = r % R, ry = (r / R) % R, rz = r / (R * R);
        const int64_t x = (tx + rx) % g.n[0], y = (ty + ry) % g.n[1], z = (tz + rz) % g.n[2];
        reg[e] = __ldg(f + npf * (c0 + cc) + z * nxy + y * g.n[0] + x);
      }
      __syncthreads();
      for (uint32_t pt = t0 + warp; pt < t1; pt += nwarps) {
        const uint32_t wi = order[pt];
        int64_t p = wi;
        if (trav) p = (int64_t)__ldg(trav + wi) - 1;
        for (int e = lane; e < 3 * W; e += 32) {  // 3W can exceed the 32 lanes (W > 10)
          const int a = e / W, i = e - a * W;
          int64_t base;
          T t;
          locate(__ldg(pos + p + m * a), g.o[a], g.d[a], base, t);
          swt[warp][e] = es_weight<W>(t, beta, i + 1 - stencil_half<W>(t));
        }
        const int ox = (int)(first[3 * (int64_t)wi] - tx), oy = (int)(first[3 * (int64_t)wi + 1] - ty),
                  oz = (int)(first[3 * (int64_t)wi + 2] - tz);
        __syncwarp();
        T acc[4] = {T(0), T(0), T(0), T(0)};  // up to four components per pass of the rows
        for (int cb = 0; cb < cg; cb += 4) {
          const int nc = min(4, cg - cb);
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[q] = T(0);
          for (int rw = lane; rw < W * W; rw += 32) {
            const int j = rw % W, k = rw / W;
            const T wyz = mul_rn(swt[warp][W + j], swt[warp][2 * W + k]);
            const T *row = reg + ((oz + k) * R + oy + j) * R + ox;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (q < nc) {
                const T *rq = row + (cb + q) * R3;
                T sx = T(0);
#pragma unroll
                for (int i = 0; i < W; ++i) sx = fma_rn(swt[warp][i], rq[i], sx);
                acc[q] = fma_rn(wyz, sx, acc[q]);
              }
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            T v = acc[q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0 && q < nc) out[p + m * (c0 + cb + q)] = v;
          }
        }
        __syncwarp();
      }
    }
  }
}

// Largest |q| over all points and components, as ordered double bits (NaN above all).
template <typename T>
__global__ void __launch_bounds__(kNThreads)
    k_nufft_qmax(const T *__restrict__ q, int64_t n, unsigned long long *qmax_bits) {
  unsigned long long mx = 0ull;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(fabs((double)q[i]));
    mx = b > mx ? b : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = other > mx ? other : mx;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(qmax_bits, mx);
}

// The fixed-point scales of a spread.  Weights are w * 2^62 (ES weights lie in [0, 1]);
// quantities q * 2^(62 - eq) with max|q| < 2^eq; a contribution is
// hi(hi(hi(Wy, Wz), Wx), |Q|) = w |q| 2^(56 - eq) < 2^56, shifted right (rounded) by
// s = max(0, em - 6) with M <= 2^em, so that no node's sum of at most M contributions can
// reach 2^62.  A node's value is its sum times 2^(eq + s - 56).
struct SpreadScale {
  int eq, s;
};
__device__ __forceinline__ SpreadScale spread_scale(unsigned long long qmax_bits, int64_t m) {
  int eq = 0, em = 0;
  frexp(__longlong_as_double((long long)qmax_bits), &eq);
  frexp((double)m, &em);
  return {eq, em > 6 ? em - 6 : 0};
}

// Spread, pass 1: each FP64 point's window weights as 64-bit fixed point (an FP32 point's are
// evaluated where they are used), its first stencil node per axis, and its
// tile (kTile^3 nodes holding the first node) with its rank there from an atomic count --
// the order within a tile does not matter, the sums being integer.  A point with a
// non-finite position goes to the extra bucket ntiles, which no tile visits.
// For the gather (out given, FP32 only) a point with a non-finite position gets NaN in out (ncomp
// components) here.
template <typename T, int W>
__global__ void __launch_bounds__(kNThreads)
    k_nufft_bin(NGrid<T> g, const T *__restrict__ pos, int64_t m, T beta, int64_t nt0, int64_t nt1,
                int64_t ntiles, const int32_t *__restrict__ trav, uint32_t *__restrict__ tcount,
                uint32_t *__restrict__ tkey, uint32_t *__restrict__ rank, int32_t *__restrict__ first,
                unsigned long long *__restrict__ wbuf, int32_t *status, ExpTable exps, T *__restrict__ out = nullptr,
                int ncomp = 0) {
  __shared__ double table[32];
  if constexpr (sizeof(T) == 8) {
    if (threadIdx.x < 32) table[threadIdx.x] = exps.v[threadIdx.x];
    __syncthreads();
  }
  for (int64_t wi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; wi < m; wi += (int64_t)gridDim.x * blockDim.x) {
    int64_t p;
    if (!nvisit(trav, wi, m, p, status)) {
      // a bad traversal entry: the visit slot wi carries no point
      tkey[wi] = (uint32_t)ntiles;
      rank[wi] = atomicAdd(tcount + ntiles, 1u);
      continue;
    }
    bool ok = true;
    int64_t s[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      int64_t base;
      T t;
      ok &= locate(__ldg(pos + p + m * a), g.o[a], g.d[a], base, t);
      const int half = stencil_half<W>(t);
      if constexpr (sizeof(T) == 8) {
#pragma unroll
        for (int i = 0; i < W; ++i)  // w * 2^62, exact to the rounding of one conversion
          wbuf[(3 * wi + a) * W + i] =
              ok ? (unsigned long long)fixed_rn(es_weight_fused<W>(t, beta, i + 1 - half, table), 62) : 0ull;
      }
      s[a] = imod(base + (1 - half), g.n[a]);
      first[3 * wi + a] = (int32_t)s[a];
    }
    if (!ok && status) atomicOr(status, GBG_DEV_NONFINITE);
    if (!ok && out)
      for (int c = 0; c < ncomp; ++c) out[p + m * c] = nan_t<T>();
    const int64_t key = ok ? ((s[2] / kTile) * nt1 + s[1] / kTile) * nt0 + s[0] / kTile : ntiles;
    tkey[wi] = (uint32_t)key;
    rank[wi] = atomicAdd(tcount + key, 1u);
  }
}

// Spread, pass 2: the visit slots in tile order.
__global__ void __launch_bounds__(kNThreads)
    k_nufft_place(int64_t m, const uint32_t *__restrict__ tkey, const uint32_t *__restrict__ rank,
                  const uint32_t *__restrict__ tstart, uint32_t *__restrict__ order) {
  for (int64_t wi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; wi < m; wi += (int64_t)gridDim.x * blockDim.x)
    order[tstart[tkey[wi]] + rank[wi]] = (uint32_t)wi;
}

// A weight in [0, 1] of FP32 as w * 2^62, from its bits (exact down to 2^-62).
__device__ __forceinline__ unsigned long long weight_fixed(float w) {
  const uint32_t b = __float_as_uint(w);
  const int sh = (int)(b >> 23) - 88;  // w = (2^23 + mantissa) 2^(exponent - 150)
  const unsigned long long man = (b & 0x7fffffu) | (b >> 23 ? 0x800000u : 0u);
  return sh >= 0 ? man << sh : (sh > -24 ? man >> -sh : 0ull);
}

// Spread, pass 3: a CTA per tile.  For a group of CG components at a time the tile's
// region ((kTile + W - 1)^3 nodes) is summed in shared memory -- a warp per point, its lanes
// over the point's W^3 nodes, each contribution hi(hi(Wyz, Wx), |Q|) formed with integer
// high products (no FP64 arithmetic per node) and rounded to s bits, then added to the
// node's 64-bit sum as 32-bit low and high words with a carry
// (native 32-bit shared atomics) -- then every nonzero node sum is added to the grid's by
// one global integer atomic.  Integer sums do not depend on the order of the adds.  A lane's nodes
// lie at the same places of every point's stencil, so up to width 8 they are worked out once per
// launch; up to three components' quantities are held in registers over a point's nodes.  Bound by
// issue on the integer pipes.  128^3 x 3, 2e6 FP32 points, W = 6: 4.1 ms, 5.0 with the places worked
// out per point and FP64 weight tables.
constexpr int kMaxGroup = 32;

template <typename T, int W>
__global__ void __launch_bounds__(kNThreads)
    k_nufft_spread_tiles(NGrid<T> g, const T *__restrict__ pos, T beta, int64_t m, const T *__restrict__ qv,
                         const int32_t *__restrict__ trav, int ncomp, int group, int64_t nt0, int64_t nt1,
                         int64_t ntiles, const uint32_t *__restrict__ tstart, const uint32_t *__restrict__ order,
                         const int32_t *__restrict__ first, const unsigned long long *__restrict__ wbuf,
                         const unsigned long long *__restrict__ qmax_bits, unsigned long long *__restrict__ acc) {
  constexpr int R = kTile + W - 1;
  constexpr int R3 = R * R * R;
  constexpr int NI = (W * W * W + 31) / 32;  // a lane's nodes
  constexpr bool kHeld = W <= 8;
  // group x R3 64-bit sums: a plane of low words, then a plane of high words
  extern __shared__ uint32_t sacc_lo[];
  uint32_t *sacc_hi = sacc_lo + group * R3;
  __shared__ unsigned long long swyz[kNThreads / 32][W * W], sw[kNThreads / 32][3 * W];
  const double qmax = __longlong_as_double((long long)*qmax_bits);
  if (!isfinite(qmax)) return;  // the field is set to NaN by k_nufft_finish
  const SpreadScale sc = spread_scale(*qmax_bits, m);
  const unsigned long long round = sc.s ? (1ull << (sc.s - 1)) : 0ull;
  const int64_t nxy = g.n[0] * g.n[1], npf = nxy * g.n[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // node idx of a stencil: its place in the region relative to the first node, its row and its x
  auto node = [&](int idx, int &rel, int &jk, int &i) {
    i = idx % W;
    jk = idx / W;
    rel = ((jk / W) * R + jk % W) * R + i;
  };
  uint32_t held[kHeld ? NI : 1];
  if constexpr (kHeld) {
#pragma unroll
    for (int t = 0; t < NI; ++t) {
      int rel, jk, i;
      node(min(lane + 32 * t, W * W * W - 1), rel, jk, i);
      held[t] = (uint32_t)rel | (uint32_t)jk << 12 | (uint32_t)i << 20;
    }
  }
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint32_t t0 = tstart[tile], t1 = tstart[tile + 1];
    if (t1 == t0) continue;  // uniform over the CTA
    const int64_t tx = (tile % nt0) * kTile, ty = ((tile / nt0) % nt1) * kTile, tz = (tile / (nt0 * nt1)) * kTile;
    for (int c0 = 0; c0 < ncomp; c0 += group) {
      const int cg = min(group, ncomp - c0);
      for (int r = threadIdx.x; r < cg * R3; r += blockDim.x) {
        sacc_lo[r] = 0u;
        sacc_hi[r] = 0u;
      }
      __syncthreads();
      for (uint32_t pt = t0 + warp; pt < t1; pt += nwarps) {
        const uint32_t wi = order[pt];
        int64_t p = wi;
        if (trav) p = (int64_t)__ldg(trav + wi) - 1;
        for (int e = lane; e < 3 * W; e += 32) {  // 3W can exceed the 32 lanes (W > 10)
          if constexpr (sizeof(T) == 8) {
            sw[warp][e] = wbuf[3 * (int64_t)wi * W + e];
          } else {
            const int a = e / W;
            int64_t base;
            T t;
            locate(__ldg(pos + p + m * a), g.o[a], g.d[a], base, t);
            sw[warp][e] = weight_fixed(es_weight<W>(t, beta, e - a * W + 1 - stencil_half<W>(t)));
          }
        }
        __syncwarp();
        for (int e = lane; e < W * W; e += 32) swyz[warp][e] = __umul64hi(sw[warp][W + e % W], sw[warp][2 * W + e / W]);
        const int origin = (int)((first[3 * (int64_t)wi + 2] - tz) * R + (first[3 * (int64_t)wi + 1] - ty)) * R +
                           (int)(first[3 * (int64_t)wi] - tx);
        __syncwarp();
        for (int cb = 0; cb < cg; cb += 3) {
          const int nc = min(3, cg - cb);
          unsigned long long mag[3], neg[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const long long qq = c < nc ? fixed_rn((double)__ldg(qv + p + m * (c0 + cb + c)), 62 - sc.eq) : 0ll;
            neg[c] = (unsigned long long)(qq >> 63);
            mag[c] = ((unsigned long long)qq ^ neg[c]) - neg[c];
          }
          auto add = [&](int rel, int jk, int i) {
            const unsigned long long w = __umul64hi(swyz[warp][jk], sw[warp][i]);
            const int r = cb * R3 + origin + rel;
#pragma unroll
            for (int c = 0; c < 3; ++c)
              if (c < nc) {
                const unsigned long long v = (__umul64hi(w, mag[c]) + round) >> sc.s;
                atomic_add_split64(sacc_lo, sacc_hi, c * R3 + r, (v ^ neg[c]) - neg[c]);
              }
          };
          if constexpr (kHeld) {
#pragma unroll
            for (int t = 0; t < NI; ++t)
              if (t < NI - 1 || lane + 32 * t < W * W * W)
                add((int)(held[t] & 0xfffu), (int)((held[t] >> 12) & 0xffu), (int)(held[t] >> 20));
          } else {
            for (int idx = lane; idx < W * W * W; idx += 32) {
              int rel, jk, i;
              node(idx, rel, jk, i);
              add(rel, jk, i);
            }
          }
        }
        __syncwarp();
      }
      __syncthreads();
      for (int e = threadIdx.x; e < cg * R3; e += blockDim.x) {
        const unsigned long long v = ((unsigned long long)sacc_hi[e] << 32) | sacc_lo[e];
        if (v == 0ull) continue;
        const int cc = e / R3, r = e - cc * R3;
        const int rx = r % R, ry = (r / R) % R, rz = r / (R * R);
        // the region may pass the end of an axis (and, for a window wider than a small
        // axis, wrap more than once): several region nodes can land on one grid node
        const int64_t x = (tx + rx) % g.n[0], y = (ty + ry) % g.n[1], z = (tz + rz) % g.n[2];
        atomicAdd(acc + npf * (c0 + cc) + z * nxy + y * g.n[0] + x, v);
      }
      __syncthreads();
    }
  }
}

// v * 2^e rounded once, from the integer's bits (a conversion and a scaling run at the FP64 rate: 0.59 ms at
// 256^3 x 3 against 0.19); what lies outside the normal range is left to ldexp.
template <typename T>
__device__ __forceinline__ T scaled_integer(long long v, int e) {
  constexpr int kBits = sizeof(T) == 8 ? 53 : 24, kDrop = 64 - kBits, kBias = sizeof(T) == 8 ? 1023 : 127;
  if (v == 0) return T(0);
  const unsigned long long sign = (unsigned long long)v >> 63;
  unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int up = __clzll((long long)a);
  a <<= up;
  const int biased = 63 - up + e + kBias;  // of the leading bit
  if (biased < 1 || biased > 2 * kBias - 1) return (T)ldexp((double)v, e);
  const unsigned long long half = 1ull << (kDrop - 1), rem = a & ((1ull << kDrop) - 1ull);
  unsigned long long man = a >> kDrop;
  man += (unsigned long long)(rem > half || (rem == half && (man & 1ull)));
  // the leading bit adds one to the exponent's field, a carry out of the mantissa another
  const unsigned long long bits = ((unsigned long long)(biased - 1) << (kBits - 1)) + man;
  if constexpr (sizeof(T) == 8) return __longlong_as_double((long long)(bits | sign << 63));
  else return __uint_as_float((uint32_t)(bits | sign << 31));
}

// The oversampled field from the fixed-point sums (NaN everywhere for a non-finite q,
// which the FFT would spread over every mode anyway).
template <typename T>
__global__ void __launch_bounds__(kNThreads)
    k_nufft_finish(const unsigned long long *__restrict__ acc, int64_t n, int64_t m,
                   const unsigned long long *__restrict__ qmax_bits, T *__restrict__ field, int32_t *status) {
  const double qmax = __longlong_as_double((long long)*qmax_bits);
  const bool finite = isfinite(qmax);  // a non-finite quantity is not an error: it yields NaN
  const SpreadScale sc = spread_scale(*qmax_bits, m);
  const int e = sc.eq + sc.s - 56;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    field[i] = finite ? scaled_integer<T>((long long)acc[i], e) : nan_t<T>();
}

gbg_status check_ngrid(const gbg_grid *g) {
  if (!g) return set_error(GBG_EARG, "null grid");
  for (int a = 0; a < 3; ++a) {
    if (g->n[a] <= 0) return set_error(GBG_EARG, "grid_size must be positive along every axis");
    if (!(std::isfinite(g->spacing[a]) && g->spacing[a] > 0))
      return set_error(GBG_EARG, "grid_spacing must be finite and positive along every axis");
    if (!std::isfinite(g->origin[a])) return set_error(GBG_EARG, "origin must be finite along every axis");
    if (g->n[a] > (int64_t(1) << 30)) return set_error(GBG_EUNSUPPORTED, "grid axis longer than 2^30");
  }
  return GBG_OK;
}

gbg_status check_nufft(const gbg_grid *g, gbg_dtype dtype, int32_t ncomp, int64_t m, int32_t width, double beta) {
  GBG_TRY(check_ngrid(g));
  if (dtype != GBG_F32 && dtype != GBG_F64) return set_error(GBG_EARG, "dtype must be GBG_F32 or GBG_F64");
  if (ncomp < 1) return set_error(GBG_EARG, "ncomp must be at least 1");
  if (m < 0) return set_error(GBG_EDIM, "negative point count");
  if (width < 1) return set_error(GBG_EARG, "NUFFT window_width must be a positive number of nodes");
  if (width > kMaxWidth) return set_error(GBG_EUNSUPPORTED, "NUFFT window_width above 16 nodes");
  if (!(std::isfinite(beta) && beta > 0)) return set_error(GBG_EARG, "NUFFT window_shape must be finite and positive");
  return GBG_OK;
}

// Calls f(std::integral_constant<int, W>) for the run-time width 1..16.
template <typename F>
gbg_status with_width(int32_t width, F &&f) {
  switch (width) {
#define GBG_W(N) \
  case N: return f(std::integral_constant<int, N>{});
    GBG_W(1) GBG_W(2) GBG_W(3) GBG_W(4) GBG_W(5) GBG_W(6) GBG_W(7) GBG_W(8)
    GBG_W(9) GBG_W(10) GBG_W(11) GBG_W(12) GBG_W(13) GBG_W(14) GBG_W(15) GBG_W(16)
#undef GBG_W
    default: return set_error(GBG_EUNSUPPORTED, "NUFFT window_width outside 1..16");
  }
}

// Interpolation.jl:1652-1662 -- _es_window_transform: psi_hat(omega) by the trapezoidal
// rule in theta (z = sin(theta)), in T.
template <typename T>
T es_window_transform(T omega, T beta, int width, int quadrature_points) {
  const T half_width = T(width) / T(2);
  const T pi = T(3.141592653589793238462643383279502884);
  T accumulated = T(0);
  for (int q = 0; q <= quadrature_points; ++q) {
    const T theta = -pi / T(2) + pi * T(q) / T(quadrature_points);
    const T trapezoidal = (q == 0 || q == quadrature_points) ? T(1) / T(2) : T(1);
    accumulated += trapezoidal * std::exp(beta * (std::cos(theta) - T(1))) * std::cos(omega * half_width * std::sin(theta)) *
                   std::cos(theta);
  }
  return half_width * (pi / T(quadrature_points)) * accumulated;
}

template <typename T>
void deconvolution_axis(int64_t n, int64_t stored, bool is_half, int sigma, int width, T beta, double *out) {
  const T pi = T(3.141592653589793238462643383279502884);
  for (int64_t i = 0; i < stored; ++i) {
    const int64_t f = (is_half || i < (n + 1) / 2) ? i : i - n;
    const T omega = T(2) * pi * T(f) / (T(sigma) * T(n));
    out[i] = (double)(T(1) / es_window_transform<T>(omega, beta, width, 256));
  }
  if (n % 2 == 0) out[is_half ? stored - 1 : n / 2] = 0.0;
}

}  // namespace
}  // namespace gbg

using namespace gbg;

extern "C" {

gbg_status gbg_nufft_deconvolution_axis(int64_t n, int32_t is_half, int32_t oversampling, int32_t width,
                                        double beta, gbg_dtype dtype, double *host_out) {
  clear_error();
  if (n < 1) return set_error(GBG_EARG, "grid_size must be positive");
  if (oversampling < 2) return set_error(GBG_EARG, "NUFFT oversampling must be at least 2");
  if (width < 1) return set_error(GBG_EARG, "NUFFT window_width must be a positive number of nodes");
  if (!(std::isfinite(beta) && beta > 0)) return set_error(GBG_EARG, "NUFFT window_shape must be finite and positive");
  if (dtype != GBG_F32 && dtype != GBG_F64) return set_error(GBG_EARG, "dtype must be GBG_F32 or GBG_F64");
  if (!host_out) return set_error(GBG_EARG, "null output");
  const int64_t stored = is_half ? n / 2 + 1 : n;
  if (dtype == GBG_F64)
    deconvolution_axis<double>(n, stored, is_half != 0, oversampling, width, beta, host_out);
  else
    deconvolution_axis<float>(n, stored, is_half != 0, oversampling, width, (float)beta, host_out);
  return GBG_OK;
}

}  // extern "C"

namespace gbg {
namespace {

struct SpreadLayout {
  unsigned long long *acc = nullptr, *qmax = nullptr;
  uint32_t *tcount = nullptr, *scan_tmp = nullptr, *tkey = nullptr, *rank = nullptr, *order = nullptr;
  int32_t *first = nullptr;
  unsigned long long *wbuf = nullptr;
  int64_t nt0 = 0, nt1 = 0, nt2 = 0, ntiles = 0;
};

// The spread's workspace, in order: node sums (ncomp per node), max|q|, tile counts (+ the
// extra bucket and the end), scan scratch, per visit slot its tile, rank and place, first
// stencil nodes (3) and fixed-point window weights (3 W).  With base == nullptr it only sizes.
size_t spread_layout(char *base, const gbg_grid &fine, gbg_dtype dtype, int32_t ncomp, int64_t m, int32_t width,
                     SpreadLayout &L, bool spread = true) {
  Arena a;
  a.base = base;
  L.nt0 = (fine.n[0] + kTile - 1) / kTile;
  L.nt1 = (fine.n[1] + kTile - 1) / kTile;
  L.nt2 = (fine.n[2] + kTile - 1) / kTile;
  L.ntiles = L.nt0 * L.nt1 * L.nt2;
  const int64_t npf = fine.n[0] * fine.n[1] * fine.n[2];
  if (spread) {
    L.acc = a.take<unsigned long long>((size_t)(npf * ncomp));
    L.qmax = a.take<unsigned long long>(1);
  }
  L.tcount = a.take<uint32_t>((size_t)L.ntiles + 2);
  L.scan_tmp = a.take<uint32_t>(scan_temp_elems(L.ntiles + 2));
  const size_t mm = (size_t)(m > 0 ? m : 1);
  L.tkey = a.take<uint32_t>(mm);
  L.rank = a.take<uint32_t>(mm);
  L.order = a.take<uint32_t>(mm);
  L.first = a.take<int32_t>(3 * mm);
  if (spread && dtype == GBG_F64) L.wbuf = a.take<unsigned long long>(3 * (size_t)width * mm);
  return a.used + 256;
}

// The tiled gather: bin, place, then a CTA per tile over the staged region.
template <typename T, int W>
gbg_status gather_run(const gbg_grid &fine, int32_t ncomp, const T *field, const T *pos, int64_t m,
                      const int32_t *trav, double beta, T *out, const SpreadLayout &L, int32_t *status,
                      cudaStream_t st) {
  const NGrid<T> g = make_ngrid<T>(fine);
  k_nufft_bin<T, W><<<launch_blocks(m, kNThreads), kNThreads, 0, st>>>(
      g, pos, m, (T)beta, L.nt0, L.nt1, L.ntiles, trav, L.tcount, L.tkey, L.rank, L.first, nullptr, status, ExpTable{}, out,
      ncomp);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  GBG_TRY(exclusive_scan_u32(L.tcount, L.tcount, L.ntiles + 2, L.scan_tmp, st));
  k_nufft_place<<<launch_blocks(m, kNThreads), kNThreads, 0, st>>>(m, L.tkey, L.rank, L.tcount, L.order);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  constexpr int R = kTile + W - 1;
  const size_t slice = sizeof(T) * (size_t)R * R * R;
  // components per pass: as many region slices as fit in 96 KB (two CTAs per SM), at least one
  const int group = (int)std::max<size_t>(1, std::min<size_t>((size_t)ncomp, 98304 / slice));
  const size_t smem = slice * group;
  auto kernel = k_nufft_gather_tiles<T, W>;
  GBG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 1, sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kNThreads, smem);
  const int blocks = (int)std::min<int64_t>(L.ntiles, (int64_t)sms * std::max(per_sm, 1));
  mark_main_start(st);
  kernel<<<blocks, kNThreads, smem, st>>>(g, field, pos, m, ncomp, group, (T)beta, trav, L.nt0, L.nt1, L.ntiles,
                                         L.tcount, L.order, L.first, out);
  mark_main_stop(st);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  return GBG_OK;
}

template <typename T, int W>
gbg_status spread_run(const gbg_grid &fine, int32_t ncomp, T *field, const T *pos, int64_t m, const T *q,
                      const int32_t *trav, double beta, const SpreadLayout &L, int32_t *status, cudaStream_t st) {
  const NGrid<T> g = make_ngrid<T>(fine);
  const int64_t n = fine.n[0] * fine.n[1] * fine.n[2] * (int64_t)ncomp;
  if (m > 0) {
    const int64_t nq = m * (int64_t)ncomp;
    k_nufft_qmax<T><<<launch_blocks(nq, kNThreads), kNThreads, 0, st>>>(q, nq, L.qmax);
    note_launch();
    k_nufft_bin<T, W><<<launch_blocks(m, kNThreads), kNThreads, 0, st>>>(
        g, pos, m, (T)beta, L.nt0, L.nt1, L.ntiles, trav, L.tcount, L.tkey, L.rank, L.first, L.wbuf, status,
        make_exp_table());
    note_launch();
    GBG_CUDA_TRY(cudaGetLastError());
    GBG_TRY(exclusive_scan_u32(L.tcount, L.tcount, L.ntiles + 2, L.scan_tmp, st));
    k_nufft_place<<<launch_blocks(m, kNThreads), kNThreads, 0, st>>>(m, L.tkey, L.rank, L.tcount, L.order);
    note_launch();
    GBG_CUDA_TRY(cudaGetLastError());
    constexpr int R = kTile + W - 1;
    const size_t slice = sizeof(unsigned long long) * (size_t)R * R * R;
    // components per pass: as many region slices as fit in 96 KB (two CTAs per SM), at least one
    const int group = (int)std::max<size_t>(1, std::min<size_t>({(size_t)ncomp, (size_t)kMaxGroup, 98304 / slice}));
    const size_t smem = slice * group;
    auto kernel = k_nufft_spread_tiles<T, W>;
    GBG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 1, sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kNThreads, smem);
    const int blocks = (int)std::min<int64_t>(L.ntiles, (int64_t)sms * std::max(per_sm, 1));
    mark_main_start(st);
    kernel<<<blocks, kNThreads, smem, st>>>(g, pos, (T)beta, m, q, trav, ncomp, group, L.nt0, L.nt1, L.ntiles, L.tcount, L.order, L.first, L.wbuf, L.qmax, L.acc);
    mark_main_stop(st);
    note_launch();
    GBG_CUDA_TRY(cudaGetLastError());
  }
  k_nufft_finish<T><<<launch_blocks(n, kNThreads), kNThreads, 0, st>>>(L.acc, n, m > 0 ? m : 1, L.qmax, field, status);
  note_launch();
  GBG_CUDA_TRY(cudaGetLastError());
  return GBG_OK;
}

}  // namespace
}  // namespace gbg

extern "C" {

gbg_status gbg_nufft_interp_workspace_size(const gbg_grid *fine, gbg_dtype dtype, int32_t ncomp, int64_t npoints,
                                           int32_t width, size_t *bytes) {
  clear_error();
  GBG_TRY(check_nufft(fine, dtype, ncomp, npoints, width, 1.0));
  if (!bytes) return set_error(GBG_EARG, "null bytes");
  SpreadLayout L;
  *bytes = spread_layout(nullptr, *fine, dtype, ncomp, npoints, width, L, false);
  return GBG_OK;
}

gbg_status gbg_nufft_interp(const gbg_grid *fine, gbg_dtype dtype, int32_t ncomp, const void *field,
                            const void *positions, int64_t npoints, const int32_t *traversal, int32_t width,
                            double beta, void *out, void *workspace, size_t workspace_bytes, int32_t *device_status,
                            void *stream) {
  clear_error();
  try {
    GBG_TRY(check_nufft(fine, dtype, ncomp, npoints, width, beta));
    if (npoints == 0) return GBG_OK;
    if (!field || !positions || !out) return set_error(GBG_EARG, "nufft_interp: null array");
    if (npoints > 0x7fffffffLL) return set_error(GBG_EUNSUPPORTED, "nufft_interp: more than 2^31-1 points");
    size_t need = 0;
    GBG_TRY(gbg_nufft_interp_workspace_size(fine, dtype, ncomp, npoints, width, &need));
    if (!workspace || workspace_bytes < need) return set_error(GBG_ENOMEM, "nufft_interp: workspace too small");
    if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
      return set_error(GBG_EARG, "nufft_interp: workspace not 256-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    SpreadLayout L;
    spread_layout(static_cast<char *>(workspace), *fine, dtype, ncomp, npoints, width, L, false);
    GBG_CUDA_TRY(cudaMemsetAsync(L.tcount, 0, sizeof(uint32_t) * ((size_t)L.ntiles + 2), st));
    return with_width(width, [&](auto wc) -> gbg_status {
      constexpr int W = decltype(wc)::value;
      if (dtype == GBG_F64) {
        mark_main_start(st);
        k_nufft_gather<W><<<launch_blocks(npoints, kNThreads), kNThreads, 0, st>>>(
            make_ngrid<double>(*fine), make_exp_table(), static_cast<const double *>(field), static_cast<const double *>(positions),
            npoints, ncomp, beta, traversal, static_cast<double *>(out), device_status);
        mark_main_stop(st);
        note_launch();
        GBG_CUDA_TRY(cudaGetLastError());
        return GBG_OK;
      }
      return gather_run<float, W>(*fine, ncomp, static_cast<const float *>(field), static_cast<const float *>(positions),
                                  npoints, traversal, beta, static_cast<float *>(out), L, device_status, st);
    });
  } catch (...) {
    return set_error(GBG_ENOMEM, "nufft_interp: host exception");
  }
}

gbg_status gbg_nufft_spread_workspace_size(const gbg_grid *fine, gbg_dtype dtype, int32_t ncomp, int64_t npoints,
                                           int32_t width, size_t *bytes) {
  clear_error();
  GBG_TRY(check_nufft(fine, dtype, ncomp, npoints, width, 1.0));
  if (!bytes) return set_error(GBG_EARG, "null bytes");
  SpreadLayout L;
  *bytes = spread_layout(nullptr, *fine, dtype, ncomp, npoints, width, L);
  return GBG_OK;
}

gbg_status gbg_nufft_spread(const gbg_grid *fine, gbg_dtype dtype, int32_t ncomp, void *field,
                            const void *positions, int64_t npoints, const void *quantities,
                            const int32_t *traversal, int32_t width, double beta, void *workspace,
                            size_t workspace_bytes, int32_t *device_status, void *stream) {
  clear_error();
  try {
    GBG_TRY(check_nufft(fine, dtype, ncomp, npoints, width, beta));
    size_t need = 0;
    GBG_TRY(gbg_nufft_spread_workspace_size(fine, dtype, ncomp, npoints, width, &need));
    if (!field) return set_error(GBG_EARG, "nufft_spread: null field");
    if (npoints > 0 && (!positions || !quantities)) return set_error(GBG_EARG, "nufft_spread: null array");
    if (npoints > 0x7fffffffLL) return set_error(GBG_EUNSUPPORTED, "nufft_spread: more than 2^31-1 points");
    if (!workspace || workspace_bytes < need) return set_error(GBG_ENOMEM, "nufft_spread: workspace too small");
    // the layout aligns its pieces to 256 bytes from the workspace's start
    if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
      return set_error(GBG_EARG, "nufft_spread: workspace not 256-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    SpreadLayout L;
    spread_layout(static_cast<char *>(workspace), *fine, dtype, ncomp, npoints, width, L);
    const int64_t n = fine->n[0] * fine->n[1] * fine->n[2] * (int64_t)ncomp;
    GBG_CUDA_TRY(cudaMemsetAsync(L.acc, 0, (size_t)n * 8, st));
    GBG_CUDA_TRY(cudaMemsetAsync(L.qmax, 0, 8, st));
    GBG_CUDA_TRY(cudaMemsetAsync(L.tcount, 0, sizeof(uint32_t) * ((size_t)L.ntiles + 2), st));
    return with_width(width, [&](auto wc) -> gbg_status {
      constexpr int W = decltype(wc)::value;
      if (dtype == GBG_F64)
        return spread_run<double, W>(*fine, ncomp, static_cast<double *>(field), static_cast<const double *>(positions),
                                     npoints, static_cast<const double *>(quantities), traversal, beta, L,
                                     device_status, st);
      return spread_run<float, W>(*fine, ncomp, static_cast<float *>(field), static_cast<const float *>(positions),
                                  npoints, static_cast<const float *>(quantities), traversal, beta, L, device_status,
                                  st);
    });
  } catch (...) {
    return set_error(GBG_ENOMEM, "nufft_spread: host exception");
  }
}

}  // extern "C"
