// One point's stencil row held by the thread that owns the point, for the
// kernels that keep a small level on chip (cg_cluster.cuh,
// bottom_cluster.cuh): the couplings are loaded once, so a smoothing step or
// a product with A reads only the vector's neighbours.
#pragma once

#include "pmg_common.cuh"

namespace pmg {

struct Offset3 {
  int x, y, z;
};

// Neighbour t of the 27-point stencil in the order sums27 adds them: eight
// in the plane, nine above, nine below.
__host__ __device__ constexpr Offset3 neighbour27(int t) {
  const int q = t < 8 ? t + 1 : t < 17 ? t - 8 : t - 17;
  const int z = t < 8 ? 0 : t < 17 ? 1 : -1;
  // C N S E W NE NW SE SW
  const int x = (q == 3 || q == 5 || q == 7) ? 1
                : (q == 4 || q == 6 || q == 8) ? -1
                                               : 0;
  const int y = (q == 1 || q == 5 || q == 6) ? 1
                : (q == 2 || q == 7 || q == 8) ? -1
                                               : 0;
  return Offset3{x, y, z};
}
// The same for the 7-point stencil (apply7's order: N S E W D U).
__host__ __device__ constexpr Offset3 neighbour7(int t) {
  return Offset3{t == 2 ? 1 : t == 3 ? -1 : 0, t == 0 ? 1 : t == 1 ? -1 : 0,
                 t == 5 ? 1 : t == 4 ? -1 : 0};
}
template <int KIND>
__host__ __device__ constexpr Offset3 neighbour(int t) {
  return KIND == 27 ? neighbour27(t) : neighbour7(t);
}

// The couplings of one point (positive, in neighbour order) and its centre
// coefficient oC + cc.
template <typename T, int KIND> struct StencilRow {
  static constexpr int N = KIND - 1;
  T c[N];
  T centre;

  __device__ __forceinline__ void load(const Op14<T> &A, const T *cc, int p,
                                       int sy, int sz) {
#pragma unroll
    for (int t = 0; t < N; ++t) {
      const Offset3 e = neighbour<KIND>(t);
      const int s = upper_slot(e.x, e.y, e.z);
      c[t] = s ? A.a[s][p]
               : A.a[upper_slot(-e.x, -e.y, -e.z)][p + e.x + e.y * sy +
                                                   e.z * sz];
    }
    centre = A.a[kOC][p] + (cc ? cc[p] : T(0));
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int t = 0; t < N; ++t)
      c[t] = T(0);
    centre = T(0);
  }

  // A v with v(dx, dy, dz) the vector at the neighbour: products and sums in
  // the order of apply7 / apply27, rounded separately
  template <class V> __device__ __forceinline__ T apply(V v) const {
    if constexpr (KIND == 27) {
      T s[3];
      sums(v, s);
      return (-s[0]) + (-s[1]) + (-s[2]) + centre * v(0, 0, 0);
    } else {
      T s = -c[0] * at<0>(v);
      s = s - c[1] * at<1>(v);
      s = s - c[2] * at<2>(v);
      s = s - c[3] * at<3>(v);
      s = s - c[4] * at<4>(v);
      s = s - c[5] * at<5>(v);
      return s + centre * v(0, 0, 0);
    }
  }
  // A v with fused products and four shorter chains, for the solves that are
  // held to rounding and not to bits
  template <class V> __device__ __forceinline__ T apply_fused(V v) const {
    T s[4] = {centre * v(0, 0, 0), T(0), T(0), T(0)};
#pragma unroll
    for (int t = 0; t < N; ++t) {
      const Offset3 e = neighbour<KIND>(t);
      s[t & 3] = fma(-c[t], v(e.x, e.y, e.z), s[t & 3]);
    }
    return (s[0] + s[1]) + (s[2] + s[3]);
  }
  // f + neighbour sums, fused in four chains
  template <class V> __device__ __forceinline__ T fused_sum(T f, V v) const {
    T s[4] = {f, T(0), T(0), T(0)};
#pragma unroll
    for (int t = 0; t < N; ++t) {
      const Offset3 e = neighbour<KIND>(t);
      s[t & 3] = fma(c[t], v(e.x, e.y, e.z), s[t & 3]);
    }
    return (s[0] + s[1]) + (s[2] + s[3]);
  }
  // f - A v in the order of resid_at (Vmresid7_1s, Vmresid27_1s)
  template <class V> __device__ __forceinline__ T resid(T f, V v) const {
    if constexpr (KIND == 27) {
      T s[3];
      sums(v, s);
      return f + s[0] + s[1] + s[2] - centre * v(0, 0, 0);
    } else {
      T s = f + c[0] * at<0>(v);
      s = s + c[1] * at<1>(v);
      s = s + c[2] * at<2>(v);
      s = s + c[3] * at<3>(v);
      s = s + c[4] * at<4>(v);
      s = s + c[5] * at<5>(v);
      return s - centre * v(0, 0, 0);
    }
  }
  // the three partial sums of sums27: in the plane, above, below
  template <class V> __device__ __forceinline__ void sums(V v, T *s) const {
    static_assert(KIND == 27, "three plane sums");
    T w[N];
#pragma unroll
    for (int t = 0; t < N; ++t) {
      const Offset3 e = neighbour27(t);
      w[t] = v(e.x, e.y, e.z);
    }
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      const int t0 = g == 0 ? 0 : g == 1 ? 8 : 17;
      const int t1 = g == 0 ? 8 : g == 1 ? 17 : 26;
      T a = c[t0] * w[t0];
#pragma unroll
      for (int t = 1; t < 9; ++t)
        if (t0 + t < t1)
          a = a + c[t0 + t] * w[t0 + t];
      s[g] = a;
    }
  }

private:
  template <int K, class V> static __device__ __forceinline__ T at(V v) {
    constexpr Offset3 e = neighbour<KIND>(K);
    return v(e.x, e.y, e.z);
  }
};

// s / c from y, the reciprocal of c rounded to nearest: two residual
// corrections of the product s y. The first leaves q within an ulp of the
// quotient, so the second gives it correctly rounded (Markstein, IBM J. Res.
// Dev. 34, 1990), the bits of the divide, in five dependent operations (a
// double divide is ~110 cycles, these ~40).
__device__ __forceinline__ double div_by_recip(double s, double c, double y) {
  double q = s * y;
  q = __fma_rn(__fma_rn(-q, c, s), y, q);
  return __fma_rn(__fma_rn(-q, c, s), y, q);
}
__device__ __forceinline__ float div_by_recip(float s, float c, float y) {
  float q = s * y;
  q = __fmaf_rn(__fmaf_rn(-q, c, s), y, q);
  return __fmaf_rn(__fmaf_rn(-q, c, s), y, q);
}

// Sum of v over the warp, the same bits in every lane.
__device__ __forceinline__ double warp_allsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

} // namespace pmg
