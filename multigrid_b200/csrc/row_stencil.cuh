// One point's stencil row held by the thread that owns the point, for the
// kernels that keep a small level on chip (cg_cluster.cuh,
// bottom_cluster.cuh): the couplings are loaded once, so a smoothing step or
// a product with A reads only the vector's neighbours.
#pragma once

#include <math.h>
#include <string.h>

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

// ---- division by a divisor that is divided by many times --------------------
// s / c, the bits of the IEEE divide, from y = recip_of(c): two residual
// corrections of the product s y. The first leaves q within an ulp of the
// quotient, so the second gives it correctly rounded (Markstein, IBM J. Res.
// Dev. 34, 1990): five dependent operations (a double divide is ~110 cycles,
// these ~40). That needs y correctly rounded, s - q c exact and the quotient
// normal, which holds where c_min <= c <= c_max and q_min <= |s y| <= q_max:
// then |s| lies between 2^-100 and 2^126 (2^-700 and 2^700 in double), and
// s - q c, a multiple of 2^-47 (2^-105) of s, does not underflow. Everything
// else takes the divide: infinities, NaN, tiny and huge numerators and
// divisors out of range (their reciprocal is NaN here). A zero numerator,
// frequent on a zero-started level, does not: the residual is taken negated,
// q c - s, so that the zero keeps its sign. The range test is one integer
// subtraction and comparison (of the upper half of a double).
template <typename T> struct DivRange;
template <> struct DivRange<float> {
  static constexpr float c_min = 0x1p-30f, c_max = 0x1p40f;
  static constexpr float q_min = 0x1p-70f, q_max = 0x1p86f;
  // twice the bits of the sizes
  static constexpr unsigned key_min = (127u - 70u) << 24,
                            key_max = (127u + 86u) << 24;
};
template <> struct DivRange<double> {
  static constexpr double c_min = 0x1p-200, c_max = 0x1p200;
  static constexpr double q_min = 0x1p-500, q_max = 0x1p500;
  static constexpr unsigned key_min = (1023u - 500u) << 21,
                            key_max = (1023u + 500u) << 21;
};
template <typename T> __host__ __device__ __forceinline__ T recip_of(T c) {
  using R = DivRange<T>;
  return c >= R::c_min && c <= R::c_max ? T(1) / c : T(NAN);
}
__host__ __device__ __forceinline__ unsigned size_key(float v) {
  unsigned u;
  memcpy(&u, &v, sizeof(u));
  return 2u * u;
}
__host__ __device__ __forceinline__ unsigned size_key(double v) {
  unsigned long long u;
  memcpy(&u, &v, sizeof(u));
  return 2u * (unsigned)(u >> 32);
}
template <typename T>
__host__ __device__ __forceinline__ T div_by_recip(T s, T c, T y) {
  using R = DivRange<T>;
  const T q0 = s * y;
  T q = fma(-fma(q0, c, -s), y, q0);
  q = fma(-fma(q, c, -s), y, q);
  const bool outside = size_key(q0) - R::key_min > R::key_max - R::key_min;
  const bool zero = (s == T(0)) & (q0 == T(0));
  if (__builtin_expect(outside & !zero, 0))
    q = s / c;
  return q;
}

// s / c in float, the bits of the IEEE divide for every s and c without a
// test: the double product of s with 1 / c held as hi + lo, rounded to float.
// hi is 1 / c rounded towards zero and lo the rest, of the same sign (never
// zero, so that an infinite s stays one and a zero keeps its sign). The fused
// sum is s / c rounded once to double up to 2^-104 of it. A quotient that is
// a float, or lies midway between two (only where those are subnormal), is a
// double with room to spare and comes out exactly; any other quotient of two
// 24-bit significands is at least 2^-49 of itself away from every such value,
// so both roundings end at the same float.
struct RecipPair {
  double hi, lo;
};
__host__ __device__ __forceinline__ RecipPair recip_pair(float c) {
  const double d = c;
  double hi = 1.0 / d;
  if (!(hi - hi == 0.0) || hi == 0.0) // c is zero, infinite or NaN
    return RecipPair{hi, hi};
  double rest = fma(-d, hi, 1.0); // exact
  if (rest < 0.0) { // hi was rounded away from zero: the next towards it
    unsigned long long u;
    memcpy(&u, &hi, sizeof(u));
    --u;
    memcpy(&hi, &u, sizeof(hi));
    rest = fma(-d, hi, 1.0);
  }
  return RecipPair{hi, rest == 0.0 ? hi * 0x1p-200 : rest * hi};
}
__host__ __device__ __forceinline__ float div_by_pair(float s, RecipPair r) {
  const double v = s;
  return (float)fma(v, r.hi, v * r.lo);
}

// Sum of v over the warp, the same bits in every lane.
__device__ __forceinline__ double warp_allsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

} // namespace pmg
