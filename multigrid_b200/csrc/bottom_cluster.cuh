// The lowest levels of a V-cycle in one launch, on a cluster of CTAs with
// every iterate on chip.
//
// Levels 1 .. top (n_top <= 17, the levels below it n <= 9) hold less work
// than a launch costs: the part of the cycle below 33^3 was 30 to 100
// launches, or, in one kernel with couplings and iterates read through shared
// memory and neighbouring planes through remote loads, 105 us of barriers and
// load latency. What bounds it is the chain of dependent steps: 32 colour
// steps per level and cycle, the coarsest CG, and the hops between CTAs.
// Each is kept as short as it can be:
//   * every thread owns one point of the top level and holds its couplings,
//     right-hand side and centre reciprocal in registers (row_stencil.cuh);
//     a colour step is 26 shared loads at immediate offsets, one product sum,
//     a divide by two corrected products, one store;
//   * a plane of the top level belongs to eight warps, two per colour, whose
//     rows of eight points fall into different banks (rows split by the
//     parity of i, pitch 20); they meet at a barrier of their own;
//   * the planes exchange values by messages (mbar.cuh): a point's new value
//     is stored into the copies that the planes above and below keep, and a
//     plane starts when the bytes it expects have arrived. No CTA reads
//     another's memory and none waits at a cluster barrier in the cycle;
//   * rank 0 receives the top level's defect as messages, runs the levels
//     below alone (all of its threads, one point each) and sends the coarse
//     iterate to every CTA, which interpolates its own planes.
// The order of the messages: an even plane waits for its odd neighbours and
// an odd plane for its even ones, so a sender can be at most one phase ahead
// of a receiver and only after the receiver has all bytes of its own phase
// (an even plane's interpolated values are not sent: its odd neighbours read
// it only after its next sweep). A wait must also be over in every warp of
// the plane before the plane sends what the mbarrier's next phase depends on:
// a warp that polls only after that phase has completed too sees the parity
// it waits for as not yet reached. In a sweep the colours' barriers see to
// that; the wait before the defect has a barrier of its own, because a warp
// without a point (every other one where the top level has at most 9 points
// per axis) sends nothing that would hold the others back.
// Measured per cycle: 105 us (levels 5^3, 9^3, 17^3 of a 257^3 mixed solve) ->
// 35 us, 90 -> 27 us at 65^3; in double, where these levels were 31 launches,
// 250 -> 46 us (129^3). The same kernel serves many concurrent solves: one CTA
// out of global memory per solve, which needs no eight idle SMs at once, gave
// 229 against 232 solves/s on 96 molecules and 210 against 219 in the serving
// loop, with p50 10.0 against 7.4 ms at a quarter of the saturation.
//
// The steps are the V-cycle's (v_cycle, PBE_pmgc_class.h:1070-1114, every
// level but the first zero-started) with the arithmetic of the per-level
// kernels; sums over threads and CTAs run in a fixed order. The level-1 CG is
// the class's (cg_cluster.cuh).
#pragma once

#include <cooperative_groups.h>
#include <stddef.h>

#include "cg_cluster.cuh"

namespace pmg {

constexpr int kBottomMaxLevels = 4;
constexpr int kBottomMaxN = 17;

template <typename T> struct BottomLevel {
  Dims d;
  Op14<T> A;       // level operator, unused on level 1
  P27<T> P;        // prolongation from this level to the next finer one
  T *x;            // iterate (the top level's is the result)
  const T *f;      // right-hand side of the top level
  double *omega;   // damping computed on this level
};

template <typename T> struct BottomArgs {
  int top; // finest level handled here (<= 4)
  BottomLevel<T> lv[kBottomMaxLevels + 1];
  Op14<double> A1; // level-1 operator (double)
  double *x1;      // level-1 iterate (double), kept between cycles
  // CG stop (cg_cluster.cuh): absolute and relative, the class's first test;
  // started from zero or from the x1 of the last cycle
  double thresh, rtol;
  int class_first_check, warm_start;
  int max_iters;
  int *status;
  int *kernel_err; // set when a message did not arrive
  // the inverse of level 1's interior operator where it is kept (null: CG)
  // and whether it may be used
  const double *inv;
  const int *inv_ok;
  // a test's delay of the warps without a point before they wait for the
  // values that the defect reads, in units of 16 us (0: none)
  int idle_delay;
  unsigned extra_tx; // a test's bytes that no message brings (0)
};

constexpr int kBcThreads = 512;
constexpr int kBcRow = 20, kBcPlane = kBcRow * kCgMaxN; // top level
constexpr int kBlMaxN = 9;                              // levels below it
constexpr int kBlRow = 18, kBlPlane = 168;
constexpr int kBlMaxLevels = 2; // levels 2 .. top-1

// Entry of point i (1-based) in a row split by parity: even i first.
template <int ODD> __host__ __device__ constexpr int split_entry(int i) {
  return (i & 1) ? ODD + (i >> 1) : (i >> 1) - 1;
}
constexpr int kBcOdd = 8, kBlOdd = 4; // even points of a row of 17 and of 9

// A point of a level in shared memory with such rows: entries of its west,
// own and east column in its row and plane.
template <int ROW, int PLANE> struct SplitPoint {
  int w, c, e;
  template <typename T>
  __device__ __forceinline__ T read(const T *a, int dx, int dy,
                                    int dz) const {
    return a[(dx < 0 ? w : dx > 0 ? e : c) + dy * ROW + dz * PLANE];
  }
};
template <int ROW, int PLANE, int ODD>
__device__ __forceinline__ SplitPoint<ROW, PLANE> split_point(int i, int j,
                                                             int k) {
  const int o = (j - 1) * ROW + k * PLANE;
  return SplitPoint<ROW, PLANE>{o + split_entry<ODD>(i - 1),
                                o + split_entry<ODD>(i),
                                o + split_entry<ODD>(i + 1)};
}

// Level 1 with at most kInvMax unknowns (7^3 points and fewer; the
// refinement paths): the inverse of its interior operator, dense, computed
// when the hierarchy is built. The CG it replaces there runs 11 to 20
// iterations of ~1500 cycles to a residual reduction of 1e-4 on 27 unknowns
// (14 of the kernel's 41 us), and more on 125; the product takes ~1000 cycles
// and solves to rounding.
// In-place Gauss-Jordan without pivoting (the operator is symmetric positive
// definite; *ok = 0 where a pivot is not positive, and the CG runs): 32 x 32
// threads, each with the elements (i, j), i = ti mod 32, j = tj mod 32, in
// registers (one of them for 27 unknowns); each step passes one row and one
// column through shared memory. A build waits for it, so a step is one
// barrier, one multiply-add per element and the row and the column set by the
// threads that hold them (two barriers and a choice of both in every element,
// and four integer divisions each at the start: 252 us for 125 unknowns, 19.5
// for 27; so 85 and 16.5).
constexpr int kInvMax = 125;
__global__ void __launch_bounds__(1024)
    level1_inverse_kernel(Dims d, const __grid_constant__ Op14<double> A,
                          double *__restrict__ inv, int *__restrict__ ok) {
  __shared__ double rowp[2][128], colp[2][128], pivp[2]; // 1 / pivot
  const int mx = d.nx - 2, my = d.ny - 2, m = mx * my * (d.nz - 2);
  const int ti = threadIdx.x & 31, tj = threadIdx.x >> 5;
  // the points of unknown 32 a + t: coordinates and place, -2 past the last
  auto point = [&](int q, int &x, int &y, int &z) {
    const int rq = q / mx;
    z = q < m ? rq / my : -2;
    x = q - rq * mx;
    y = rq - z * my;
  };
  int ix[4], iy[4], iz[4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
    point(ti + 32 * a, ix[a], iy[a], iz[a]);
  double v[4][4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    int jx, jy, jz;
    point(tj + 32 * b, jx, jy, jz);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      v[a][b] = 0.0;
      const int ex = jx - ix[a], ey = jy - iy[a], ez = jz - iz[a];
      if (iz[a] >= 0 && jz >= 0 && abs(ex) <= 1 && abs(ey) <= 1 &&
          abs(ez) <= 1) {
        const int p = d.at(ix[a] + 2, iy[a] + 2, iz[a] + 2);
        const int s = upper_slot(ex, ey, ez);
        v[a][b] = ex == 0 && ey == 0 && ez == 0 ? A.a[kOC][p]
                  : s                           ? -A.a[s][p]
                      : -A.a[upper_slot(-ex, -ey, -ez)]
                            [p + ex + ey * d.sy() + ez * d.sz()];
      }
    }
  }
  bool good = true;
#pragma unroll
  for (int pb = 0; pb < 4; ++pb) { // step p = 32 pb + pl
#pragma unroll 1
    for (int pl = 0; pl < 32 && 32 * pb + pl < m; ++pl) {
      double *row = rowp[pl & 1], *col = colp[pl & 1];
      if (ti == pl)
#pragma unroll
        for (int b = 0; b < 4; ++b)
          row[tj + 32 * b] = v[pb][b];
      if (tj == pl)
#pragma unroll
        for (int a = 0; a < 4; ++a)
          col[ti + 32 * a] = v[a][pb];
      if (ti == pl && tj == pl) {
        pivp[pl & 1] = 1.0 / v[pb][pb];
        good = good && v[pb][pb] > 0.0;
      }
      __syncthreads(); // (the next step's row and column go to the other half)
      const double y = pivp[pl & 1];
      double r[4];
#pragma unroll
      for (int b = 0; b < 4; ++b)
        r[b] = row[tj + 32 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        if (32 * a >= m)
          break;
        const double c = col[ti + 32 * a] * y;
#pragma unroll
        for (int b = 0; b < 4; ++b)
          v[a][b] = fma(-c, r[b], v[a][b]);
        if (tj == pl)
          v[a][pb] = -c;
      }
      if (ti == pl) {
#pragma unroll
        for (int b = 0; b < 4; ++b)
          v[pb][b] = tj == pl && b == pb ? y : y * r[b];
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = ti + 32 * a, j = tj + 32 * b;
      if (i < m && j < m) {
        inv[j * m + i] = v[a][b];
        good = good && isfinite(v[a][b]);
      }
    }
  good = __syncthreads_and(good);
  if (threadIdx.x == 0)
    *ok = good;
}

template <typename T> struct alignas(16) BcSmem {
  // the two plane groups' planes k-1, k, k+1 of x
  T x[2][3 * kBcPlane];
  // level top-1's iterate and its damping, sent by one copy
  alignas(16) T xc[kBlMaxN * kBlMaxN * kBlMaxN];
  double omega;
  double red[2][kBcThreads / 32];
  uint64_t bar_x[2], bar_c; // messages: neighbours' planes, the coarse level
  // rank 0
  uint64_t bar_r, bar_d; // messages: the top level's defect, its damping
  double dsum[kCgMaxN][2];
  T r[(kCgMaxN + 1) * kBcPlane];
  // x and f of the levels between, the defect of one of them
  T lx[kBlMaxLevels][kBlMaxN * kBlPlane];
  T lf[kBlMaxLevels][kBlMaxN * kBlPlane];
  T lr[(kBlMaxN + 1) * kBlPlane];
  T x1[kBlMaxN * kBlMaxN * kBlMaxN]; // level 1
  alignas(16) double p1[kBlMaxN * kCgPlane];
};

template <typename T> bool bc_fits(const BottomArgs<T> &a) {
  if (a.top < 2 || a.top - 2 > kBlMaxLevels)
    return false;
  const Dims &d = a.lv[a.top].d;
  if (d.nx > kCgMaxN || d.ny > kCgMaxN || d.nz > kCgMaxN)
    return false;
  for (int L = 1; L < a.top; ++L) {
    const Dims &c = a.lv[L].d;
    if (c.nx > kBlMaxN || c.ny > kBlMaxN || c.nz > kBlMaxN)
      return false;
  }
  return true;
}

// barrier of `threads` threads of the CTA (whole warps)
__device__ __forceinline__ void named_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// coarse f at (I, J, K) = restriction of the defect r, rows split with ODD
// (restrict_kernel's order), with the point's 27 weights
template <int ROW, int PLANE, int ODD, typename T>
__device__ __forceinline__ T bc_restrict_with(const T *r, const T (&w)[27],
                                              int I, int J, int K) {
  // r holds planes from 1 on
  const auto s =
      split_point<ROW, PLANE, ODD>(2 * I - 1, 2 * J - 1, 2 * K - 2);
  T pl[3];
#pragma unroll
  for (int z = 0; z < 3; ++z) {
    const int dz = z == 0 ? 0 : z == 1 ? 1 : -1;
    // C N S E W NE NW SE SW
    T a = w[z * 9] * s.read(r, 0, 0, dz);
    a = a + w[z * 9 + 1] * s.read(r, 0, 1, dz);
    a = a + w[z * 9 + 2] * s.read(r, 0, -1, dz);
    a = a + w[z * 9 + 3] * s.read(r, 1, 0, dz);
    a = a + w[z * 9 + 4] * s.read(r, -1, 0, dz);
    a = a + w[z * 9 + 5] * s.read(r, 1, 1, dz);
    a = a + w[z * 9 + 6] * s.read(r, -1, 1, dz);
    a = a + w[z * 9 + 7] * s.read(r, 1, -1, dz);
    a = a + w[z * 9 + 8] * s.read(r, -1, -1, dz);
    pl[z] = a;
  }
  return pl[0] + pl[1] + pl[2];
}
template <int ROW, int PLANE, int ODD, typename T>
__device__ __forceinline__ T bc_restrict_at(const T *r, const P27<T> &P,
                                            int pc, int I, int J, int K) {
  T w[27];
#pragma unroll
  for (int q = 0; q < 27; ++q)
    w[q] = P.p[q][pc];
  return bc_restrict_with<ROW, PLANE, ODD>(r, w, I, J, K);
}

// The interpolation weights of one fine point: those of the corners of its
// coarse cell that it lies between (interp_kernel's order).
template <typename T> struct BcInterp {
  T w[8];
  int px, py, pz; // 1 where the fine index is between two coarse ones
  int cc;         // the cell's first corner
  __device__ __forceinline__ void load(const P27<T> &P, const Dims &cd, int i,
                                       int j, int k, bool own) {
    px = (i & 1) ^ 1;
    py = (j & 1) ^ 1;
    pz = (k & 1) ^ 1;
    cc = cd.at((i + 1) >> 1, (j + 1) >> 1, (k + 1) >> 1);
    const int cy = cd.sy(), cz = cd.sz();
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int bx = b & 1, by = (b >> 1) & 1, bz = b >> 2;
      w[b] = T(0);
      if (own && bx <= px && by <= py && bz <= pz)
        w[b] = P.p[pslot(px - 2 * bx, py - 2 * by, pz - 2 * bz)]
                  [cc + bx + by * cy + bz * cz];
    }
  }
  // xc(bx, by, bz): the coarse iterate at a corner
  template <class X> __device__ __forceinline__ T eval(X xc) const {
    if (px + py + pz == 0)
      return xc(0, 0, 0);
    T e = w[0] * xc(0, 0, 0);
#pragma unroll
    for (int b = 1; b < 8; ++b) {
      const int bx = b & 1, by = (b >> 1) & 1, bz = b >> 2;
      if (bx <= px && by <= py && bz <= pz)
        e = e + w[b] * xc(bx, by, bz);
    }
    return e;
  }
};

// (f + neighbour sums) / centre: the colour step at a point. Double: the
// class's products and sums (the FP64 path's bits); float: fused, in four
// chains (half the instructions; the mixed path is held to its tolerance).
template <typename T, class V>
__device__ __forceinline__ T bc_relax(const StencilRow<T, 27> &row, T recip,
                                      T f, V v) {
  if constexpr (sizeof(T) == sizeof(float)) {
    return div_by_recip(row.fused_sum(f, v), row.centre, recip);
  } else {
    T s[3];
    row.sums(v, s);
    return div_by_recip(f + (s[0] + s[1] + s[2]), row.centre, recip);
  }
}

// Level 1 on rank 0 by the inverse of its interior operator
// (level1_inverse_kernel): one point per thread of the CTA's last `threads`.
// The product is the solution to rounding, so its damping (f . x) / (x . A x)
// is 1.
template <typename T>
__device__ __forceinline__ void
bc_level1_direct(const BottomArgs<T> &a, BcSmem<T> &sm, int threads, bool own,
                 int u, int nat, T f) {
  const Dims &d = a.lv[1].d;
  const int m = (d.nx - 2) * (d.ny - 2) * (d.nz - 2);
  double *sf = sm.p1;
  if (own)
    sf[u] = (double)f;
  if (threads == 32)
    __syncwarp();
  else
    named_barrier(3, threads);
  const double *inv = a.inv + (own ? u : 0);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 9
  for (int t = 0; t + 3 <= m; t += 3) { // (m is a cube of an odd number: 1,
    s[0] = fma(inv[t * m], sf[t], s[0]); // 27, 125: three terms a turn and
    s[1] = fma(inv[(t + 1) * m], sf[t + 1], s[1]); // the rest below)
    s[2] = fma(inv[(t + 2) * m], sf[t + 2], s[2]);
  }
  for (int t = m - m % 3; t < m; ++t)
    s[3] = fma(inv[t * m], sf[t], s[3]);
  const T x = (T)((s[0] + s[1]) + (s[2] + s[3]));
  if (own)
    sm.x1[nat] = x;
  a.status[0] = 0;
  a.status[1] = 0;
}

// Level 1 on rank 0: the class's CG on the CTA's last `threads` threads
// (whole warps; one point each; row: the point's couplings), then the
// damping. Leaves the iterate, rounded to T, in x1 and returns omega. The
// products with A (start, search direction, damping) share one piece of
// code: the kernel is so short that fetching instructions counts.
template <typename T>
__device__ __forceinline__ double
bc_level1(const BottomArgs<T> &a, BcSmem<T> &sm, int threads, bool own, int i,
          int j, int k, const StencilRow<double, 27> &row, double f) {
  const Dims &d = a.lv[1].d;
  const int lane = threadIdx.x & 31, nw = threads >> 5;
  const int warp = (threadIdx.x >> 5) - (kBcThreads / 32 - nw);
  double *sP = sm.p1;
  auto barrier = [&]() {
    if (nw == 1)
      __syncwarp();
    else
      named_barrier(3, threads);
  };
  auto allsum = [&](double v, int set) -> double {
    v = warp_allsum(v);
    if (nw == 1)
      return v;
    if (lane == 0)
      sm.red[set][warp] = v;
    barrier();
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int w = 0; w < kBcThreads / 32; ++w)
      if (w < nw)
        s[w & 3] += sm.red[set][w];
    return (s[0] + s[1]) + (s[2] + s[3]);
  };
  const int gi = d.at(i, j, k);
  // (threads without a point stay in bounds; their rows are zero)
  const int sl = (min(k, kBlMaxN - 1) - 1) * kCgPlane + (j - 1) * kCgRow +
                 (i - 1);
  auto pval = [&](int dx, int dy, int dz) {
    return sP[sl + dx + dy * kCgRow + dz * kCgPlane];
  };
  double xv = own && a.warm_start ? a.x1[gi] : 0.0;
  double rv = f, v = xv, rs = 0.0, rs_old = 0.0, stop2 = 0.0, omega = 0.0;
  int it = a.warm_start ? -1 : 0; // -1: A x of the start, -2: of the result
  bool capped = false;
  if (it == 0) {
    rs = allsum(rv * rv, 0);
    v = rv;
  }
#pragma unroll 1
  for (;;) {
    if (own)
      sP[sl] = v;
    barrier();
    const double av = row.apply_fused(pval);
    const double vav = allsum(av * v, 1);
    if (it == -2) {
      omega = allsum(f * xv, 0) / vav;
      break;
    }
    if (it == -1) {
      rv = f - av;
      rs = allsum(rv * rv, 0);
      v = rv;
      it = 0;
      continue;
    }
    bool done = false;
    if (it == 0) {
      const double r0 = sqrt(rs);
      const double stop = fmax(a.thresh, a.rtol * r0);
      stop2 = stop * stop;
      const double res = a.class_first_check ? sqrt(r0) : r0;
      done = vav == 0.0 || !(res > stop) || a.max_iters <= 0;
      capped = vav != 0.0 && res > stop && a.max_iters <= 0;
    }
    if (!done) {
      const double alpha = vav == 0.0 ? 0.0 : rs / vav;
      ++it;
      xv += alpha * v;
      rv = rv - alpha * av;
      rs_old = rs;
      rs = allsum(rv * rv, 0);
      capped = rs > stop2 && it >= a.max_iters;
      done = !(rs > stop2) || capped;
      v = rv + (rs_old == 0.0 ? 0.0 : rs / rs_old) * v;
    }
    if (done) {
      a.status[0] = it; // (the same value from every thread)
      a.status[1] = capped ? 1 : 0;
      v = xv;
      it = -2;
    }
  }
  if (own) {
    sm.x1[gi] = (T)xv;
    if (a.warm_start)
      a.x1[gi] = xv;
  }
  return omega;
}

template <typename T>
__device__ __forceinline__ void bottom_cluster_body(const BottomArgs<T> &a) {
  namespace cgs = cooperative_groups;
  cgs::cluster_group cluster = cgs::this_cluster();
  extern __shared__ __align__(16) unsigned char bc_raw[];
  BcSmem<T> &sm = *reinterpret_cast<BcSmem<T> *>(bc_raw);
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int top = a.top;
  bool lost = false;

  // ---- this thread's point of the top level ----
  const Dims td = a.lv[top].d;
  const int nx = td.nx, ny = td.ny, nz = td.nz;
  const int klo = cg_plane_lo(rank, nz);
  const int khi = cg_plane_lo(rank + 1, nz) - 1;
  const int colour = warp >> 1, g = colour >> 2;
  const int q = (warp & 1) * 32 + lane;
  const int k = klo + ((g - klo) & 1); // the CTA's plane of parity g
  const bool active = k <= khi;
  const int i = 2 + (colour & 1) + 2 * (q & 7);
  const int j = 2 + ((colour >> 1) & 1) + 2 * (q >> 3);
  const bool own = active && i <= nx - 1 && j <= ny - 1;
  const int gi = own ? td.at(i, j, k) : 0;
  // in the group's planes 0 .. 2 (without a point: other entries of sm, read
  // and discarded)
  const auto pt = split_point<kBcRow, kBcPlane, kBcOdd>(i, j, 1);
  T *xs = sm.x[g];
  const BottomLevel<T> &v = a.lv[top];
  const Dims cd = a.lv[top - 1].d; // the level below the top
  StencilRow<T, 27> row;
  // (threads without a point: couplings of zero, and 1 / 1 in the divide, so
  // that they stay on its short path)
  T f = T(1), recip = T(1);
  auto load_row = [&]() {
    row.clear();
    if (own) {
      row.load(v.A, nullptr, gi, td.sy(), td.sz());
      f = v.f[gi];
      recip = recip_of(row.centre);
    }
  };
  load_row();

  // what rank 0 will wait for on the levels below, into L2 (at the large
  // grids it has left L2 since the last cycle)
  {
    auto prefetch = [&](const void *base, int bytes, int part, int parts) {
      for (int o = 128 * part; o < bytes; o += 128 * parts)
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"((const char *)base +
                                                        o));
    };
    const int part = rank * (kBcThreads / 64) + tid / 64; // of 64 parts
    for (int L = 1; L < top; ++L) {
      const BottomLevel<T> &b = a.lv[L];
      const int n = (int)b.d.count();
      const int t = tid & 63;
      if (t < 27)
        prefetch(b.P.p[t], n * (int)sizeof(T), part, 64);
      else if (t < 41 && L > 1)
        prefetch(b.A.a[t - 27], n * (int)sizeof(T), part, 64);
      else if (t < 41 && !a.inv)
        prefetch(a.A1.a[t - 27], n * 8, part, 64);
      else if (t == 41 && L == 1 && a.inv)
        prefetch(a.inv, 8 * kInvMax * kInvMax, part, 64);
    }
  }

  // ---- shared memory, mbarriers ----
  for (int t = tid; t < (int)(sizeof(BcSmem<T>) / 16); t += kBcThreads)
    reinterpret_cast<int4 *>(bc_raw)[t] = int4{0, 0, 0, 0};
  static_assert(sizeof(BcSmem<T>) % 16 == 0, "zeroed by 16 bytes");
  __syncthreads();
  const int mij = (nx - 2) * (ny - 2);
  const unsigned x_bytes =
      (unsigned)sizeof(T) * mij * ((k > 2) + (k < nz - 1)) + a.extra_tx;
  constexpr unsigned kXcBytes =
      (unsigned)(offsetof(BcSmem<T>, omega) - offsetof(BcSmem<T>, xc) + 8 +
                 15) &
      ~15u;
  const bool first = (warp & 7) == 0 && lane == 0; // of its group
  if (first && active) {
    mbar_init(&sm.bar_x[g], 1);
    mbar_expect_tx(&sm.bar_x[g], x_bytes);
  }
  if (tid == 0) {
    mbar_init(&sm.bar_c, 1);
    mbar_expect_tx(&sm.bar_c, kXcBytes + a.extra_tx);
    if (rank == 0) {
      mbar_init(&sm.bar_r, 1);
      mbar_expect_tx(&sm.bar_r,
                     (unsigned)sizeof(T) * mij * (nz - 2) + a.extra_tx);
      mbar_init(&sm.bar_d, 1);
      mbar_expect_tx(&sm.bar_d, 16u * (nz - 2) + a.extra_tx);
    }
  }
  fence_mbar_init();
  cluster.sync(); // zeroed and armed before anyone sends

  // ---- level 1 (rank 0): up to 32 points in the last warp, else rows of
  // eight lanes over the CTA's last warps. r: the defect of level 2 ----
  const Dims d1 = a.lv[1].d;
  const int m1x = d1.nx - 2, m1y = d1.ny - 2, m1z = d1.nz - 2;
  const bool packed = m1x * m1y * m1z <= 32;
  const bool direct = a.inv && *a.inv_ok;
  const int threads1 = packed ? 32 : (8 * m1y * m1z + 31) & ~31;
  const int t1 = tid - (kBcThreads - threads1); // >= 0: a thread of level 1
  auto level1 = [&]() {
    const int l1 = packed ? m1x : 8;
    const int r1 = t1 / l1, p1 = r1 / m1y;
    const bool own1 = t1 - r1 * l1 < m1x && p1 < m1z;
    const int i1 = 2 + t1 - r1 * l1, j1 = 2 + r1 - p1 * m1y, k1 = 2 + p1;
    const int nat = own1 ? d1.at(i1, j1, k1) : 0;
    T f1 = T(0);
    if (own1)
      f1 = top == 2 ? bc_restrict_at<kBcRow, kBcPlane, kBcOdd>(
                          sm.r, a.lv[1].P, nat, i1, j1, k1)
                    : bc_restrict_at<kBlRow, kBlPlane, kBlOdd>(
                          sm.lr, a.lv[1].P, nat, i1, j1, k1);
    double omega = 1.0;
    if (direct) {
      bc_level1_direct(a, sm, threads1, own1,
                       i1 - 2 + m1x * (j1 - 2 + m1y * (k1 - 2)), nat, f1);
    } else {
      StencilRow<double, 27> row1;
      row1.clear();
      if (own1)
        row1.load(a.A1, nullptr, nat, d1.sy(), d1.sz());
      omega = bc_level1(a, sm, threads1, own1, i1, j1, k1, row1, (double)f1);
    }
    sm.omega = omega;
    if (top == 2 && own1)
      sm.xc[nat] = sm.x1[nat];
  };

  {
    // the copies of this point that the planes below and above keep
    unsigned dn = 0, dn_bar = 0, up = 0, up_bar = 0;
    if (own && k > 2) {
      const int r = cg_plane_owner(k - 1, nz);
      dn = cluster_addr(&sm.x[1 - g][pt.c + kBcPlane], r);
      dn_bar = cluster_addr(&sm.bar_x[1 - g], r);
    }
    if (own && k < nz - 1) {
      const int r = cg_plane_owner(k + 1, nz);
      up = cluster_addr(&sm.x[1 - g][pt.c - kBcPlane], r);
      up_bar = cluster_addr(&sm.bar_x[1 - g], r);
    }
    auto push = [&](T val) {
      send(dn, val, dn_bar);
      send(up, val, up_bar);
    };
    unsigned x_parity = 0;
    auto group_barrier = [&]() { named_barrier(1 + g, kBcThreads / 2); };
    auto xval = [&](int dx, int dy, int dz) {
      return pt.read(xs, dx, dy, dz);
    };
    // phase 0: smooth from zero, defect to rank 0; 1: correction, smooth,
    // damping (one loop: the code of the sweeps once)
    BcInterp<T> w;
#pragma unroll 1
    for (int phase = 0; phase < 2; ++phase) {
      // (every CTA takes delivery, also one without a plane: nothing is in
      // flight to it when it leaves)
      if (phase == 1 && rank != 0)
        lost |= !mbar_wait_cluster(&sm.bar_c, 0, lost);
      if (active) {
        if (phase == 1) {
          const int cy = cd.sy(), cz = cd.sz();
          T val = T(0);
          if (own) {
            const T e = w.eval([&](int bx, int by, int bz) {
              return sm.xc[w.cc + bx + by * cy + bz * cz];
            });
            val = xs[pt.c] + (T)sm.omega * e;
            xs[pt.c] = val;
          }
          if (g == 1)
            push(val);
          group_barrier();
        }
        // two eight-colour sweeps (the even planes' four colours, then the
        // odd ones') and, as a third turn of the loop, A x
        T ax = T(0);
#pragma unroll 1
        for (int s = 0; s < 3; ++s) {
          if (s == 2 && a.idle_delay && !__any_sync(0xffffffffu, own))
            for (int q16 = 0; q16 < a.idle_delay; ++q16)
              __nanosleep(16384);
          if (s == 2 ? g == 0 : g == 1 || s > 0 || phase == 1) {
            lost |= !mbar_wait_cluster(&sm.bar_x[g], x_parity, lost);
            x_parity ^= 1u;
            mbar_expect_tx_if(first && !lost, &sm.bar_x[g], x_bytes);
          }
          if (s == 2) {
            if (g == 0)
              group_barrier(); // every warp has seen that phase
            break;
          }
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            if ((colour & 3) == c) { // whole warps (no point: zeros)
              const T val = bc_relax(row, recip, f, xval);
              if (own)
                xs[pt.c] = val;
              push(val);
            }
            group_barrier();
          }
        }
        ax = row.apply(xval);
        if (phase == 0) {
          const unsigned bar = cluster_addr(&sm.bar_r, 0);
          send(bar - smem_addr(&sm.bar_r) +
                   smem_addr(&sm.r[pt.c + (k - 2) * kBcPlane]),
               f - ax, own ? bar : 0u);
        } else {
          const T xv = own ? xs[pt.c] : T(0);
          if (own)
            v.x[gi] = xv;
          const double s0 = warp_allsum((double)f * (double)xv);
          const double s1 = warp_allsum(own ? (double)xv * (double)ax : 0.0);
          if (lane == 0) {
            sm.red[0][warp] = s0;
            sm.red[1][warp] = s1;
          }
          group_barrier();
          double t0 = 0.0, t1 = 0.0;
#pragma unroll
          for (int w8 = 0; w8 < 8; ++w8) {
            t0 += sm.red[0][8 * g + w8];
            t1 += sm.red[1][8 * g + w8];
          }
          const unsigned bar = first ? cluster_addr(&sm.bar_d, 0) : 0u;
          send(cluster_addr(&sm.dsum[k - 2][0], 0), t0, bar);
          send(cluster_addr(&sm.dsum[k - 2][1], 0), t1, bar);
        }
      }
      if (phase == 1)
        break;

      // ---- the levels below on rank 0, one point per thread in the order
      // of the colours ----
      if (rank == 0 && top == 2) {
        lost |= !mbar_wait_cluster(&sm.bar_r, 0, lost);
        if (t1 >= 0)
          level1();
      }
      if (rank == 0 && top > 2) {
        const int li = 2 + (colour & 1) + 2 * (q & 3);
        const int lj = 2 + ((colour >> 1) & 1) + 2 * ((q >> 2) & 3);
        const int lk = 2 + (colour >> 2) + 2 * (q >> 4);
        const auto lp = split_point<kBlRow, kBlPlane, kBlOdd>(li, lj, lk - 1);
        StencilRow<T, 27> lrow;
        lrow.clear();
        T lrecip = T(1); // (1 / 1 again without a point)
        double omega = 0.0;

        // down the levels and up again (one loop: their code once)
        const int down = top - 2;
#pragma unroll 1
        for (int st = 0; st < 2 * down; ++st) {
          const bool ascend = st >= down;
          const int L = ascend ? 2 + st - down : top - 1 - st;
          const BottomLevel<T> &b = a.lv[L];
          const bool mine =
              li <= b.d.nx - 1 && lj <= b.d.ny - 1 && lk <= b.d.nz - 1;
          const int pc = b.d.at(li, lj, lk);
          T *x = sm.lx[L - 2], *lf = sm.lf[L - 2];
          auto lval = [&](int dx, int dy, int dz) {
            return lp.read(x, dx, dy, dz);
          };
          // (the first level up is the last one down: its row is here)
          auto load_local = [&]() {
            lrow.clear();
            lrecip = T(1);
            if (mine) {
              lrow.load(b.A, nullptr, pc, b.d.sy(), b.d.sz());
              lrecip = recip_of(lrow.centre);
            }
          };
          // (the row and the restriction's weights are loaded together where
          // the registers hold both)
          constexpr bool kBoth = sizeof(T) == sizeof(float);
          if (st != down && (kBoth || ascend))
            load_local();
          T fl = T(1);
          if (!ascend) {
            T w27[27];
#pragma unroll
            for (int t = 0; t < 27; ++t)
              w27[t] = mine ? b.P.p[t][pc] : T(0);
            if (st == 0) {
              lost |= !mbar_wait_cluster(&sm.bar_r, 0, lost);
              fl = bc_restrict_with<kBcRow, kBcPlane, kBcOdd>(sm.r, w27, li,
                                                              lj, lk);
            } else {
              fl = bc_restrict_with<kBlRow, kBlPlane, kBlOdd>(sm.lr, w27, li,
                                                              lj, lk);
              __syncthreads(); // lr is read before it is written again
            }
            if (mine)
              lf[lp.c] = fl;
            else
              fl = T(1);
            if (!kBoth)
              load_local();
          } else {
            const Dims c = a.lv[L - 1].d;
            BcInterp<T> wi;
            wi.load(a.lv[L - 1].P, c, li, lj, lk, mine);
            if (L == 2) {
              if (t1 >= 0) {
                level1();
                load_local(); // (not held over level 1)
              }
              __syncthreads();
              omega = sm.omega;
            }
            if (mine) {
              const int ci = (li + 1) >> 1, cj = (lj + 1) >> 1,
                        ck = (lk + 1) >> 1;
              const T e = wi.eval([&](int bx, int by, int bz) {
                return L == 2 ? sm.x1[c.at(ci + bx, cj + by, ck + bz)]
                              : sm.lx[kBlMaxLevels - 2]
                                     [(ck + bz - 1) * kBlPlane +
                                      (cj + by - 1) * kBlRow +
                                      split_entry<kBlOdd>(ci + bx)];
              });
              fl = lf[lp.c];
              x[lp.c] = x[lp.c] + (T)omega * e;
            }
            __syncthreads();
          }
#pragma unroll 1
          for (int c = 0; c < 16; ++c) {
            if (colour == (c & 7)) { // whole warps
              const T val = bc_relax(lrow, lrecip, fl, lval);
              if (mine)
                x[lp.c] = val;
            }
            __syncthreads();
          }
          const T ax = lrow.apply(lval);
          if (!ascend) {
            if (mine)
              sm.lr[lp.c] = fl - ax;
            __syncthreads();
          } else {
            // damping of this level
            const T xv = mine ? x[lp.c] : T(0);
            const double s0 = warp_allsum((double)fl * (double)xv);
            const double s1 =
                warp_allsum(mine ? (double)xv * (double)ax : 0.0);
            if (lane == 0) {
              sm.red[0][warp] = s0;
              sm.red[1][warp] = s1;
            }
            __syncthreads();
            double t0[4] = {}, t1[4] = {};
#pragma unroll
            for (int u = 0; u < kBcThreads / 32; ++u) {
              t0[u & 3] += sm.red[0][u];
              t1[u & 3] += sm.red[1][u];
            }
            omega = ((t0[0] + t0[1]) + (t0[2] + t0[3])) /
                    ((t1[0] + t1[1]) + (t1[2] + t1[3]));
            if (L == top - 1 && mine)
              sm.xc[pc] = xv;
            sm.omega = omega; // (the same value from every thread)
            fence_proxy_async_smem();
            __syncthreads(); // red is read before it is written again
          }
        }
      }
      // level top-1's iterate and damping to the other CTAs
      if (rank == 0) {
        if (top == 2) {
          fence_proxy_async_smem();
          __syncthreads();
        }
        if (warp == 0) {
          const int r = lane & (kCgCtas - 1);
          copy_to_cta_if(lane < kCgCtas && r != 0, cluster_addr(sm.xc, r),
                         sm.xc, kXcBytes, cluster_addr(&sm.bar_c, r));
        }
      }
      // again, so that it is not held over the levels below
      load_row();
      w.load(a.lv[top - 1].P, cd, i, j, k, own);
    }
  }
  if (rank == 0 && warp == 15) {
    // the damping of the top level, planes in order
    lost |= !mbar_wait_cluster(&sm.bar_d, 0, lost);
    double t0 = 0.0, t1 = 0.0;
    for (int p = 0; p < nz - 2; ++p) {
      t0 += sm.dsum[p][0];
      t1 += sm.dsum[p][1];
    }
    *v.omega = t0 / t1;
  }
  if (lost)
    *a.kernel_err = 1;
  leave_cluster(lost);
}

__global__ void __cluster_dims__(kCgCtas, 1, 1)
    __launch_bounds__(kBcThreads, 1)
        bottom_cluster_f_kernel(BottomArgs<float> a) {
  bottom_cluster_body<float>(a);
}
__global__ void __cluster_dims__(kCgCtas, 1, 1)
    __launch_bounds__(kBcThreads, 1)
        bottom_cluster_d_kernel(BottomArgs<double> a) {
  bottom_cluster_body<double>(a);
}

} // namespace pmg
