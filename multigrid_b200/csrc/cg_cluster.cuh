// Conjugate gradients on a small level held on chip: the coarsest-level CG of
// the class and the APBS layer's Vcghs.
//
// The iteration is a chain of latencies, not of work: a 17^3 level has 3375
// unknowns, 0.2 us of arithmetic for one SM's worth of FP64 units, but each
// iteration needs two global sums. So everything that a sum waits for is kept
// short:
//   * each thread owns one point and holds its couplings, x, r, p and A p in
//     registers for the whole solve; p is also in shared memory, where A p
//     reads 26 neighbours at immediate offsets (fixed pitch);
//   * levels up to 9^3 run in one CTA; larger ones are split by planes over a
//     cluster of kCgCtas CTAs;
//   * no CTA reads another's memory (a remote load is ~220 cycles) or waits
//     at a cluster barrier (~550 with remote stores before it): the CTAs send
//     their sums to each other as messages (mbar.cuh), and the owner of a
//     plane at a CTA's edge sends the new r to the neighbour's copy with the
//     r.r sum; the neighbour forms the same p = r + beta p for its copy.
// Measured, against couplings in shared memory, neighbouring planes read
// remotely and three cluster barriers per iteration: a coarsest solve of 11^3
// (a 161^3 FP64 solve) 284 -> 157 us, 17 x 15 x 16 576 -> 279 us, 5^3 48 -> 18
// us; with the remote reads replaced but cluster barriers kept, 206 and 368 us
// for the first two. Vcghs at 9^3, which was three launches and a read-back
// per iteration (38 us), takes 1.3 us per iteration.
//
// Replaces CG_solver (CG_Solver.h:45-242, via solve_by_cg<1>) and Vcghs
// (pmgc/cgd.cc:60-125); the arithmetic per point is theirs.
#pragma once

#include <cooperative_groups.h>

#include "cluster_planes.cuh"
#include "mbar.cuh"
#include "reduce_kernels.cuh"
#include "row_stencil.cuh"

namespace pmg {

// One CTA up to this many threads and interior planes (9^3: 392 and 7).
constexpr int kCgCtaThreads = 448;
constexpr int kCgCtaPlanes = 9;

struct CgArgs {
  Dims d;
  Op14<double> A;
  const double *cc; // Vcghs: added to oC; the class: null
  const double *rhs;
  double *x;
  // Vcghs: its work arrays, written at the end
  double *r, *p, *ap;
  // the class: sqrt(r.r) <= max(thresh, rel_tol sqrt(r0.r0)), the first test
  // on sqrt(sqrt(r.r)) with class_first_check; Vcghs: sqrt(r.r) <= errtol
  // sqrt(r0.r0)
  double thresh, rel_tol, errtol;
  int class_first_check;
  // the class on level 1 of a V-cycle: a float right-hand side and result
  // (mixed) and a start from zero; omega receives the damping of the result
  const float *rhs32;
  float *x32;
  int zero_start;
  double *omega;
  int max_iters;
  int *status; // [0] iterations, the class: [1] stopped by the cap
  // set to err_value, after status, when a message did not arrive (a bounded
  // wait ran out)
  int *err;
  int err_value;
  unsigned extra_tx; // a test's bytes that no message brings (0)
};

inline bool cg_cluster_fits(const Dims &d) {
  return d.nx <= kCgMaxN && d.ny <= kCgMaxN && d.nz <= kCgMaxN &&
         d.px == d.nx;
}
// A row of the level is 8 or 16 neighbouring threads (the last ones idle),
// and rows of p lie 24 doubles apart: the sixteen lanes of a half warp then
// read sixteen different 8-byte banks at every neighbour offset, one row of
// 16 or two of 8. Points packed without idle lanes at a pitch of 17 met
// 3-way conflicts in most loads.
__host__ __device__ inline int cg_row_lanes(int nx) {
  return nx - 2 <= 8 ? 8 : 16;
}
constexpr int kCgRow = 24;               // pitch of a row of p
constexpr int kCgPlane = kCgRow * kCgMaxN; // and of a plane
inline int cg_threads(const Dims &d, int planes) {
  return (cg_row_lanes(d.nx) * (d.ny - 2) * planes + 31) & ~31;
}
inline bool cg_one_cta(const Dims &d) {
  return d.nz - 2 <= kCgCtaPlanes && cg_threads(d, d.nz - 2) <= kCgCtaThreads;
}

template <int KIND, bool APBS, int C>
__device__ __forceinline__ void cg_on_chip(const CgArgs &a) {
  namespace cgs = cooperative_groups;
  constexpr int kPlanes = C == 1 ? kCgCtaPlanes : kCgMaxPlanes;
  // p: planes klo - 1 .. khi + 1 (the outer two are copies, or shell zeros)
  __shared__ double sP[(kPlanes + 2) * kCgPlane];
  // the neighbours' r on those two planes
  __shared__ double sR[C == 1 ? 1 : 2 * kCgPlane];
  // warp sums of this CTA; the CTAs' sums, by rank
  __shared__ double sWarp[2][kCgThreads / 32];
  __shared__ double sCta[2][C];
  __shared__ uint64_t bar[2]; // the messages of the two sums
  const Dims &d = a.d;
  const int nx = d.nx, nz = d.nz, mi = d.nx - 2, mij = mi * (d.ny - 2);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = blockDim.x, nw = nt >> 5;
  int rank = 0;
  if constexpr (C > 1)
    rank = (int)cgs::this_cluster().block_rank();
  const int klo = C == 1 ? 2 : cg_plane_lo(rank, nz);
  const int khi = C == 1 ? nz - 1 : cg_plane_lo(rank + 1, nz) - 1;
  const int np = khi - klo + 1; // may be 0

  for (int q = tid; q < (kPlanes + 2) * kCgPlane; q += nt)
    sP[q] = 0.0;
  for (int q = tid; q < 2 * (kCgThreads / 32); q += nt)
    (&sWarp[0][0])[q] = 0.0;
  if constexpr (C > 1)
    for (int q = tid; q < 2 * kCgPlane; q += nt)
      sR[q] = 0.0;

  // this thread's point
  const int lanes = cg_row_lanes(nx), mj = d.ny - 2;
  const int trow = tid / lanes, tplane = trow / mj;
  const bool own = tid - trow * lanes < mi && tplane < np;
  const int i = 2 + tid - trow * lanes, j = 2 + trow - tplane * mj;
  const int k = klo + tplane;
  const int gi = own ? d.at(i, j, k) : 0;
  // (idle lanes read their own columns of the padded rows, so that they meet
  // no one else's bank, and discard them)
  const int sl = (min(tplane, kPlanes - 1) + 1) * kCgPlane +
                 (j - 1) * kCgRow + (i - 1);
  StencilRow<double, KIND> row;
  row.clear();
  double fv = 0.0, xv = 0.0, rv = 0.0, pv = 0.0, apv = 0.0;
  if (own) {
    row.load(a.A, a.cc, gi, nx, nx * d.ny);
    const double *x = a.x;
    const int sy = nx, sz = nx * d.ny;
    auto xval = [&](int dx, int dy, int dz) {
      return x[gi + dx + dy * sy + dz * sz];
    };
    fv = !APBS && a.rhs32 ? (double)a.rhs32[gi] : a.rhs[gi];
    if (!APBS && a.zero_start) {
      rv = fv;
    } else {
      xv = x[gi];
      rv = APBS ? row.resid(fv, xval) : fv - row.apply(xval);
    }
  }
  auto pval = [&](int dx, int dy, int dz) {
    return sP[sl + dx + dy * kCgRow + dz * kCgPlane];
  };

  // Messages (C > 1). The r.r sum also waits for the neighbours' r on the
  // copied planes, so its bytes include them; the senders store each r with
  // its bytes on the neighbour's mbarrier.
  unsigned msg_bytes[2] = {8u * C + a.extra_tx, 8u * C + a.extra_tx};
  unsigned parity[2] = {0u, 0u};
  unsigned dn = 0, dn_bar = 0, up = 0, up_bar = 0; // cluster addresses
  bool lost = false;
  if constexpr (C > 1) {
    const int o = (j - 1) * kCgRow + (i - 1);
    if (np > 0)
      msg_bytes[0] += 8u * mij * ((klo > 2) + (khi < nz - 1));
    if (own && k == klo && klo > 2) {
      const int r = cg_plane_owner(klo - 1, nz);
      dn = cluster_addr(sR + kCgPlane + o, r);
      dn_bar = cluster_addr(&bar[0], r);
    }
    if (own && k == khi && khi < nz - 1) {
      const int r = cg_plane_owner(khi + 1, nz);
      up = cluster_addr(sR + o, r);
      up_bar = cluster_addr(&bar[0], r);
    }
    if (tid == 0) {
      for (int q = 0; q < 2; ++q) {
        mbar_init(&bar[q], 1);
        mbar_expect_tx(&bar[q], msg_bytes[q]);
      }
      fence_mbar_init();
    }
    cgs::this_cluster().sync(); // zeroed and armed before anyone sends
  } else {
    __syncthreads();
  }
  auto push = [&]() {
    send(dn, rv, dn_bar);
    send(up, rv, up_bar);
  };
  // the points of the two copied planes this thread keeps (at most two)
  int h0 = -1, h1 = -1; // entry in sR, or -1
  if (C > 1 && np > 0) {
    auto entry = [&](int q) {
      const int side = q / mij, r2 = q - side * mij;
      const int jj = r2 / mi;
      const int kk = side == 0 ? klo - 1 : khi + 1;
      return q < 2 * mij && kk >= 2 && kk <= nz - 1
                 ? side * kCgPlane + (jj + 1) * kCgRow + r2 - jj * mi + 1
                 : -1;
    };
    h0 = entry(tid);
    h1 = entry(tid + nt);
  }
  auto copy_at = [&](int h) { // its entry in sP
    return h < kCgPlane ? h : h + np * kCgPlane;
  };

  // Sum over every thread of the cluster, the same bits in each: warp sums,
  // then the CTA's, then the CTAs' in one fixed tree. A set's arrays and
  // mbarrier are used again only after the other set's sum, which every
  // thread joins after it has read them.
  auto allsum = [&](double v, int set) -> double {
    v = warp_allsum(v);
    if (C == 1 && nw == 1)
      return v;
    if (lane == 0)
      sWarp[set][warp] = v;
    __syncthreads();
    double s[4] = {0.0, 0.0, 0.0, 0.0}; // (the entries past nw are zero)
    if (C == 1 || warp == 0) {
#pragma unroll
      for (int w = 0; w < kCgThreads / 32; ++w)
        s[w & 3] += sWarp[set][w];
    }
    v = (s[0] + s[1]) + (s[2] + s[3]);
    if constexpr (C > 1) {
      send(cluster_addr(&sCta[set][rank], lane & (C - 1)), v,
           tid < C ? cluster_addr(&bar[set], lane & (C - 1)) : 0u);
      lost |= !mbar_wait_cluster(&bar[set], parity[set], lost);
      parity[set] ^= 1u;
      mbar_expect_tx_if(tid == 0 && !lost, &bar[set], msg_bytes[set]);
      const double *t = sCta[set];
      v = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
      static_assert(C == 8, "the tree of the CTAs' sums");
    }
    return v;
  };

  push();
  double rs = allsum(rv * rv, 0), rs_old = 0.0;
  const double r0 = sqrt(rs);
  // the stop tests as bounds on r.r
  const double stop = APBS ? a.errtol * r0 : fmax(a.thresh, a.rel_tol * r0);
  const double stop2 = stop < 0.0 ? -1.0 : stop * stop;
  int it = 0;
  bool capped = false;
  for (;;) {
    // the new direction, on the CTA's points and the copied planes
    const double beta =
        it == 0 || (!APBS && rs_old == 0.0) ? 0.0 : rs / rs_old;
    const double inv = APBS && it > 0 ? 1.0 / beta : 0.0;
    auto direction = [&](double r, double p) {
      if (it == 0)
        return r;
      return APBS ? (p + inv * r) * beta : r + beta * p;
    };
    const double pnew = direction(rv, pv);
    if (own)
      sP[sl] = pnew;
    if constexpr (C > 1) {
      if (h0 >= 0)
        sP[copy_at(h0)] = direction(sR[h0], sP[copy_at(h0)]);
      if (h1 >= 0)
        sP[copy_at(h1)] = direction(sR[h1], sP[copy_at(h1)]);
    }
    // (threads that gave a message up may hold other sums than the rest of
    // the CTA: every branch on a sum comes after a vote on that)
    if constexpr (C == 1) {
      __syncthreads();
    } else {
      lost = __syncthreads_or(lost);
      if (lost)
        break;
    }
    if constexpr (APBS) {
      if ((it == 0 && (r0 == 0.0 || r0 / r0 <= a.errtol)) ||
          (it > 0 && rs <= stop2) || it >= a.max_iters)
        break;
    } else if (it > 0) {
      if (!(rs > stop2))
        break;
      if (it >= a.max_iters) {
        capped = true;
        break;
      }
    }
    pv = pnew;
    // (every lane: threads without a point hold a row of zeros)
    apv = row.apply(pval);
    const double pap = allsum(apv * pv, 1);
    if (!APBS && it == 0) {
      if constexpr (C > 1) {
        lost = __syncthreads_or(lost);
        if (lost)
          break;
      }
      if (pap == 0.0)
        break;
      const double res = a.class_first_check ? sqrt(r0) : r0;
      if (!(res > stop) || a.max_iters <= 0) {
        capped = res > stop;
        break;
      }
    }
    const double alpha = !APBS && pap == 0.0 ? 0.0 : rs / pap;
    ++it;
    xv += alpha * pv;
    rv = rv - alpha * apv;
    push();
    rs_old = rs;
    rs = allsum(rv * rv, 0);
  }
  if constexpr (!APBS)
    if (a.omega && !lost) {
      // the damping (f . x) / (x . A x), x exchanged like r. (The sums'
      // sets alternate: the last one was r.r unless no iteration ran.)
      if (it > 0)
        allsum(0.0, 1);
      rv = xv;
      push();
      const double up_sum = allsum(fv * xv, 0);
      if (own)
        sP[sl] = xv;
      if constexpr (C > 1) {
        if (h0 >= 0)
          sP[copy_at(h0)] = sR[h0];
        if (h1 >= 0)
          sP[copy_at(h1)] = sR[h1];
      }
      __syncthreads();
      const double lo_sum = allsum(own ? xv * row.apply(pval) : 0.0, 1);
      if (rank == 0 && tid == 0)
        *a.omega = up_sum / lo_sum;
    }
  if (own) {
    if (!APBS && a.x32)
      a.x32[gi] = (float)xv;
    else if (!APBS || it > 0)
      a.x[gi] = xv;
    if constexpr (APBS) {
      a.r[gi] = rv;
      if (it > 0) {
        a.p[gi] = pv;
        a.ap[gi] = apv;
      }
    }
  }
  if (rank == 0 && tid == 0) {
    a.status[0] = it;
    if constexpr (!APBS)
      a.status[1] = capped ? 1 : 0;
  }
  if constexpr (C > 1) {
    leave_cluster(lost);
    if (lost && a.err)
      *a.err = a.err_value;
  }
}

template <int KIND, bool APBS>
__global__ void __cluster_dims__(kCgCtas, 1, 1) __launch_bounds__(kCgThreads)
    cg_cluster_kernel(CgArgs a) {
  cg_on_chip<KIND, APBS, kCgCtas>(a);
}
template <int KIND, bool APBS>
__global__ void __launch_bounds__(kCgCtaThreads)
    cg_cta_kernel(CgArgs a) {
  cg_on_chip<KIND, APBS, 1>(a);
}

// One solve of a level that cg_cluster_fits, queued on s.
template <int KIND, bool APBS>
int launch_cg_on_chip(CgArgs a, cudaStream_t s) {
  a.extra_tx = test_message_extra_tx();
  const int mk = a.d.nz - 2;
  if (cg_one_cta(a.d))
    cg_cta_kernel<KIND, APBS><<<1, cg_threads(a.d, mk), 0, s>>>(a);
  else
    cg_cluster_kernel<KIND, APBS>
        <<<kCgCtas, cg_threads(a.d, (mk + kCgCtas - 1) / kCgCtas), 0, s>>>(a);
  PMG_LAUNCH_CHECK();
  return PMG_OK;
}

} // namespace pmg
