// Fine-level set-up from atoms on the GPU: the host set-up of pmg_setup.cc
// (the reference class's initialize_epsilons, set_up_rhs and
// initialize_boundary, PBE_pmgc_class.h:141-349) restated as kernels, so a
// request only moves its atoms to the device instead of six n^3 arrays.
//
//   marking   every sphere (atom, inflated atom, probe) marks the grid points
//             the host's sphere walk marks (same index bounds, same chord
//             square roots); marks are idempotent, so any order gives the
//             host's masks bit for bit.
//   probes    the accessibility test of each probe centre is an OR over all
//             other inflated spheres (the host's cell list only skips atoms
//             that cannot contain the point); probe centres use the host's
//             direction table, so they are the same doubles.
//   oC        the host's per-point sum, same order.
//   charges   the trilinear contributions are sorted by grid point with a
//             stable sort over records generated in atom order, and each
//             point sums its run in that order: the host's serial sum, bit
//             for bit.
//   boundary  the multiple Debye-Hueckel sum over atoms on the six faces, in
//             another order than the host's and with its own exp and square
//             root: equal to a few ulp of the sum's largest terms.
// All work is stream-ordered on the caller's stream; scratch comes from the
// library's stream-ordered pool.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <limits.h>
#include <cmath>
#include <vector>

#include "pmg_common.cuh"
#include "pmg_physics.h"

namespace pmg {
namespace {

constexpr int kSetupThreads = 256;

struct SphereSet {
  const double *centers; // rows of `stride` doubles, x y z first
  int stride;
  int count;            // (an upper bound where count_dev is given)
  const double *radius; // radius of row q at radius[q * stride] or null
  double radius_add;    // added to the row radius (or the radius if null)
  const int *count_dev; // the count, on the device (or null)
  unsigned char *mask;  // set to 1 at the marked points
};
// Up to three sets marked by one launch.
struct SphereSets {
  SphereSet set[3];
  int axis; // centres shifted by -h/2 along this axis (-1: no)
};

// The points of sphere q of a set: part `part` of `parts`, by one warp.
__device__ __forceinline__ void mark_sphere(int n, double h,
                                            const SphereSet &set, int axis,
                                            int q, int part, int parts,
                                            int lane) {
  const double *row = set.centers + (size_t)q * set.stride;
  const double hx = 0.5 * h;
  const double c[3] = {axis == 0 ? row[0] - hx : row[0],
                       axis == 1 ? row[1] - hx : row[1],
                       axis == 2 ? row[2] - hx : row[2]};
  const double r = set.radius ? set.radius[(size_t)q * set.stride] +
                                    set.radius_add
                              : set.radius_add;
  const int lo0 = (int)ceil((c[0] - r) / h);
  const int hi0 = (int)((c[0] + r) / h);
  const int blo1 = (int)ceil((c[1] - r) / h) - 1;
  const int bhi1 = (int)((c[1] + r) / h) + 1;
  const int w0 = hi0 - lo0 + 1, w1 = bhi1 - blo1 + 1;
  if (w0 <= 0 || w1 <= 0)
    return;
  for (int t = lane + 32 * part; t < w0 * w1; t += 32 * parts) {
    const int i0 = lo0 + t / w1, i1 = blo1 + t % w1;
    if (i0 < 0 || i1 < 0 || i0 >= n || i1 >= n)
      continue;
    double s1 = r * r - ((c[0] - h * i0) * (c[0] - h * i0));
    if (s1 < 0)
      s1 = 0;
    const double ww1 = sqrt(s1);
    const int lo1 = (int)ceil((c[1] - ww1) / h);
    const int hi1 = (int)((c[1] + ww1) / h);
    if (i1 < lo1 || i1 > hi1)
      continue;
    double s2 = r * r - ((c[0] - h * i0) * (c[0] - h * i0) +
                         (c[1] - h * i1) * (c[1] - h * i1));
    if (s2 < 0)
      s2 = 0;
    const double ww2 = sqrt(s2);
    const int lo2 = (int)ceil((c[2] - ww2) / h);
    const int hi2 = (int)((c[2] + ww2) / h);
    unsigned char *m = set.mask + ((size_t)i0 * n + i1) * n;
    for (int i2 = lo2 < 0 ? 0 : lo2; i2 <= hi2 && i2 < n; ++i2)
      m[i2] = 1;
  }
}

// Marks the grid points of every sphere of the sets (for_dots_in_sphere of
// the host set-up): axis-0 range ceil((c0 - r)/h) .. trunc((c0 + r)/h), chord
// half-widths from sqrt of the clamped squared remainders on axes 1 and 2.
// One warp per sphere, lanes over the (i0, i1) bounding rectangle (~60 points
// of a probe sphere); the warps of a grid that fills the GPU once stride over
// the spheres. A block per sphere, with the probe positions that are not free
// among them, spent its time starting blocks (3000 atoms, 129^3: 850 -> 216 us
// for all marks, with the three sets of an axis in one launch; a warp per
// sphere with the unfree ones skipped, 272 us). Where the spheres are fewer
// than the grid's warps, each is split over as many warps as there are for it:
// a few large spheres (fine grids) otherwise leave most of the GPU idle (12
// atoms, 129^3 points 0.05 A apart: whole set-up 33 ms with a warp per sphere,
// 6.3 with a block per sphere, 1.3 so).
__global__ void __launch_bounds__(kSetupThreads)
    mark_spheres_kernel(int n, double h, SphereSets sets) {
  const int lane = threadIdx.x & 31;
  const unsigned warps = (gridDim.x * blockDim.x) >> 5;
  unsigned count[3]; // (their sum may pass 2^31)
#pragma unroll
  for (int t = 0; t < 3; ++t)
    count[t] =
        sets.set[t].count_dev ? *sets.set[t].count_dev : sets.set[t].count;
  const unsigned total = count[0] + count[1] + count[2];
  const unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned parts = total < warps ? warps / total : 1; // (total > 0)
  const unsigned part = w % parts;
  for (unsigned g = w / parts; g < total; g += warps / parts) {
    if (g < count[0])
      mark_sphere(n, h, sets.set[0], sets.axis, (int)g, part, parts, lane);
    else if (g < count[0] + count[1])
      mark_sphere(n, h, sets.set[1], sets.axis, (int)(g - count[0]), part,
                  parts, lane);
    else
      mark_sphere(n, h, sets.set[2], sets.axis,
                  (int)(g - count[0] - count[1]), part, parts, lane);
  }
}
// Blocks for the sets, whose radii are at most rmax: a warp per 32 columns of
// every sphere, up to a grid that fills the GPU once.
unsigned mark_blocks(const SphereSets &s, int n, double h, double rmax) {
  const double q = (double)s.set[0].count + s.set[1].count + s.set[2].count;
  const double side = std::min(2.0 * rmax / h + 2.0, (double)n);
  const double warps = q * std::ceil(side * side / 32.0);
  return (unsigned)std::min(std::ceil(warps * 32.0 / kSetupThreads),
                            148.0 * 8);
}

__global__ void face_from_masks_kernel(long count, const unsigned char *inside,
                                       const unsigned char *sas,
                                       const unsigned char *carved,
                                       double v_in, double v_out,
                                       double *face) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < count;
       q += (long)gridDim.x * blockDim.x) {
    const bool solute = inside[q] || (sas && sas[q] && !carved[q]);
    face[q] = solute ? v_in : v_out;
  }
}

// oC = sum of the six faces (+ kappa^2 eps_out outside the ion-exclusion
// spheres) on the interior, 0 on the shell; the host's summation order.
__global__ void centre_kernel(int n, const double *uC, const double *oN,
                              const double *oE, const unsigned char *ion,
                              double kterm, double *oC) {
  const long n3 = (long)n * n * n;
  const long s1 = n, s0 = (long)n * n;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n3;
       q += (long)gridDim.x * blockDim.x) {
    const long i0 = q / s0, i1 = (q / s1) % n, i2 = q % n;
    if (i0 < 1 || i1 < 1 || i2 < 1 || i0 > n - 2 || i1 > n - 2 ||
        i2 > n - 2) {
      oC[q] = 0.0;
      continue;
    }
    double c = ((uC[q] + uC[q - s0]) + (oN[q] + oN[q - s1])) +
               (oE[q] + oE[q - 1]);
    c += ion[q] ? 0.0 : kterm;
    oC[q] = c;
  }
}

// Trilinear charge records in atom order: key = grid point (or INT_MAX when
// the corner is outside the grid), value = 8 * atom + corner.
__global__ void charge_records_kernel(const double *atoms, int natoms, int n,
                                      double h, int *keys, int *vals) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= 8 * natoms)
    return;
  const int a = r >> 3, corner = r & 7;
  long c[3];
  for (int d = 0; d < 3; ++d) {
    const double s = atoms[5 * a + d] / h;
    const long lo = (long)s;
    c[d] = lo + ((corner >> d) & 1);
  }
  const bool in = c[0] < n && c[1] < n && c[2] < n;
  keys[r] = in ? (int)((c[0] * n + c[1]) * n + c[2]) : 0x7fffffff;
  vals[r] = r;
}

// Sums every run of equal keys in record order (= atom order):
// f[q] = ((0 + t_1) + t_2) + ..., t = charge * wt / vol as on the host.
__global__ void charge_sum_kernel(const double *atoms, int nrec, double h,
                                  double eps0, double vol,
                                  const int *keys, const int *vals,
                                  double *f) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrec || keys[r] == 0x7fffffff)
    return;
  if (r > 0 && keys[r - 1] == keys[r])
    return; // not the head of its run
  double acc = 0.0;
  for (int t = r; t < nrec && keys[t] == keys[r]; ++t) {
    const int a = vals[t] >> 3, corner = vals[t] & 7;
    const double charge = atoms[5 * a + 4] / eps0;
    double wt = 1;
    for (int d = 0; d < 3; ++d) {
      const double s = atoms[5 * a + d] / h;
      const long lo = (long)s;
      const double w = ((corner >> d) & 1) ? (s - lo) : (lo + 1 - s);
      wt *= w;
    }
    acc += charge * wt / vol;
  }
  f[keys[r]] = acc;
}

// Probe centres on the sphere of radius r_a + probe around every atom; a
// centre is kept when no other inflated sphere contains it
// (d^2 < R_b^2 (1 - 1e-12), the host's test). Output: the kept centres as rows
// (x, y, z), in any order (their marks do not depend on it), *kept of them. The
// atoms are found through a cell list: a centre lies within the largest
// inflated radius (<= the cell edge) of any sphere containing it, so only
// the 27 cells around it are searched; "kept" is an AND over atoms, so the
// order of the atoms within a cell does not matter.
__global__ void __launch_bounds__(kSetupThreads)
    probe_centres_cells_kernel(const double *atoms, int natoms, double probe,
                               const ProbeDir *dirs, double cell, int dim,
                               const int *cell_start, const int *cell_atoms,
                               double *centres, int *kept) {
  const long g = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (g >= (long)natoms * kProbePoints)
    return;
  const int a = (int)(g / kProbePoints), s = (int)(g % kProbePoints);
  const double R = atoms[5 * a + 3] + probe;
  const ProbeDir u = dirs[s];
  double pc[3];
  pc[0] = atoms[5 * a] + R * u.rr * u.c;
  pc[1] = atoms[5 * a + 1] + R * u.rr * u.s;
  pc[2] = atoms[5 * a + 2] + R * u.zz;
  int cc[3];
  for (int d = 0; d < 3; ++d)
    cc[d] = (int)floor(pc[d] / cell);
  bool free = true;
  for (int dz = -1; dz <= 1 && free; ++dz)
    for (int dy = -1; dy <= 1 && free; ++dy)
      for (int dx = -1; dx <= 1 && free; ++dx) {
        const int c0 = cc[0] + dx, c1 = cc[1] + dy, c2 = cc[2] + dz;
        if (c0 < 0 || c1 < 0 || c2 < 0 || c0 >= dim || c1 >= dim ||
            c2 >= dim)
          continue;
        const int cid = (c2 * dim + c1) * dim + c0;
        for (int q = cell_start[cid]; q < cell_start[cid + 1]; ++q) {
          const int b = cell_atoms[q];
          if (b == a)
            continue;
          const double Rb = atoms[5 * b + 3] + probe;
          double d2 = 0;
          for (int d = 0; d < 3; ++d) {
            const double e = pc[d] - atoms[5 * b + d];
            d2 += e * e;
          }
          if (d2 < Rb * Rb * (1 - 1e-12)) {
            free = false;
            break;
          }
        }
      }
  if (!free)
    return;
  const size_t slot = (size_t)atomicAdd(kept, 1); // (3 slot may pass 2^31)
  centres[3 * slot + 0] = pc[0];
  centres[3 * slot + 1] = pc[1];
  centres[3 * slot + 2] = pc[2];
}

// Cell list of the atoms: cell of each atom and per-cell counts
__global__ void atom_cells_kernel(const double *atoms, int natoms, double cell,
                                  int dim, int *cid, int *count) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= natoms)
    return;
  int c[3];
  for (int d = 0; d < 3; ++d)
    c[d] = min((int)floor(atoms[5 * a + d] / cell), dim - 1);
  cid[a] = (c[2] * dim + c[1]) * dim + c[0];
  atomicAdd(&count[cid[a]], 1);
}

// atoms into their cells' ranges (fill: a copy of the ranges' starts)
__global__ void atom_scatter_kernel(int natoms, const int *cid, int *fill,
                                    int *cell_atoms) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < natoms)
    cell_atoms[atomicAdd(&fill[cid[a]], 1)] = a;
}

// ---- multiple Debye-Hueckel boundary ----------------------------------------
// x0(p) = sum over atoms of f_a exp(-kappa (d - r_a)) / d on the six faces,
// f_a = q / (pref (1 + kappa r_a)). 10^8 to 10^9 terms in double, bound by the
// FP64 units: with CUDA's sqrt, exp and divide a term is ~88 of their
// operations. Here it is ~27:
//   * a thread takes kDhPoints points of one face row, which share two of the
//     three squared distances;
//   * 1 / d from the hardware's reciprocal square root estimate and one
//     third-order correction (relative error e -> O(e^3), e <= 2^-20), d as
//     d^2 / d;
//   * exp by a table of 2^(j/64) and a degree-5 polynomial (Tang, ACM TOMS
//     15, 1989): y = d' (-kappa 64 / ln 2) = m + f, the product in two parts
//     so that f keeps its last bits, exp = 2^(m/64) e^(f ln 2 / 64).
// That holds for normal results and a 32-bit m. The host bounds the arguments
// by the grid's diagonal and the largest radius; beyond +-700 the kernel with
// CHECK runs, whose threads take CUDA's exp for the four points of an atom
// where one of them needs it (in the usual range the checks cost 6%: 129^3,
// 3000 atoms, 80 registers in place of 64).
// The block's eight warps take the same points and every eighth atom each;
// their sums are added in warp order (deterministic; without that split a
// 65^3 grid has too few points to fill the GPU). Every face point belongs to
// one thread. 3000 atoms, 129^3: 1.43 -> 0.63 ms; against long double, the
// largest error relative to the sum of the terms' sizes 3.6e-16 -> 1.4e-16.
constexpr int kDhPoints = 4;
constexpr int kDhWarps = 8;
// (ln 2 / 64)^k / k!
__device__ constexpr double kDhTerm[6] = {1.0,
                                          0.010830424696249145,
                                          5.86490495505617e-05,
                                          2.1173137155464776e-07,
                                          5.732851688640402e-10,
                                          1.2417843701716925e-12};

struct DhParams {
  int n;
  double h, pref, kappa;
  double khi, klo; // -kappa 64 / ln 2 = khi + klo
};

// exp(-kappa (d - r)) from the squared distance, for any argument
__device__ __noinline__ double dh_exp(double kappa, double d2, double r) {
  return exp(-kappa * (sqrt(d2) - r));
}

// the plain sum at one point (where the fast one met a zero distance)
__device__ double dh_plain(const double *atoms, int natoms, const DhParams &b,
                           long i0, long i1, long i2) {
  double acc = 0.0;
  for (int t = 0; t < natoms; ++t) {
    const double *at = atoms + 5 * t;
    const double d0 = i0 * b.h - at[0], d1 = i1 * b.h - at[1],
                 d2 = i2 * b.h - at[2];
    const double dist = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    acc += at[4] / (b.pref * (1 + b.kappa * at[3])) *
           exp(-b.kappa * (dist - at[3])) / dist;
  }
  return acc;
}

template <bool CHECK>
__global__ void __launch_bounds__(32 * kDhWarps)
    boundary_kernel(const double *__restrict__ atoms, int natoms, DhParams b,
                    double *__restrict__ x0) {
  constexpr int kTile = 32 * kDhWarps;
  __shared__ double sa[kTile * 5];
  __shared__ double table[64];
  __shared__ double part[kDhWarps][32 * kDhPoints];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 64)
    table[threadIdx.x] = exp2(threadIdx.x / 64.0);
  // the thread's points: face, row a, points from c on. Faces 0, 1: i0 = 0,
  // n - 1 over all (i1, i2); 2, 3: i1 = 0, n - 1 over interior i0, all i2;
  // 4, 5: i2 = 0, n - 1 over interior i0 and i1.
  const int n = b.n, groups = (n + kDhPoints - 1) / kDhPoints;
  const long rows01 = n, rows = n - 2;
  long t = blockIdx.x * 32L + lane;
  long row = t / groups;
  const int c = (int)(t - row * groups) * kDhPoints;
  int face = -1;
  long a = 0;
  if (row < 2 * rows01) {
    face = row < rows01 ? 0 : 1;
    a = row - face * rows01;
  } else if (row < 2 * rows01 + 4 * rows) {
    row -= 2 * rows01;
    face = 2 + (int)(row / rows);
    a = 1 + row % rows;
  }
  const int ax = face < 2 ? 0 : face < 4 ? 1 : 2; // the face's axis
  const int row_ax = ax == 0 ? 1 : 0;             // of a
  const int run_ax = ax == 2 ? 1 : 2;             // of the thread's points
  const double xa = (face & 1) ? (n - 1) * b.h : 0.0;
  const double xr = a * b.h;
  double xc[kDhPoints], acc[kDhPoints];
#pragma unroll
  for (int q = 0; q < kDhPoints; ++q) {
    xc[q] = (c + q) * b.h;
    acc[q] = 0.0;
  }
  for (int b0 = 0; b0 < natoms; b0 += kTile) {
    __syncthreads();
    if (b0 + (int)threadIdx.x < natoms) {
      const double *at = atoms + 5 * (size_t)(b0 + threadIdx.x);
      double *o = sa + 5 * threadIdx.x;
      for (int d = 0; d < 4; ++d)
        o[d] = at[d];
      o[4] = at[4] / (b.pref * (1 + b.kappa * at[3]));
    }
    __syncthreads();
    const int nb = natoms - b0 < kTile ? natoms - b0 : kTile;
    if (face < 0)
      continue;
    for (int u = warp; u < nb; u += kDhWarps) {
      const double *at = sa + 5 * u;
      const double da = xa - at[ax], dr = xr - at[row_ax];
      const double s = fma(da, da, dr * dr), pos = at[run_ax];
      const double rad = at[3], fac = at[4];
      double w[kDhPoints], inv[kDhPoints];
      bool out = false;
#pragma unroll
      for (int q = 0; q < kDhPoints; ++q) {
        const double dc = xc[q] - pos;
        const double d2 = fma(dc, dc, s);
        double y;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d2));
        const double e = fma(-d2 * y, y, 1.0);
        y = fma(y * e, fma(e, 0.375, 0.5), y);
        const double dist = fma(d2, y, -rad); // minus the radius
        // m = the nearest integer, by the addend 1.5 2^52
        const double big = fma(dist, b.khi, 6755399441055744.0);
        const int m = __double2loint(big);
        const double mr = big - 6755399441055744.0;
        const double f = fma(dist, b.klo, fma(dist, b.khi, -mr));
        double p = fma(f, kDhTerm[5], kDhTerm[4]);
        p = fma(f, p, kDhTerm[3]);
        p = fma(f, p, kDhTerm[2]);
        p = f * fma(f, p, kDhTerm[1]);
        double v = table[m & 63];
        v = fma(v, p, v);
        const int k = m >> 6;
        w[q] = __hiloint2double(__double2hiint(v) + (k << 20),
                                __double2loint(v));
        inv[q] = y;
        // v >= 2^-1: a normal result for k in [-1021, 1023]; the upper half
        // of the addend, with m's sign, where m has 32 bits
        if constexpr (CHECK)
          out |= (unsigned)(k + 1021) > 2044u ||
                 __double2hiint(big) != 0x43380000 + (m >> 31);
      }
      if (CHECK && out) {
#pragma unroll
        for (int q = 0; q < kDhPoints; ++q) {
          const double dc = xc[q] - pos;
          w[q] = dh_exp(b.kappa, fma(dc, dc, s), rad);
        }
      }
#pragma unroll
      for (int q = 0; q < kDhPoints; ++q)
        acc[q] = fma(fac * w[q], inv[q], acc[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < kDhPoints; ++q)
    part[warp][q * 32 + lane] = acc[q];
  __syncthreads();
  if (warp >= kDhPoints || face < 0)
    return;
  const int i = c + warp; // warp q adds up the points q
  if (i >= n || (face >= 4 && (i < 1 || i > n - 2)))
    return;
  double v = 0.0;
  for (int w = 0; w < kDhWarps; ++w)
    v += part[w][warp * 32 + lane];
  const long end = (face & 1) ? n - 1 : 0;
  const long i0 = ax == 0 ? end : a;
  const long i1 = ax == 0 ? a : ax == 1 ? end : i;
  const long i2 = ax == 2 ? end : i;
  if (!isfinite(v))
    v = dh_plain(atoms, natoms, b, i0, i1, i2);
  x0[((size_t)i0 * n + i1) * n + i2] = v;
}

unsigned grid_for(long count) {
  const long b = (count + kSetupThreads - 1) / kSetupThreads;
  return (unsigned)(b < 1 ? 1 : (b > 148L * 32 ? 148L * 32 : b));
}

// Stream-ordered scratch freed at scope exit (after the work queued on the
// stream, by stream order).
struct Scratch {
  cudaStream_t s;
  std::vector<void *> ptrs;
  explicit Scratch(cudaStream_t st) : s(st) {}
  ~Scratch() {
    for (void *p : ptrs)
      scratch_free(p, s);
  }
  template <typename T> cudaError_t take(T **p, size_t count) {
    void *q = nullptr;
    const cudaError_t e = scratch_alloc(&q, sizeof(T) * (count ? count : 1),
                                        s);
    if (e == cudaSuccess)
      ptrs.push_back(q);
    *p = (T *)q;
    return e;
  }
};

} // namespace

// Device set-up into device arrays; atoms are host rows (validated here).
int setup_fine_device(int n, double h, const double *atoms_host, int natoms,
                      const pmg_physics *ph, double *oC, double *oE,
                      double *oN, double *uC, double *f, double *x0,
                      cudaStream_t st) {
  if (n < 3 || n > 1025 || !(h > 0) || (natoms > 0 && !atoms_host) ||
      natoms < 0 || !ph || !oC || !oE || !oN || !uC || !f || !x0) {
    set_last_message("setup_fine_device: bad argument");
    return PMG_ERR_ARG;
  }
  const bool probe = ph->probe_radius > 0;
  if (probe && (long)natoms * kProbePoints > INT_MAX) {
    set_last_message("setup_fine_device: more than 2^31 probe positions");
    return PMG_ERR_ARG;
  }
  for (int a = 0; a < natoms; ++a) {
    for (int d = 0; d < 3; ++d) {
      const double x = atoms_host[5 * a + d];
      if (!(x >= 0 && x <= h * (n - 1))) {
        set_last_message("setup_fine_device: atom outside the grid");
        return PMG_ERR_ARG;
      }
    }
    if (!(atoms_host[5 * a + 3] >= 0)) {
      set_last_message("setup_fine_device: negative radius");
      return PMG_ERR_ARG;
    }
  }
  double rmax = 0.0;
  for (int a = 0; a < natoms; ++a)
    rmax = std::max(rmax, atoms_host[5 * a + 3]);
  const long n3 = (long)n * n * n;
  const Physics p = physics(*ph);
  const double h2 = h * h;
  const double v_out = p.eps_out / h2, v_in = p.eps_in / h2;
  Scratch sc(st);
  double *d_atoms = nullptr;
  unsigned char *inside = nullptr, *sas = nullptr, *carved = nullptr,
                *ion = nullptr;
  double *centres = nullptr;
  int *kept = nullptr; // probe centres kept (device)
  ProbeDir *d_dirs = nullptr;
  PMG_CUDA_TRY(sc.take(&d_atoms, 5 * (size_t)natoms));
  // inside, and with a probe sas and carved: one block, cleared by one memset
  const long mask_n = (n3 + 15) & ~15L;
  const size_t mask_bytes = (probe && natoms > 0 ? 3 : 1) * mask_n;
  PMG_CUDA_TRY(sc.take(&inside, mask_bytes));
  PMG_CUDA_TRY(sc.take(&ion, n3));
  if (natoms > 0)
    PMG_CUDA_TRY(cudaMemcpyAsync(d_atoms, atoms_host,
                                 sizeof(double) * 5 * natoms,
                                 cudaMemcpyHostToDevice, st));
  if (probe && natoms > 0) {
    ProbeDir dirs[kProbePoints];
    probe_directions(dirs);
    sas = inside + mask_n;
    carved = sas + mask_n;
    PMG_CUDA_TRY(sc.take(&centres, 3 * (size_t)natoms * kProbePoints));
    PMG_CUDA_TRY(sc.take(&d_dirs, kProbePoints));
    PMG_CUDA_TRY(cudaMemcpyAsync(d_dirs, dirs, sizeof(dirs),
                                 cudaMemcpyHostToDevice, st));
    const long np = (long)natoms * kProbePoints;
    const unsigned pgrid = (unsigned)((np + kSetupThreads - 1) / kSetupThreads);
    // cell list of the atoms, built on the stream: edge >= the largest
    // inflated radius, at most 64 cells per axis of the grid's extent
    const double extent = h * (n - 1);
    const double cell = std::max(rmax + ph->probe_radius, extent / 63);
    const int dim = (int)(extent / cell) + 1;
    const int ncells = dim * dim * dim;
    int *d_cid = nullptr, *d_count = nullptr, *d_cstart = nullptr,
        *d_fill = nullptr, *d_cat = nullptr;
    PMG_CUDA_TRY(sc.take(&d_cid, (size_t)natoms));
    PMG_CUDA_TRY(sc.take(&d_count, (size_t)ncells + 2));
    kept = d_count + ncells + 1;
    PMG_CUDA_TRY(sc.take(&d_cstart, (size_t)ncells + 1));
    PMG_CUDA_TRY(sc.take(&d_fill, (size_t)ncells + 1));
    PMG_CUDA_TRY(sc.take(&d_cat, (size_t)natoms));
    PMG_CUDA_TRY(
        cudaMemsetAsync(d_count, 0, sizeof(int) * (ncells + 2), st));
    atom_cells_kernel<<<(natoms + 255) / 256, 256, 0, st>>>(
        d_atoms, natoms, cell, dim, d_cid, d_count);
    size_t scan_bytes = 0;
    PMG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, d_count,
                                               d_cstart, ncells + 1, st));
    unsigned char *scan_tmp = nullptr;
    PMG_CUDA_TRY(sc.take(&scan_tmp, scan_bytes));
    PMG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, d_count,
                                               d_cstart, ncells + 1, st));
    PMG_CUDA_TRY(cudaMemcpyAsync(d_fill, d_cstart,
                                 sizeof(int) * (ncells + 1),
                                 cudaMemcpyDeviceToDevice, st));
    atom_scatter_kernel<<<(natoms + 255) / 256, 256, 0, st>>>(
        natoms, d_cid, d_fill, d_cat);
    probe_centres_cells_kernel<<<pgrid, kSetupThreads, 0, st>>>(
        d_atoms, natoms, ph->probe_radius, d_dirs, cell, dim, d_cstart, d_cat,
        centres, kept);
    PMG_LAUNCH_CHECK();
  }

  // face coefficients, axis 0 -> uC, 1 -> oN, 2 -> oE
  double *face[3] = {uC, oN, oE};
  const int np = probe ? natoms * kProbePoints : 0;
  for (int axis = 0; axis < 3; ++axis) {
    PMG_CUDA_TRY(cudaMemsetAsync(inside, 0, mask_bytes, st));
    if (natoms > 0) {
      SphereSets m{};
      m.axis = axis;
      m.set[0] = SphereSet{d_atoms, 5, natoms, d_atoms + 3, 0.0, nullptr,
                           inside};
      if (probe) {
        m.set[1] = SphereSet{d_atoms,          5,       natoms, d_atoms + 3,
                             ph->probe_radius, nullptr, sas};
        m.set[2] = SphereSet{centres,          3,         np, nullptr,
                             ph->probe_radius, kept, carved};
      }
      const unsigned blocks = mark_blocks(
          m, n, h, probe ? rmax + ph->probe_radius : rmax);
      mark_spheres_kernel<<<blocks, kSetupThreads, 0, st>>>(n, h, m);
    }
    face_from_masks_kernel<<<grid_for(n3), kSetupThreads, 0, st>>>(
        n3, inside, probe && natoms > 0 ? sas : nullptr, carved, v_in, v_out,
        face[axis]);
    PMG_LAUNCH_CHECK();
  }

  // ion-exclusion mask and the centre coefficient
  PMG_CUDA_TRY(cudaMemsetAsync(ion, 0, n3, st));
  if (natoms > 0) {
    SphereSets m{};
    m.axis = -1;
    m.set[0] = SphereSet{d_atoms, 5, natoms, d_atoms + 3, ph->ion_radius,
                         nullptr, ion};
    mark_spheres_kernel<<<mark_blocks(m, n, h, rmax + ph->ion_radius),
                          kSetupThreads, 0, st>>>(n, h, m);
  }
  centre_kernel<<<grid_for(n3), kSetupThreads, 0, st>>>(
      n, uC, oN, oE, ion, p.kappa * p.kappa * p.eps_out, oC);
  PMG_LAUNCH_CHECK();

  // charges
  PMG_CUDA_TRY(cudaMemsetAsync(f, 0, sizeof(double) * n3, st));
  if (natoms > 0) {
    const int nrec = 8 * natoms;
    int *k_in, *k_out, *v_in_, *v_out_;
    PMG_CUDA_TRY(sc.take(&k_in, nrec));
    PMG_CUDA_TRY(sc.take(&k_out, nrec));
    PMG_CUDA_TRY(sc.take(&v_in_, nrec));
    PMG_CUDA_TRY(sc.take(&v_out_, nrec));
    charge_records_kernel<<<(nrec + 255) / 256, 256, 0, st>>>(
        d_atoms, natoms, n, h, k_in, v_in_);
    PMG_LAUNCH_CHECK();
    size_t tmp_bytes = 0;
    PMG_CUDA_TRY(cub::DeviceRadixSort::SortPairs(
        nullptr, tmp_bytes, k_in, k_out, v_in_, v_out_, nrec, 0, 32, st));
    unsigned char *tmp = nullptr;
    PMG_CUDA_TRY(sc.take(&tmp, tmp_bytes));
    PMG_CUDA_TRY(cub::DeviceRadixSort::SortPairs(
        tmp, tmp_bytes, k_in, k_out, v_in_, v_out_, nrec, 0, 32, st));
    charge_sum_kernel<<<(nrec + 255) / 256, 256, 0, st>>>(
        d_atoms, nrec, h, p.eps0, h * (h * h), k_out, v_out_, f);
    PMG_LAUNCH_CHECK();
  }

  // Debye-Hueckel boundary
  PMG_CUDA_TRY(cudaMemsetAsync(x0, 0, sizeof(double) * n3, st));
  if (natoms > 0) {
    DhParams b{n, h, 4 * kPi * (p.eps0 * p.eps_out), p.kappa, 0.0, 0.0};
    // -kappa 64 / ln 2 to about 100 bits
    const long double k = -(long double)p.kappa * 64.0L /
                          0.693147180559945309417232121458176568L;
    b.khi = (double)k;
    b.klo = (double)(k - b.khi);
    const long threads =
        (2L * n + 4L * (n - 2)) * ((n + kDhPoints - 1) / kDhPoints);
    const double reach = std::max(2.0 * h * (n - 1), rmax); // over sqrt(3)
    const unsigned blocks = (unsigned)((threads + 31) / 32);
    if (p.kappa * reach <= 700.0)
      boundary_kernel<false>
          <<<blocks, 32 * kDhWarps, 0, st>>>(d_atoms, natoms, b, x0);
    else
      boundary_kernel<true>
          <<<blocks, 32 * kDhWarps, 0, st>>>(d_atoms, natoms, b, x0);
    PMG_LAUNCH_CHECK();
  }
  return PMG_OK;
}

} // namespace pmg

extern "C" int pmg_setup_fine_d(int n, double h, const double *atoms,
                                int natoms, const pmg_physics *phys,
                                double *oC, double *oE, double *oN,
                                double *uC, double *f, double *x0,
                                pmg_stream_t stream) {
  return pmg::setup_fine_device(n, h, atoms, natoms, phys, oC, oE, oN, uC, f,
                                x0, (cudaStream_t)stream);
}
