// Pseudo-atomic orbital tabulation on the grid (FP64).
//
//   phi_{l,p,m}(r) = R_{lp}(|r - tau|) * Y_lm(angles of r - tau)
//
// on every point of each atom's cutoff-sphere list, and with GRAD the
// gradient tables of Set_dOrbitals_Grid.  Follows
// src/Matrix/Set_Orbitals_Grid.jl:94-274 and
// src/Matrix/Set_dOrbitals_Grid.jl:88-359: the same radial spline (binary
// search on the PAO log mesh + 4-point Hermite cubic, polynomial extrapolation
// below RV[1], zero beyond RV[end]), real Y_lm for l <= 3 in the reference's
// m order, and the reference's derivative chain rule with the 1e-13 shift of
// points that sit on the atom.
//
// Both kernels take the spline from per-interval cubic coefficients computed
// once per species on the host (the same Hermite interpolant: value and slope
// at both mesh nodes of the interval, written as c0 + c1 u + c2 u^2 + c3 u^3
// in u = (R - RV[m-1]) / (RV[m] - RV[m-1])), find the interval from a table of
// log2(R) buckets and a short forward scan instead of a binary search, and
// form Y_lm from the unit vector (x, y, z)/R (the edge convention of
// src/utils/xyz_to_spherical.jl, theta = pi/2 and phi = 0 at R < 1e-14, is
// kept).  That takes the FP64 work per point from the spline's divisions and
// the per-function Hermite set-up to one Horner evaluation per radial function.
//
// The gradients are taken in Cartesian form.  With Y = P(x, y, z) of degree l
// on the unit sphere, G = grad P there, and q = R_lp / r,
//
//   grad phi = (R_lp' - l q) Y u + q G,   u = (x, y, z)/r,
//
// seven FP64 operations per function on top of its value (G is shared by the
// functions of one l), where the reference's chain rule over r, theta and phi
// (the same derivative, src/Matrix/Set_dOrbitals_Grid.jl:257-300) needs twenty
// and the angles' sines and cosines.  Both kernels are bound by the FP64 pipe
// (two operations a clock and SM): values and gradients of a random 16-atom
// 13-orbital cell took 1.90 ms by the chain rule and 0.49 ms this way.  The
// code of one l at a time, with compile-time loops over m, keeps Y and G in
// registers: the same cell's values alone took 0.33 ms with a loop over l
// that indexed them in local memory, and 0.22 ms.
//
// One thread per sphere point; a block stages its points x NO values per
// table in shared memory and writes them back as contiguous, 16-byte
// vectorised stores (the table is point-major, NO values per point).
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "lcp_device.h"

namespace lcp {

namespace {

constexpr int kTabPoints = 64;  // points of a gradient block: four tables of staging
constexpr double kPi = 3.14159265358979323846;

// Real Y_lm of one l in the orbital order of src/Matrix/Set_Orbitals_Grid.jl:242-268
// (src/utils/Ylm_real.jl:1-53), from the unit vector u = (x, y, z) / R:
// sin(theta) cos(phi) = ux, sin(theta) sin(phi) = uy, cos(theta) = uz.
__device__ __forceinline__ void ylm_unit(int l, double ux, double uy, double uz, double* Y) {
  const double pi = kPi;
  if (l == 0) {
    Y[0] = 0.5 * sqrt(1 / pi);
  } else if (l == 1) {
    const double c = sqrt(3 / 4.0 / pi);
    Y[0] = c * ux;
    Y[1] = c * uy;
    Y[2] = c * uz;
  } else if (l == 2) {
    const double s = sqrt(15 / pi);
    Y[0] = 0.25 * sqrt(5 / pi) * (3 * uz * uz - 1);
    Y[1] = 0.25 * s * (ux * ux - uy * uy);
    Y[2] = 0.5 * s * ux * uy;
    Y[3] = 0.5 * s * ux * uz;
    Y[4] = 0.5 * s * uy * uz;
  } else {
    const double a = sqrt(35 / 2.0 / pi), b = sqrt(105 / pi), c = sqrt(21 / 2.0 / pi), d = sqrt(7 / pi);
    const double z2 = uz * uz;
    Y[0] = 0.25 * d * (5 * z2 * uz - 3 * uz);
    Y[1] = 0.25 * c * ux * (5 * z2 - 1);
    Y[2] = 0.25 * c * uy * (5 * z2 - 1);
    Y[3] = 0.25 * b * uz * (ux * ux - uy * uy);
    Y[4] = 0.5 * b * uz * ux * uy;
    Y[5] = 0.25 * a * (ux * ux * ux - 3 * ux * uy * uy);
    Y[6] = 0.25 * a * (3 * ux * ux * uy - uy * uy * uy);
  }
}

// Gradients of the Y_lm's homogeneous polynomials at the unit vector.
template <int l>
__device__ __forceinline__ void ylm_grad(double ux, double uy, double uz, double (*G)[3]) {
  const double pi = kPi;
  if (l == 0) {
    G[0][0] = G[0][1] = G[0][2] = 0.0;
  } else if (l == 1) {
    const double c = sqrt(3 / 4.0 / pi);
    for (int m = 0; m < 3; ++m)
      for (int d = 0; d < 3; ++d) G[m][d] = m == d ? c : 0.0;
  } else if (l == 2) {
    const double s = 0.5 * sqrt(15 / pi), k = 0.5 * sqrt(5 / pi);
    G[0][0] = -k * ux, G[0][1] = -k * uy, G[0][2] = 2 * k * uz;  // k/2 (2 z^2 - x^2 - y^2)
    G[1][0] = s * ux, G[1][1] = -s * uy, G[1][2] = 0.0;          // s/2 (x^2 - y^2)
    G[2][0] = s * uy, G[2][1] = s * ux, G[2][2] = 0.0;           // s x y
    G[3][0] = s * uz, G[3][1] = 0.0, G[3][2] = s * ux;           // s x z
    G[4][0] = 0.0, G[4][1] = s * uz, G[4][2] = s * uy;           // s y z
  } else {
    const double a = 0.75 * sqrt(35 / 2.0 / pi), b = 0.5 * sqrt(105 / pi), c = 0.25 * sqrt(21 / 2.0 / pi),
                 d = 0.75 * sqrt(7 / pi);
    const double xx = ux * ux, yy = uy * uy, zz = uz * uz, xy = ux * uy, xz = ux * uz, yz = uy * uz;
    G[0][0] = -2 * d * xz, G[0][1] = -2 * d * yz, G[0][2] = d * (2 * zz - xx - yy);             // d/3 (2 z^3 - 3 z (x^2 + y^2))
    G[1][0] = c * (4 * zz - 3 * xx - yy), G[1][1] = -2 * c * xy, G[1][2] = 8 * c * xz;          // c x (4 z^2 - x^2 - y^2)
    G[2][0] = -2 * c * xy, G[2][1] = c * (4 * zz - xx - 3 * yy), G[2][2] = 8 * c * yz;          // c y (4 z^2 - x^2 - y^2)
    G[3][0] = b * xz, G[3][1] = -b * yz, G[3][2] = 0.5 * b * (xx - yy);                         // b/2 z (x^2 - y^2)
    G[4][0] = b * yz, G[4][1] = b * xz, G[4][2] = b * xy;                                       // b x y z
    G[5][0] = a * (xx - yy), G[5][1] = -2 * a * xy, G[5][2] = 0.0;                              // a/3 (x^3 - 3 x y^2)
    G[6][0] = 2 * a * xy, G[6][1] = a * (xx - yy), G[6][2] = 0.0;                               // a/3 (3 x^2 y - y^3)
  }
}

// A sphere point relative to its atom.
__device__ __forceinline__ void point_xyz(const DevGeom& g, int atom, int64_t k, double* xyz) {
  const int gn = g.glist[k];
  const int cell = g.clist[k];
  const int N2 = g.ngrid[1], N3 = g.ngrid[2];
  const int n1 = gn / (N2 * N3);
  const int n2 = (gn - n1 * N2 * N3) / N3;
  const int n3 = gn - n1 * N2 * N3 - n2 * N3;
  for (int d = 0; d < 3; ++d) {
    double c = n1 * g.glat[0 * 3 + d] + n2 * g.glat[1 * 3 + d] + n3 * g.glat[2 * 3 + d] + g.origin[d];
    xyz[d] = c + g.atv[cell * 3 + d] - g.gxyz[atom * 3 + d];
  }
}

// Where a point lies on a species' radial mesh: its distance, unit vector and
// interval record (none beyond RV[n-1] and, with inner, below RV[0]).
struct TabPoint {
  double R, ir, ux, uy, uz, u;
  const double* rec;
  int m;
  bool inner;
};
__device__ __forceinline__ TabPoint locate(const DevSpecies& sp, const double* __restrict__ radial,
                                           const int32_t* __restrict__ buckets, const double* xyz) {
  TabPoint q;
  const double r2 = xyz[0] * xyz[0] + xyz[1] * xyz[1] + xyz[2] * xyz[2];
  if (r2 < 1e-28) {
    // R < 1e-14: theta = pi/2, phi = 0 (src/utils/xyz_to_spherical.jl)
    q.R = sqrt(r2);
    q.ir = 0.0;
    q.ux = 1.0;
    q.uy = 0.0;
    q.uz = 6.123233995736766e-17;  // cos(pi/2) in double precision
  } else {
    q.ir = rsqrt(r2);
    q.R = r2 * q.ir;
    q.ux = xyz[0] * q.ir;
    q.uy = xyz[1] * q.ir;
    q.uz = xyz[2] * q.ir;
  }
  const int n = sp.nmesh;
  const double* rv = radial + sp.rv_off;
  const bool outside = rv[n - 1] < q.R;
  q.inner = q.R < rv[0];
  q.rec = nullptr;
  q.m = 0;
  q.u = 0.0;
  if (!outside && !q.inner) {
    // the interval: first mesh index >= 1 with RV >= R, from one bucket down
    int b = (int)((__log2f((float)q.R) - sp.bk_lo) * sp.bk_inv) - 1;
    b = min(max(b, 0), kSplineBuckets - 1);
    int i = buckets[sp.bk_off + b];
    while (i < n - 1 && rv[i] < q.R) ++i;
    q.m = min(max(i, 2), n - 2);
    q.rec = radial + sp.iv_off + (size_t)q.m * (2 + 4 * sp.nrad);
    q.u = (q.R - q.rec[0]) * q.rec[1];
  }
  return q;
}

// The functions of one l at a point: values (WPHI), and the gradients with
// respect to the atom's position (WGRAD: -grad phi, as the reference's tables).
template <int l, bool WPHI, bool WGRAD>
__device__ __forceinline__ void eval_l(const DevSpecies& sp, const double* __restrict__ radial, const TabPoint& q,
                                       int& rad, int& ist, double* srow, double* sx, double* sy, double* sz) {
  double Y[2 * l + 1], G[2 * l + 1][3];
  ylm_unit(l, q.ux, q.uy, q.uz, Y);
  if (WGRAD) ylm_grad<l>(q.ux, q.uy, q.uz, G);
  // the last interval's values have f4 = f1, its gradients have not (record nmesh - 1)
  const bool last = q.rec && q.m == sp.nmesh - 2;
  const double* grec = last ? q.rec + 2 + 4 * sp.nrad : q.rec;
  for (int p = 0; p < sp.nb[l]; ++p, ++rad) {
    double rf = 0.0, rg = 0.0, dr = 0.0;  // of the values; of the gradients, and its derivative
    if (q.rec) {
      const double* c = grec + 2 + 4 * rad;
      rg = ((c[3] * q.u + c[2]) * q.u + c[1]) * q.u + c[0];
      dr = ((3 * c[3] * q.u + 2 * c[2]) * q.u + c[1]) * q.rec[1];
      rf = rg;
      if (WPHI && last) {
        const double* v = q.rec + 2 + 4 * rad;
        rf = ((v[3] * q.u + v[2]) * q.u + v[1]) * q.u + v[0];
      }
    } else if (q.inner) {
      const double* e = radial + sp.ex_off + 4 * rad;
      rg = rf = ((e[0] * q.R + e[1]) * q.R + e[2]) * q.R + e[3];
      dr = (3 * e[0] * q.R + 2 * e[1]) * q.R + e[2];
    }
    const double w = q.R > 1.0e-13 ? -rg * q.ir : 0.0;  // no angular part there
    const double v = -dr - l * w;
#pragma unroll
    for (int m = 0; m < 2 * l + 1; ++m, ++ist) {
      if (WPHI) srow[ist] = rf * Y[m];
      if (WGRAD) {
        const double t = v * Y[m];
        sx[ist] = t * q.ux + w * G[m][0];
        sy[ist] = t * q.uy + w * G[m][1];
        sz[ist] = t * q.uz + w * G[m][2];
      }
    }
  }
}
template <bool WPHI, bool WGRAD>
__device__ __forceinline__ void eval_point(const DevSpecies& sp, const double* __restrict__ radial, const TabPoint& q,
                                           double* srow, double* sx, double* sy, double* sz) {
  int rad = 0, ist = 0;
  eval_l<0, WPHI, WGRAD>(sp, radial, q, rad, ist, srow, sx, sy, sz);
  if (sp.max_l >= 1) eval_l<1, WPHI, WGRAD>(sp, radial, q, rad, ist, srow, sx, sy, sz);
  if (sp.max_l >= 2) eval_l<2, WPHI, WGRAD>(sp, radial, q, rad, ist, srow, sx, sy, sz);
  if (sp.max_l >= 3) eval_l<3, WPHI, WGRAD>(sp, radial, q, rad, ist, srow, sx, sy, sz);
}

// Value tables: one thread per sphere point, kTabBlock points per block.
__global__ void __launch_bounds__(kTabBlock) tabulate_values_kernel(DevGeom g, const DevSpecies* __restrict__ spes,
                                                                     const double* __restrict__ radial,
                                                                     const int32_t* __restrict__ buckets,
                                                                     const int32_t* __restrict__ block_atom,
                                                                     const int64_t* __restrict__ block_start,
                                                                     double* phi) {
  extern __shared__ double stage[];
  const int atom = block_atom[blockIdx.x];
  const int64_t first = block_start[blockIdx.x];
  const int64_t s0 = g.sph_off[atom], s1 = g.sph_off[atom + 1];
  const int npts = (int)((s1 - first) < kTabBlock ? (s1 - first) : kTabBlock);
  const DevSpecies sp = spes[g.spe[atom]];
  const int NO = sp.no;
  const int t = threadIdx.x;
  if (t < npts) {
    double xyz[3];
    point_xyz(g, atom, first + t, xyz);
    const TabPoint q = locate(sp, radial, buckets, xyz);
    double* srow = stage + (size_t)t * NO;
    eval_point<true, false>(sp, radial, q, srow, nullptr, nullptr, nullptr);
  }
  __syncthreads();
  const int64_t base = g.phi_off[atom] + (first - s0) * NO;
  const int total = npts * NO;
  double* dst = phi + base;
  const int head = (int)(((uintptr_t)dst & 15) ? 1 : 0);
  if (t == 0 && head && total > 0) dst[0] = stage[0];
  const int nvec = (total - head) / 2;
  double2* dv = reinterpret_cast<double2*>(dst + head);
  for (int i = t; i < nvec; i += blockDim.x) dv[i] = make_double2(stage[head + 2 * i], stage[head + 2 * i + 1]);
  const int tail = head + 2 * nvec;
  if (t == 0 && tail < total) dst[tail] = stage[tail];
}

// Value and gradient tables: one thread per sphere point, kTabPoints per block.
__global__ void __launch_bounds__(kTabPoints) tabulate_gradients_kernel(DevGeom g, const DevSpecies* __restrict__ spes,
                                                                        const double* __restrict__ radial,
                                                                        const int32_t* __restrict__ buckets,
                                                                        const int32_t* __restrict__ block_atom,
                                                                        const int64_t* __restrict__ block_start,
                                                                        double* phi, double* dpx, double* dpy,
                                                                        double* dpz) {
  extern __shared__ double stage[];
  const int atom = block_atom[blockIdx.x];
  const int64_t first = block_start[blockIdx.x];
  const int64_t s0 = g.sph_off[atom], s1 = g.sph_off[atom + 1];
  const int npts = (int)((s1 - first) < kTabPoints ? (s1 - first) : kTabPoints);
  const DevSpecies sp = spes[g.spe[atom]];
  const int NO = sp.no;
  const int t = threadIdx.x;

  if (t < npts) {
    double xyz[3];
    point_xyz(g, atom, first + t, xyz);
    double* srow = stage + (size_t)t * NO;
    double* sx = stage + (size_t)kTabPoints * NO + (size_t)t * NO;
    double* sy = sx + (size_t)kTabPoints * NO;
    double* sz = sy + (size_t)kTabPoints * NO;
    const TabPoint q = locate(sp, radial, buckets, xyz);
    if (q.R < 1.0e-13) {
      // the gradient tables shift points that sit on the atom
      // (src/Matrix/Set_dOrbitals_Grid.jl:107-112); the values do not
      eval_point<true, false>(sp, radial, q, srow, sx, sy, sz);
      for (int d = 0; d < 3; ++d) xyz[d] += 1.0e-13;
      eval_point<false, true>(sp, radial, locate(sp, radial, buckets, xyz), srow, sx, sy, sz);
    } else {
      eval_point<true, true>(sp, radial, q, srow, sx, sy, sz);
    }
  }
  __syncthreads();

  // contiguous write-back: the block's points occupy rows [first-s0, +npts)
  const int64_t base = g.phi_off[atom] + (first - s0) * NO;
  const int total = npts * NO;
  double* outs[4] = {phi, dpx, dpy, dpz};
  for (int tab = 0; tab < 4; ++tab) {
    const double* src = stage + (size_t)tab * kTabPoints * NO;
    double* dst = outs[tab] + base;
    // 16-byte stores where the destination is 16-byte aligned
    const int head = (int)(((uintptr_t)dst & 15) ? 1 : 0);
    if (t == 0 && head && total > 0) dst[0] = src[0];
    const int nvec = (total - head) / 2;
    double2* dv = reinterpret_cast<double2*>(dst + head);
    for (int i = t; i < nvec; i += blockDim.x) dv[i] = make_double2(src[head + 2 * i], src[head + 2 * i + 1]);
    const int tail = head + 2 * nvec;
    if (t == 0 && tail < total) dst[tail] = src[tail];
  }
}

__global__ void f64_to_f32_kernel(const double* __restrict__ s, float* __restrict__ d, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    d[i] = (float)s[i];
}

}  // namespace

cudaError_t launch_tabulate(const DevGeom& g, const DevSpecies* dspe, const double* radial, const int32_t* buckets,
                            int64_t nblocks, const int32_t* block_atom, const int64_t* block_start, double* phi,
                            double* dphi_x, double* dphi_y, double* dphi_z, int max_no, cudaStream_t st) {
  if (nblocks == 0) return cudaSuccess;
  const bool grad = dphi_x != nullptr;
  if (!grad) {
    const size_t smem = (size_t)kTabBlock * max_no * sizeof(double);
    LCP_CUDA_TRY(raise_smem(tabulate_values_kernel, smem));
    tabulate_values_kernel<<<(unsigned)nblocks, kTabBlock, smem, st>>>(g, dspe, radial, buckets, block_atom,
                                                                        block_start, phi);
    return cudaGetLastError();
  }
  // the gradient kernel takes blocks of kTabPoints points
  const size_t smem = (size_t)kTabPoints * max_no * sizeof(double) * 4;
  LCP_CUDA_TRY(raise_smem(tabulate_gradients_kernel, smem));
  tabulate_gradients_kernel<<<(unsigned)nblocks, kTabPoints, smem, st>>>(g, dspe, radial, buckets, block_atom,
                                                                         block_start, phi, dphi_x, dphi_y, dphi_z);
  return cudaGetLastError();
}

// Per-interval cubic of the tables' spline for interval m of one
// radial function w (src/Matrix/Set_Orbitals_Grid.jl:187-238): the Hermite
// interpolant through (RV[m-1], f2) and (RV[m], f3) with the slopes g1, g2 of
// the reference, as coefficients of u = (R - RV[m-1]) / h2; at m = N-2 the
// reference's values (not its gradients) substitute f4 = f1 (:226-229).
static void interval_cubic(const double* rv, const double* w, int n, int m, bool values, double* c) {
  const double h1 = rv[m - 1] - rv[m - 2], h2 = rv[m] - rv[m - 1], h3 = rv[m + 1] - rv[m];
  const double f1 = w[m - 2], f2 = w[m - 1], f3 = w[m];
  const double f4 = values && m == n - 2 ? f1 : w[m + 1];
  double dum = h1 + h2;
  const double dum1 = h1 / h2 / dum, dum2 = h2 / h1 / dum;
  dum = h2 + h3;
  const double dum3 = h2 / h3 / dum, dum4 = h3 / h2 / dum;
  const double g1 = (f3 - f2) * dum1 + (f2 - f1) * dum2;
  const double g2 = (f4 - f3) * dum3 + (f3 - f2) * dum4;
  c[0] = f2;
  c[1] = h2 * g1;
  c[2] = 3 * (f3 - f2) - 2 * h2 * g1 - h2 * g2;
  c[3] = 2 * (f2 - f3) + h2 * g1 + h2 * g2;
}

// The polynomial continuation below RV[0] (src/Matrix/Set_Orbitals_Grid.jl:122-185):
// value and slope of the spline at rm = RV[4] (mesh point 4, 0-based), then
// a R^3 + b R^2 + c R + d by l.
static void inner_cubic(const double* rv, const double* w, int l, double* e) {
  const int m = 4;
  const double rm = rv[m];
  const double h1 = rv[m - 1] - rv[m - 2], h2 = rv[m] - rv[m - 1], h3 = rv[m + 1] - rv[m];
  const double y1 = (rm - rv[m - 1]) / h2, y2 = (rm - rv[m]) / h2;
  double dum = h1 + h2;
  const double dum1 = h1 / h2 / dum, dum2 = h2 / h1 / dum;
  dum = h2 + h3;
  const double dum3 = h2 / h3 / dum, dum4 = h3 / h2 / dum;
  const double f1 = w[m - 2], f2 = w[m - 1], f3 = w[m], f4 = w[m + 1];
  const double d32 = f3 - f2;
  const double g1 = d32 * dum1 + (f2 - f1) * dum2;
  const double g2 = (f4 - f3) * dum3 + d32 * dum4;
  const double A = 3 * f2 + h2 * g1, B = 2 * f2 + h2 * g1, C = 3 * f3 - h2 * g2, D = 2 * f3 - h2 * g2;
  const double E = A + B * y2, F = C - D * y1;
  const double y12 = y1 * y1, y22 = y2 * y2;
  const double f = y22 * E + y12 * F;
  const double df = (2 * y2 / h2) * E + y22 * B / h2 + (2 * y1 / h2) * F - y12 * D / h2;
  double a = 0, b = 0, c = 0, d = 0;
  if (l == 0) {
    b = 0.5 * df / rm;
    d = f - b * (rm * rm);
  } else if (l == 1) {
    a = (rm * df - f) / (2 * (rm * rm * rm));
    c = df - 3 * a * (rm * rm);
  } else {
    b = (3 * f - rm * df) / (rm * rm);
    a = (f - b * (rm * rm)) / (rm * rm * rm);
  }
  e[0] = a;
  e[1] = b;
  e[2] = c;
  e[3] = d;
}

void append_spline_tables(const double* rv, const double* rwf, int n, const int* num_basis, int max_l,
                          DevSpecies& d, std::vector<double>& radial, std::vector<int32_t>& buckets) {
  int nrad = 0;
  for (int l = 0; l <= max_l; ++l) nrad += num_basis[l];
  const int rec = 2 + 4 * nrad;
  d.iv_off = (int64_t)radial.size();
  radial.resize(radial.size() + (size_t)n * rec, 0.0);
  for (int k = 2; k <= n - 1; ++k) {  // the last record: interval n - 2 of the gradients
    const int m = std::min(k, n - 2);
    double* r = radial.data() + d.iv_off + (size_t)k * rec;
    r[0] = rv[m - 1];
    r[1] = 1.0 / (rv[m] - rv[m - 1]);
    for (int q = 0; q < nrad; ++q) interval_cubic(rv, rwf + (size_t)q * n, n, m, k == m, r + 2 + 4 * q);
  }
  d.ex_off = (int64_t)radial.size();
  radial.resize(radial.size() + (size_t)4 * nrad, 0.0);
  int q = 0;
  for (int l = 0; l <= max_l; ++l)
    for (int p = 0; p < num_basis[l]; ++p, ++q) inner_cubic(rv, rwf + (size_t)q * n, l, radial.data() + d.ex_off + 4 * q);
  // buckets of log2(R) over [log2 RV[1], log2 RV[n-1]]: each holds the first
  // mesh index >= 1 whose RV reaches the bucket's lower edge
  const double lo = std::log2(rv[1]), hi = std::log2(rv[n - 1]);
  const double inv = kSplineBuckets / std::max(hi - lo, 1e-30);
  d.bk_lo = (float)lo;
  d.bk_inv = (float)inv;
  d.bk_off = (int64_t)buckets.size();
  int i = 1;
  for (int b = 0; b < kSplineBuckets; ++b) {
    // the edge as the device computes bucket numbers (in float), lowered by
    // a bucket's width of margin through the device's b - 1
    const double edge = std::exp2((double)d.bk_lo + b / (double)d.bk_inv);
    while (i < n - 1 && rv[i] < edge) ++i;
    buckets.push_back(i);
  }
}

cudaError_t launch_convert_f32(const double* src, float* dst, int64_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 152 * 16);
  f64_to_f32_kernel<<<blocks, 256, 0, st>>>(src, dst, n);
  return cudaGetLastError();
}

}  // namespace lcp
