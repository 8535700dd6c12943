// elmm_kernels.cuh -- the sm_100a kernels of one RK3 stage of TMarchRK3
// (src/tsteps.f90:24-243), templated on the storage/arithmetic type T
// (double: plain FP64 path; float: mixed path, whose reductions, singular
// Poisson mode and divergence residual stay in FP64).
//
// Every kernel walks a flattened list of tiles that may span several domains
// (a batch); find_dom() maps a tile to its domain.  The grid is sized to the
// number of resident blocks and each block strides over the tiles.
//
// Per stage:
//   k_sgs       SubgridStresses: Smagorinsky viscosity (dynamics.f90:869-908);
//               beside it k_wm_points, the wall-model fluxes
//   k_momentum  Convection + OtherTerms: CDS2 advection, diffusion with the
//               wall-flux corrections, RK combine, old-pressure gradient,
//               U2 += U (dynamics.f90:230-499, tsteps.f90:263-358)
//   k_fftx_fwd_reg, _any   divergence RHS (pressure.f90:688-717) fused with
//               the real FFT along x (elmm_poisson_reg.cuh for the lengths
//               with a register FFT, elmm_poisson_any.cuh for the others)
//   k_wsum, k_zero_mode   the (0,0) mode, beside the transforms
//   k_ffty_reg, _any   complex FFT along y (forward, then inverse)
//   k_tri_tile, k_tri  tridiagonal solve in z per wavenumber pair (tiled, or
//               for tall columns and periodic z)
//   k_fftx_inv_reg, _any   inverse real FFT along x -> Phi
//   k_project   PostPoisson (pressure.f90:728-991): U = U2 - coef grad Phi,
//               Pr += Phi, top-layer partial sums for FixPressureToReference
//   k_ghosts    ghost shells of the fields written; after the projection
//               also the pressure reference (pressure.f90:1160-1220)
#pragma once

#include "elmm_common.cuh"
#include "elmm_fft.cuh"

namespace elmm {

constexpr int TX = 32, TY = 4;  // cell tile of the stencil kernels

struct Launch {
  const int *starts;  // per-domain first tile, nd + 1 entries (device)
  int nd;
  int total;          // total tiles
  int kc;             // planes of a tile's column (kernels that march up a chunk of planes)
};

template <typename T>
__device__ __forceinline__ T ld(const T *p, long long o) { return __ldg(p + o); }

// gfortran's NORM2: scaled sum of squares
__device__ __forceinline__ double norm2_3(const double *x) {
  double scale = 0, ssq = 1;
#pragma unroll
  for (int m = 0; m < 3; m++) {
    if (x[m] != 0) {
      double ax = fabs(x[m]);
      if (scale < ax) { double r = scale / ax; ssq = 1 + ssq * (r * r); scale = ax; }
      else { double r = ax / scale; ssq = ssq + r * r; }
    }
  }
  return scale * sqrt(ssq);
}

// WMFlatUstar / WMRoughUstar, src/wallmodels.f90:1190-1335
__device__ inline double wm_flat_ustar(double ustar, double vel, double dist, double nu) {
  if (nu <= 0) return 0;
  double ustar_lam = sqrt(nu * vel / dist);
  if ((dist * ustar_lam / nu) < 5.0) return ustar_lam;
  for (int i = 1;; i++) {  // at most 50 iterations (wallmodels.f90:1230)
    double ustar2 = ustar;
    double z_pl = dist * ustar2 / nu;
    if (z_pl <= 5.0) ustar = sqrt(nu * vel / dist);
    else if (z_pl < 30.0) ustar = vel / (5 * log(z_pl) - (double)3.05f);
    else ustar = vel / (log(z_pl) / 0.4 + 5.5);
    if (fabs(ustar - ustar2) / fabs(ustar) < 1e-4) return ustar;
    if (i >= 50) return 0;
  }
}

__device__ inline double wm_rough_ustar(double ustar, double vel, double dist, double z0, double nu) {
  if (nu > 0) {
    ustar = sqrt(nu * vel / dist);
    if (dist * ustar / nu < 11.225 * 1.1) return ustar;
  }
  if (dist <= z0 * 2) return nu > 0 ? wm_flat_ustar(ustar, vel, dist, nu) : 0.0;
  return vel * 0.41 / log(dist / z0);
}

// the u* of a wall point: WMRoughStress with a roughness length, else
// WMFlatStress (src/wallmodels.f90:2262-2275, 1243-1265); ustar is the
// point's value from the stage before (the start of the flat iteration)
__device__ inline double wm_ustar(double ustar, double vel, double dist, double z0, double nu) {
  return z0 > 0 ? wm_rough_ustar(ustar, vel, dist, z0, nu) : wm_flat_ustar(ustar, vel, dist, nu);
}

// PsiM_MO, the Businger-Dyer stability function of momentum
// (src/wallmodels.f90:1546-1556)
__device__ inline double psim_mo(double zeta) {
  if (zeta < 0) {
    const double x = pow(1 - 15.0 * zeta, 0.25), h = (1 + x) / 2.0;
    return log(((1 + x * x) / 2.0) * (h * h)) - 2.0 * atan(x) + 3.141592653589793 / 2;
  }
  return -4.8 * zeta;
}

// WM_MO_Flux_ustar (src/wallmodels.f90:1606-1660): u* of a rough wall under
// a prescribed surface temperature flux, the log law corrected by PsiM_MO at
// the Obukhov stability z/L, both relaxed by halves from the point's u* of
// the stage before.  The tolerances 1e-3, 1e-4 and 1e-5 are default-real
// literals in the reference (their float values widened).
__device__ inline double wm_mo_flux_ustar(double ustar, double vel, double dist, double z0, double tflux,
                                          double tref, double g, double nu) {
  if (dist <= z0) {
    if (nu <= 0) return 0;
    if ((dist * ustar / nu) < 11.225) return sqrt(nu * vel / dist);
    return vel / (log(fabs(ustar * dist / nu)) / 0.4 + 5.2);
  }
  double zL = 0, Psi = 0;
  for (int i = 1;; i++) {  // at most 50 iterations
    const double ustar2 = ustar;
    ustar = ustar + (fmax(vel * 0.4 / log(fmax((dist / z0) - Psi, (double)1e-5f)), 0.0) - ustar) / 2;
    if (ustar < (double)1e-4f) {
      zL = -10000;
    } else {  // Obukhov_zL (src/wallmodels.f90:1598-1602)
      const double zL2 = dist * (0.4 * (g / tref) * tflux) / (-(ustar * ustar * ustar));
      zL = zL + (zL2 - zL) / 2;
    }
    Psi = psim_mo(zL);
    if (fabs(ustar - ustar2) / fmax(fabs(ustar), 1e-3) < (double)1e-3f) return ustar;
    if (i >= 50) return 0;
  }
}

// PsiM_MO_mod / PsiH_MO_mod, the stability functions of Zilitinkevich and
// Esau (2006) with L defined with the von Karman constant k_U
// (src/wallmodels.f90:1572-1595)
__device__ inline double psim_mo_mod(double zeta, double kU) {
  if (zeta < 0) {
    const double x = pow(1 - 6.0 * zeta * kU, 0.25), h = (1 + x) / 2.0;
    return log(((1 + x * x) / 2.0) * (h * h)) - 2.0 * atan(x) + 3.141592653589793 / 2;
  }
  return -(3 * pow(zeta * kU, 5.0 / 6.0));
}
__device__ inline double psih_mo_mod(double zeta, double kU) {
  if (zeta < 0) {
    const double x = pow(1 - 6.0 * zeta * kU, 0.25);
    return 2.0 * log((1 + x * x) / 2.0);
  }
  return -(2.5 * pow(zeta * kU, 4.0 / 5.0));
}

// WM_MO_Dirichlet_ustar_tfl (src/wallmodels.f90:1664-1716): u* and the
// surface temperature flux of a rough wall with a prescribed surface
// temperature, tempdif = theta(point) - theta(surface).  tflux comes in as
// the point's flux of the stage before (the start of the stability
// iteration, relaxed until z/L changes by less than 1e-3); its 1.1 is a
// default-real literal in the reference.
template <typename T>
__device__ inline void wm_mo_dirichlet(const Dom<T> &d, double &ustar, double &tflux, double dist, double z0,
                                       double vel, double tempdif) {
  const double kU = 0.4, kT = 0.47, nu = d.nu_mol;
  ustar = wm_rough_ustar(ustar, vel, dist, z0, nu);
  double dist_plus = 1.7976931348623157e308;  // huge()
  if (nu > 0) dist_plus = dist * sqrt(nu * vel / dist) / nu;
  if (dist <= z0 || dist_plus < (double)1.1f * 11.225) {
    tflux = -d.kappa_mol * tempdif / dist;
    return;
  }
  double zL = 0, zL0 = -10000.0;
  int i = 0;
  for (;;) {
    i++;
    zL = -dist * d.grav * tflux / (kU * d.tref * (ustar * ustar * ustar));
    const double pm = psim_mo_mod(zL, kU), ph = psih_mo_mod(zL, kU);
    ustar = vel * kU / (log(dist / z0) - pm);
    tflux = -tempdif * ustar * kT / (log(dist / z0) - ph);  // z0H = z0
    if (i > 1 && fabs(zL - zL0) / fmax(fabs(zL), 1e-4) < 1e-3) break;
    if (i >= 50 || zL > 10000) break;
    zL0 = zL;
  }
  if (i >= 50 || zL > 10000) {
    ustar = sqrt(nu * vel / dist);
    tflux = -d.kappa_mol * tempdif / dist;
  }
}

// ComputeViscsWM for the Pr point next to side f (bottom or top) at cell
// (i, j, k) with a prescribed surface temperature (WM_MO_Dirichlet,
// src/wallmodels.f90:1858-1884, 2080-2111): the point's u* and surface
// temperature flux from the cell-centred velocity and theta at the start of
// the stage (Tm); the viscosity it forms is overwritten by SubgridModel in
// the reference and is not kept.
template <typename T>
__device__ void wm_pr_dirichlet(const Dom<T> &d, int f, int i, int j, int k, const T *Tm) {
  if (!(d.z0[f] > 0)) return;  // smooth wall: the flat branch leaves u* and the flux of a Pr point alone
  const long long c = bidx(d, i, j, k);
  double ou = 0, ov = 0;
  if constexpr (sizeof(T) == 4) { ou = (double)vel_off(d, 0, k); ov = (double)vel_off(d, 1, k); }
  const double uv[3] = {(((double)ld(d.U, c) + ou) + ((double)ld(d.U, c - 1) + ou)) / 2.0,
                        (((double)ld(d.V, c) + ov) + ((double)ld(d.V, c - d.pitch) + ov)) / 2.0,
                        ((double)ld(d.W, c) + (double)ld(d.W, c - d.plane)) / 2.0};
  const double distz = f == SIDE_BO ? d.zW[0 + 2] - d.zPr[1 + 2] : d.zW[d.ext[2][2] + 1 + 2] - d.zPr[d.nz + 2];
  const double dv[3] = {0.0, 0.0, distz};
  const double dist = sqrt((dv[0] * dv[0] + dv[1] * dv[1]) + dv[2] * dv[2]);
  const double dot = (uv[0] * dv[0] + uv[1] * dv[1]) + uv[2] * dv[2];
  double vect[3];
#pragma unroll
  for (int m = 0; m < 3; m++) vect[m] = uv[m] - dot * dv[m] / (dist * dist);
  const double vel = sqrt((vect[0] * vect[0] + vect[1] * vect[1]) + vect[2] * vect[2]);
  const double tdif = ((double)ld(Tm, c) + d.toff) - d.tsurf[f];
  const int h = f == SIDE_BO ? 0 : 1;
  const long long q = (long long)(i - 1) + (long long)d.nx * (j - 1);
  double ustar = d.wm_pr_us[h][q], tfl = d.wm_pr_tf[h][q];
  wm_mo_dirichlet(d, ustar, tfl, dist, d.z0[f], vel, tdif);
  if (ustar < 0) ustar = 0;
  d.wm_pr_us[h][q] = ustar;
  d.wm_pr_tf[h][q] = tfl;
}

// ComputeUVWFluxesWM / fluxes for the point of component comp next to side f
// (bottom or top: x and y are periodic for every domain) at column (i, j),
// point pidx of the face (src/wallmodels.f90:2159-2338); the wall-point
// distance is the one of GetOutsideBoundariesWM_UVW (src/wallmodels.f90:690-909).
template <typename T>
__device__ void wm_point(const Dom<T> &d, int comp, int f, int i, int j, int pidx, const T *Tm) {
  const bool hi = f & 1;
  const int k = hi ? d.ext[comp][2] : 1;
  const T *U = d.U, *V = d.V, *W = d.W;
  const long long c = bidx(d, i, j, k), sx = 1, sy = d.pitch, sz = d.plane;
  const int face = comp * 6 + f;
  double ustar = d.wm_ustar[face][pidx];
  // full velocities: stored values plus the per-level offsets of U and V of
  // the mixed path (the FP64 path reads the stored values alone), in FP64
  const double ou0 = (double)vel_off(d, 0, k), ov0 = (double)vel_off(d, 1, k);
  auto lu = [&](long long o, double off) {
    if constexpr (sizeof(T) == 4) return (double)ld(U, c + o) + off;
    else return (double)ld(U, c + o);
  };
  auto lv = [&](long long o, double off) {
    if constexpr (sizeof(T) == 4) return (double)ld(V, c + o) + off;
    else return (double)ld(V, c + o);
  };
  double vel[3];
  if (comp == 0) {
    vel[0] = lu(0, ou0);
    vel[1] = (lv(sx, ov0) + lv(0, ov0) + lv(sx - sy, ov0) + lv(-sy, ov0)) / 4.0;
    vel[2] = ((double)ld(W, c + sx) + (double)ld(W, c) + (double)ld(W, c + sx - sz) + (double)ld(W, c - sz)) / 4.0;
  } else if (comp == 1) {
    vel[0] = (lu(sy, ou0) + lu(0, ou0) + lu(-sx + sy, ou0) + lu(-sx, ou0)) / 4.0;
    vel[1] = lv(0, ov0);
    vel[2] = ((double)ld(W, c + sy) + (double)ld(W, c) + (double)ld(W, c + sy - sz) + (double)ld(W, c - sz)) / 4.0;
  } else {
    const double ou1 = (double)vel_off(d, 0, k + 1), ov1 = (double)vel_off(d, 1, k + 1);
    vel[0] = (lu(sz, ou1) + lu(0, ou0) + lu(-sx + sz, ou1) + lu(-sx, ou0)) / 4.0;
    vel[1] = (lv(sz, ov1) + lv(0, ov0) + lv(-sy + sz, ov1) + lv(-sy, ov0)) / 4.0;
    vel[2] = (double)ld(W, c);
  }
  // distance to the wall with the staggered coordinate of the component; the
  // velocity along it (wall velocity 0) taken off
  const double distz = d.zW[hi ? d.ext[2][2] + 1 + 2 : 0 + 2] - (comp == 2 ? d.zW[k + 2] : d.zPr[k + 2]);
  const double dd = fabs(distz);
  const double t[3] = {vel[0], vel[1], vel[2] - vel[2] * distz * distz / (dd * dd)};
  const double tv = sqrt((t[0] * t[0] + t[1] * t[1]) + t[2] * t[2]);
  if (d.z0[f] > 0 && d.tdir[f]) {  // WM_MO_DirichletStress (src/wallmodels.f90:1922-1938, 2228-2253)
    // local_value of theta at the point (src/wallmodels.f90:2340-2353), x and y periodic
    const int i2 = comp == 0 ? (i + 1 > d.nx ? 1 : i + 1) : i, j2 = comp == 1 ? (j + 1 > d.ny ? 1 : j + 1) : j;
    const double temp = (((double)ld(Tm, bidx(d, i2, j2, comp == 2 ? k + 1 : k)) + d.toff) +
                         ((double)ld(Tm, bidx(d, i, j, k)) + d.toff)) / 2;
    double tfl = d.wm_tfl[face][pidx];
    wm_mo_dirichlet(d, ustar, tfl, dd, d.z0[f], tv, temp - d.tsurf[f]);
    d.wm_tfl[face][pidx] = tfl;
  } else if (d.z0[f] > 0 && d.tflux[f] > 0)  // WM_MO_FluxStress (src/wallmodels.f90:1836-1854, 2255-2259)
    ustar = tv != 0 ? wm_mo_flux_ustar(ustar, tv, dd, d.z0[f], d.tflux[f], d.tref, d.grav, d.nu_mol) : 0.0;
  else if (tv != 0)
    ustar = wm_ustar(ustar, tv, dd, d.z0[f], d.nu_mol);
  if (ustar < 0) ustar = 0;
  d.wm_ustar[face][pidx] = ustar;
  double fp = 0, fm = 0;
  if (tv > 1.4901161193847656e-08) {
    fp = (t[comp] / tv) * (ustar * ustar);
    if (d.vz) {
      // U and V: the heights of the cells either side of the face, W: of the levels
      const double *h = comp < 2 ? d.dzPr : d.dzW;
      const int kp = f == SIDE_BO ? k : k + 1;
      fm = fp / h[kp - 1 + 2];
      fp = fp / h[kp + 2];
    } else {
      fp = fp * (1 / d.dz);
      fm = fp;
    }
    if (!hi) { fp = -fp; fm = -fm; }  // MINUSX/Y/Z directions are odd
  }
  d.wm_fluxp[face][pidx] = (T)fp;
  d.wm_fluxm[face][pidx] = (T)fm;
}

// SubgridStresses' wall model (src/dynamics.f90:879-888): ComputeViscsWM
// for the Pr points with a prescribed surface temperature, and
// ComputeUVWFluxesWM for every velocity point on a wall-model face, from the
// state at the start of the stage (tb: its temperature buffer).  One thread
// a point, in faces of nx ny points (i + nx j): the Pr points of the bottom
// and top, then per component the bottom and the top.  The parts touch
// disjoint state.  Launched beside k_sgs (whose viscosity they do not read)
// and, with the initial fields, at the end of the initial projection.  On a
// small grid k_momentum waits for it: a thread's time is its chain of
// descriptor loads, integer divisions and FP64 divisions, roots and
// logarithms, so the face comes from one 32-bit division and the norm of the
// tangential velocity is formed once, without scaling (128 x 128 x 64 with a
// scalar: a step of 0.482 -> 0.469 ms).
constexpr int kWmThreads = 128;
template <typename T>
__host__ __device__ inline long long wm_points_of(const Dom<T> &d) {
  const int faces = (d.tdir[SIDE_BO] != 0) + (d.tdir[SIDE_TO] != 0) + 3 * ((d.wall[SIDE_BO] != 0) + (d.wall[SIDE_TO] != 0));
  return (long long)faces * d.nx * d.ny;
}
template <typename T>
__global__ void __launch_bounds__(kWmThreads) k_wm_points(const Dom<T> *__restrict__ doms, Launch L, int tb) {
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    const int nx = d.nx, np = nx * d.ny;
    const int pr_bo = d.tdir[SIDE_BO] != 0, pr_to = d.tdir[SIDE_TO] != 0;
    const int bo = d.wall[SIDE_BO] != 0, to = d.wall[SIDE_TO] != 0;
    const int p = (t - __ldg(L.starts + di)) * kWmThreads + threadIdx.x;
    int face = p / np;
    const int q = p - face * np, j = q / nx + 1, i = q - (j - 1) * nx + 1;
    const T *Tm = d.buoy ? d.slot[0].buf[tb] : nullptr;
    if (face < pr_bo + pr_to) {
      const int f = pr_bo && face == 0 ? SIDE_BO : SIDE_TO;
      wm_pr_dirichlet(d, f, i, j, f == SIDE_BO ? 1 : d.nz, Tm);
      continue;
    }
    face -= pr_bo + pr_to;
    const int per = bo + to;
    if (face >= 3 * per) continue;
    const int comp = per == 2 ? face >> 1 : face;
    wm_point(d, comp, bo && (per == 1 || !(face & 1)) ? SIDE_BO : SIDE_TO, i, j, q, Tm);
  }
}

}  // namespace elmm

#include "elmm_momentum.cuh"

namespace elmm {

// ------------------------------------------------------------- Poisson
// The (0,0) mode of the Poisson problem (src/poisson.f90:23-60) from FP64 sums
// of W2 over each level.  The mean divergence of a level, whose x and y parts
// telescope to nothing, is the difference of two of these sums, so the flux
// of the mode through a level's top is the sum itself (less the bottom's) and
// its solution one prefix sum, its mean pinned to zero.  Taken from the FP32
// transform instead, the mode's rounding, independent from level to level, is
// integrated twice: a large and, as one mode's, a very uneven part of the
// error of the mixed pressure (64 x 64 x 32 after 40 steps: 3.2e-4 of the
// pressure, 1.4e-4 with the sums); and the serial sum was the longest chain
// of the z solve on small grids.
//
// The sums come from the forward x transform, which has W2 in registers
// (Dom::wrows: large domains), or from k_wsum beside it.  Both add them in an
// order that depends on nx and ny alone, so that a level has one sum wherever
// a domain is cut into slabs.

// zsol[1..nz] from the level sums (level(k), k = 0..nz, with the boundary
// conditions applied); c: norm / coef; every thread of the block calls it.
// One block size for every caller, so that a domain, alone or in slabs, has
// one result.
constexpr int kZeroThreads = 512;
template <typename F>
__device__ __forceinline__ void zero_mode_solve(int nz, int zper, const double *__restrict__ dzf, double c, F &&level,
                                                double *zsol, double *red) {
  constexpr int NT = kZeroThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // x(k + 1) = x(k) + (F(k) + F0) dzf(k) with F(k) = (level(k) - level(0)) norm / coef
  const double l0 = level(0);
  auto block_sum = [&](double v, double &before) -> double {  // the block's sum, and the sum of the threads before
    double x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) red[warp] = x;
    __syncthreads();
    double tot = 0, pre = 0;
    for (int w = 0; w < NT / 32; w++) {
      if (w < warp) pre += red[w];
      tot += red[w];
    }
    before = pre + (x - v);
    return tot;
  };
  const int per = (nz + NT - 1) / NT, k0 = 1 + threadIdx.x * per, k1 = min(nz, k0 + per - 1);
  double F0 = 0, before;
  if (zper) {  // so that x is periodic: sum_k dzf(k) (F(k) + F0) = 0
    double a = 0, b = 0;
    for (int q = k0; q <= k1; q++) { a += (level(q) - l0) * c * dzf[q]; b += dzf[q]; }
    const double sa = block_sum(a, before), sb = block_sum(b, before);
    F0 = -sa / sb;
  }
  double g = 0;  // the increments of this thread's levels
  for (int q = k0; q <= k1; q++) g += ((level(q) - l0) * c + F0) * dzf[q];
  block_sum(g, before);
  double x = before, sx = 0;
  for (int q = k0; q <= k1; q++) { sx += x; x += ((level(q) - l0) * c + F0) * dzf[q]; }
  double unused;
  const double mean = block_sum(sx, unused) / nz;
  x = before;
  for (int q = k0; q <= k1; q++) { zsol[q] = x - mean; x += ((level(q) - l0) * c + F0) * dzf[q]; }
  __syncthreads();
}

// the level sums from the forward x transform's np tiles a level, a thread a level
__device__ __forceinline__ void sum_tiles(const double *part, int np, int nz, double *wsum) {
  for (int k = 1 + threadIdx.x; k <= nz; k += kZeroThreads) {
    double s = 0;
#pragma unroll 4
    for (int q = 0; q < np; q++) s += __ldcg(part + (long long)(k - 1) * np + q);
    wsum[k] = s;
  }
  __syncthreads();
}
template <typename T>
__device__ __forceinline__ void zero_mode(const Dom<T> &d, double coef, double *red) {
  auto level = [&](int g) {
    const Fold f = fold_vel(g, d.ext[2][2], d.bt[4], d.bt[5], true);
    return f.zero ? 0.0 : f.sign * __ldcg(d.wsum + f.src);
  };
  zero_mode_solve(d.nz, d.zper, d.dzf, 1.0 / coef * (1.0 / ((double)d.nx * (double)d.ny)), level, d.zsol, red);
}

// the domains whose level sums the forward x transform left per tile: a block
// a domain
// domains whose W2 is larger leave their sums per tile (init_domain), if a
// level's rows fill whole tiles or, in the generic transform, whose tiles of 2
// to 64 rows then start anew at each level, leave at most ny / kTileSumPad rows
// empty: a step with k_wsum and with such tiles, FP32, 300 x 270 x 50 (1 in 270)
// 0.901 and 0.875 ms, 135 x 135 x 75 with the temperature (1 in 15) 0.6395 and 0.6343.  The
// register transforms' tiles of 32 and more rows gain nothing so (256 x 240 x 100, 1 in 15,
// 1.037 and 1.038; 400 x 300 x 60 1.256 and 1.250), and the small domains' pay 0.4 us a stage.
constexpr long long kTileSumBytes = 5 << 20;
constexpr int kTileSumPad = 14;
template <typename T>
__global__ void __launch_bounds__(kZeroThreads) k_zero_mode(const Dom<T> *__restrict__ doms, int nd, double coef_alpha2,
                                                            int use_dt) {
  __shared__ double red[kZeroThreads / 32];
  for (int di = blockIdx.x; di < nd; di += gridDim.x) {
    const Dom<T> &d = doms[di];
    if (!d.wrows) continue;
    sum_tiles(d.wpart, d.wtiles(), d.nz, d.wsum);
    zero_mode(d, use_dt ? coef_alpha2 * d.dt : coef_alpha2, red);
  }
}

// Sums of W2 over each level, one block a level in a fixed order, wide blocks
// with kVec vectors in flight per thread; the last block of a domain (of no
// slab) solves.
constexpr int kWsumThreads = kZeroThreads;
template <typename T>
__global__ void __launch_bounds__(kWsumThreads, 2) k_wsum(const Dom<T> *__restrict__ doms, Launch L, double coef_alpha2,
                                                       int use_dt) {
  __shared__ double red[kWsumThreads / 32];
  __shared__ int last;
  constexpr int kVec = 8, VE = 16 / (int)sizeof(T);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    const int k = t - __ldg(L.starts + di) + 1;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    if (k <= d.ext[2][2]) {
      const long long pitch = d.pitch;
      const T *W = d.W2 + bidx(d, 1, 1, k);
      double s = 0;
      const int nv = (nx + VE - 1) / VE, n = nv * ny;  // 16-byte vectors of the level, a row's last one into its padding
      for (int q0 = threadIdx.x; q0 < n; q0 += kWsumThreads * kVec) {
        float4 v[kVec];
        int left[kVec];  // values of the row from the vector's first on
#pragma unroll
        for (int u = 0; u < kVec; u++) {
          const int q = q0 + u * kWsumThreads, j = q / nv, c = q - j * nv;
          left[u] = q < n ? nx - c * VE : 0;
          v[u] = q < n ? __ldg(reinterpret_cast<const float4 *>(W + j * pitch) + c) : make_float4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < kVec; u++) {
          const T *e = reinterpret_cast<const T *>(&v[u]);
#pragma unroll
          for (int c = 0; c < VE; c++) s += c < left[u] ? (double)e[c] : 0.0;
        }
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) red[warp] = s;
      __syncthreads();
      if (threadIdx.x == 0) {
        double tot = 0;
        for (int w = 0; w < kWsumThreads / 32; w++) tot += red[w];
        d.wsum[k] = tot;
      }
    }
    if (threadIdx.x == 0) {
      __threadfence();
      last = atomicAdd(d.wticket, 1) == nz - 1;  // nz tiles
      if (last) *d.wticket = 0;
    }
    __syncthreads();
    if (last && d.zsol) {
      __threadfence();
      zero_mode(d, use_dt ? coef_alpha2 * d.dt : coef_alpha2, red);
    }
    __syncthreads();
  }
}

// Tridiagonal solve in z for each (kx, ky): the Thomas algorithm in FP64 on
// the rows of Residue_variable_z (poisson.f90:23-60), Neumann rows at the
// ends or a cyclic system for periodic z; the (0,0) mode is singular: its
// solution is given (zsol), or, for a right-hand side that is not a divergence, it
// is solved by two prefix sums with its mean pinned to zero.
constexpr int kTriThreads = 64;

template <typename T>
__global__ void __launch_bounds__(kTriThreads) k_tri(const Dom<T> *__restrict__ doms, Launch L, int gate, int zsol) {
  typedef typename Vec2<T>::type T2;
  extern __shared__ double cps[];  // [nz][kTriThreads]
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    if (gate && !*d.refine_flag) continue;  // defect-correction sweep not needed
    const int lt = t - __ldg(L.starts + di);
    const int col = lt * kTriThreads + threadIdx.x;
    const int ky = col / d.spitch, kx = col - ky * d.spitch;
    if (ky >= d.ny || kx >= d.nxh) continue;
    const int nz = d.nz;
    const long long ps = (long long)d.ny * d.spitch;
    T2 *S = d.S + (long long)ky * d.spitch + kx;
    const double norm = 1.0 / ((double)d.nx * (double)d.ny);
    const double lam = d.lamx[kx] + d.lamy[ky];
    const double *Ab = d.Ab, *At = d.At;
    if (kx == 0 && ky == 0) {
      if (zsol) {  // solved beside the transforms
#pragma unroll 4
        for (int k = 1; k <= nz; k++) {
          T2 o; o.x = (T)d.zsol[k]; o.y = (T)0;
          S[(long long)(k - 1) * ps] = o;
        }
        continue;
      }
      // singular mode: F(k) = F(k-1) + dzc(k) r(k) is the flux (x(k+1)-x(k))/dzf(k);
      // the right-hand sides are fetched kPre at a time, so that their loads
      // are in flight together
      constexpr int kPre = 8;
      auto rhs = [&](int kb2, int ke2, double (&rx)[kPre], double (&ry)[kPre]) {
#pragma unroll
        for (int q = 0; q < kPre; q++) {
          rx[q] = ry[q] = 0;
          if (kb2 + q <= ke2) {
            const T2 r = S[(long long)(kb2 + q - 1) * ps];
            rx[q] = ((double)r.x * norm) * d.dzc[kb2 + q];
            ry[q] = ((double)r.y * norm) * d.dzc[kb2 + q];
          }
        }
      };
      double F0x = 0, F0y = 0;
      if (d.zper) {  // choose F(0) so that x is periodic: sum_k dzf(k) F(k) = 0
        double Fx = 0, Fy = 0, swx = 0, swy = 0, sd = 0;
        for (int kb2 = 1; kb2 <= nz; kb2 += kPre) {
          double rx[kPre], ry[kPre];
          rhs(kb2, nz, rx, ry);
#pragma unroll
          for (int q = 0; q < kPre; q++) {
            const int k = kb2 + q;
            if (k > nz) break;
            Fx = Fx + rx[q];
            Fy = Fy + ry[q];
            swx += Fx * d.dzf[k]; swy += Fy * d.dzf[k]; sd += d.dzf[k];
          }
        }
        F0x = -swx / sd; F0y = -swy / sd;
      }
      double Fx = 0, Fy = 0, xx = 0, xy = 0, sx = 0, sy = 0;
      for (int kb2 = 1; kb2 <= nz - 1; kb2 += kPre) {
        double rx[kPre], ry[kPre];
        rhs(kb2, nz - 1, rx, ry);
#pragma unroll
        for (int q = 0; q < kPre; q++) {
          const int k = kb2 + q;
          if (k > nz - 1) break;
          Fx = Fx + rx[q];
          Fy = Fy + ry[q];
          T2 o; o.x = (T)xx; o.y = (T)xy;
          S[(long long)(k - 1) * ps] = o;  // x(k)
          sx += xx; sy += xy;
          xx = xx + (Fx + F0x) * d.dzf[k];
          xy = xy + (Fy + F0y) * d.dzf[k];
        }
      }
      sx += xx; sy += xy;
      sx = sx / nz; sy = sy / nz;
      T2 last; last.x = (T)(xx - sx); last.y = (T)(xy - sy);
      for (int k = 0; k < nz - 1; k++) {
        T2 v = S[(long long)k * ps];
        v.x = (T)((double)v.x - sx);
        v.y = (T)((double)v.y - sy);
        S[(long long)k * ps] = v;
      }
      S[(long long)(nz - 1) * ps] = last;
      continue;
    }
    double *cp = cps + threadIdx.x;
    if (!d.zper) {
      // Thomas algorithm; rows are fetched kPre at a time so that the loads of
      // a batch are in flight together (the recurrence only needs the values)
      constexpr int kPre = 8;
      double px = 0, py = 0, cprev = 0;
      for (int kb = 1; kb <= nz; kb += kPre) {
        T2 rr[kPre];
#pragma unroll
        for (int q = 0; q < kPre; q++)
          if (kb + q <= nz) rr[q] = S[(long long)(kb + q - 1) * ps];
#pragma unroll
        for (int q = 0; q < kPre; q++) {
          const int k = kb + q;
          if (k > nz) break;
          double den = (-(Ab[k] + At[k]) + lam) - (k > 1 ? Ab[k] * cprev : 0.0);
          double iv = 1.0 / den;
          cprev = At[k] * iv;
          cp[(k - 1) * kTriThreads] = cprev;
          if (k == 1) {
            px = (double)rr[q].x * norm * iv;
            py = (double)rr[q].y * norm * iv;
          } else {
            px = ((double)rr[q].x * norm - Ab[k] * px) * iv;
            py = ((double)rr[q].y * norm - Ab[k] * py) * iv;
          }
          T2 ok; ok.x = (T)px; ok.y = (T)py;
          S[(long long)(k - 1) * ps] = ok;
        }
      }
      // back substitution (px, py hold x(nz))
      for (int kt = nz - 1; kt >= 1; kt -= kPre) {
        T2 rr[kPre];
#pragma unroll
        for (int q = 0; q < kPre; q++)
          if (kt - q >= 1) rr[q] = S[(long long)(kt - q - 1) * ps];
#pragma unroll
        for (int q = 0; q < kPre; q++) {
          const int k = kt - q;
          if (k < 1) break;
          const double c = cp[(k - 1) * kTriThreads];
          px = (double)rr[q].x - c * px;
          py = (double)rr[q].y - c * py;
          T2 ok; ok.x = (T)px; ok.y = (T)py;
          S[(long long)(k - 1) * ps] = ok;
        }
      }
    } else {
      // cyclic system (periodic z) by Sherman-Morrison; c2 and z in shared memory
      double *zz = cps + (long long)nz * kTriThreads + threadIdx.x;
      const double alpha = At[nz], beta = Ab[1];
      const double b0 = -(Ab[1] + At[1]) + lam;
      const double gamma = -b0;
      double bb = b0 - gamma;
      double inv = 1.0 / bb;
      cp[0] = At[1] * inv;
      T2 r = S[0];
      double yx = (double)r.x * norm * inv, yy = (double)r.y * norm * inv;
      double z_ = gamma * inv;
      zz[0] = z_;
      T2 o; o.x = (T)yx; o.y = (T)yy;
      S[0] = o;
      for (int k = 2; k <= nz; k++) {
        double bk = -(Ab[k] + At[k]) + lam;
        if (k == nz) bk = bk - alpha * beta / gamma;
        double den = bk - Ab[k] * cp[(k - 2) * kTriThreads];
        double iv = 1.0 / den;
        cp[(k - 1) * kTriThreads] = At[k] * iv;
        T2 rk = S[(long long)(k - 1) * ps];
        yx = ((double)rk.x * norm - Ab[k] * yx) * iv;
        yy = ((double)rk.y * norm - Ab[k] * yy) * iv;
        double uk = (k == nz) ? alpha : 0.0;
        z_ = (uk - Ab[k] * z_) * iv;
        zz[(k - 1) * kTriThreads] = z_;
        T2 ok; ok.x = (T)yx; ok.y = (T)yy;
        S[(long long)(k - 1) * ps] = ok;
      }
      for (int k = nz - 1; k >= 1; k--) {
        T2 dk = S[(long long)(k - 1) * ps];
        yx = (double)dk.x - cp[(k - 1) * kTriThreads] * yx;
        yy = (double)dk.y - cp[(k - 1) * kTriThreads] * yy;
        z_ = zz[(k - 1) * kTriThreads] - cp[(k - 1) * kTriThreads] * z_;
        zz[(k - 1) * kTriThreads] = z_;
        T2 ok; ok.x = (T)yx; ok.y = (T)yy;
        S[(long long)(k - 1) * ps] = ok;
      }
      // now S holds y, zz holds z; x = y - fac z
      T2 y0 = S[0], yn = S[(long long)(nz - 1) * ps];
      double z0 = zz[0], zn = zz[(nz - 1) * kTriThreads];
      double den = 1.0 + z0 + beta * zn / gamma;
      double fx = ((double)y0.x + beta * (double)yn.x / gamma) / den;
      double fy = ((double)y0.y + beta * (double)yn.y / gamma) / den;
      for (int k = 0; k < nz; k++) {
        T2 v = S[(long long)k * ps];
        double zk = zz[k * kTriThreads];
        v.x = (T)((double)v.x - fx * zk);
        v.y = (T)((double)v.y - fy * zk);
        S[(long long)k * ps] = v;
      }
    }
  }
}

}  // namespace elmm
