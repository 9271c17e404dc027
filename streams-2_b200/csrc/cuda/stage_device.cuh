// Stage kernels of the B200 backend (FP64 and mixed forms).
//
// One Runge-Kutta stage (rk_sync, code/src/singleideal/singleideal_cpu.F90:332-409) runs as:
//   k_apply_shift  the pending force_var energy shift of the previous stage, on interior w
//   k_aux      w -> primitive/thermo fields at interior and face-ghost points; ghost values are
//              produced on the fly (periodic wrap, staggered isothermal wall mirror)
//   k_xflux    x-face hybrid fluxes + divergence (fl = ...); a warp takes groups of 32 consecutive
//              faces of the rows' face sequence from a buffer of its own, shuffles between lanes
//   k_visc_tiled  reduced 2nd-order viscous terms, conservative face Laplacian in x, y, z,
//              div/3, stage-3 Ducros sensor, wall shear; planes in a ring in shared memory
//   k_march<1> y-face fluxes + divergence (fl += ...); rounds of faces from a ring in shared memory
//   k_march<2> z-face fluxes + divergence + grad(mu div/3) term; block partials of force_rhs
//   k_finish_rhs  bulk quantities and the forcing correction (deterministic order)
//   k_update   RK register fln, forcing correction, w += fln, force_var / residual partials
//   k_finish_upd  bulk temperature -> pending energy shift; residual and min/max
// No face flux array is stored.  All reductions are block partials summed in a fixed order, so
// results do not depend on scheduling.
//
// Precision: template parameter R is the arithmetic type of the fluxes and viscous terms and the
// storage type of the primitive fields (aux) and div/3.  R = double is the FP64 form; R = float
// the mixed form, where w, the RK registers fl, the temperature recovery from the total energy,
// the Ducros sensor, the time step and all reductions stay FP64 and the face fluxes are summed and
// differenced in FP64.
#pragma once

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "flux.cuh"
#include "kernels.hpp"

namespace sb200 {

namespace {

constexpr int AUX_NT = 256;
constexpr int XF_TX = 32, XF_TY = 4, XF_NT = XF_TX * XF_TY;  // x faces: 4 warps per block
// y / z passes: blocks of LW = 4 warps, up to MT_MAXW in small boxes; segments of at most MT_SEG cells
constexpr int MT_MAXW = 9, MT_SEG = 2048;
// Registers of the flux kernels, as the threads an SM shall hold (y / z: 65536 / MT_MAXT_* registers
// for blocks of any size) or the blocks of 128 (x, WENO faces).  FP64 takes 128 registers
// (1024x256x192 boundary layer, ms per step: y 11.0, z 12.5, x 10.7 at 16 warps per SM, without
// spills; an earlier form at 20 warps and 96 registers, spilling 30-130 bytes: 12.7, 14.4, 11.8
// against 11.5, 13.2, 11.0).  FP32: 96 in y and z (1024x256x128 shock interaction z 8.7, y 7.2
// against 9.3, 7.3 at 80; 512x256x256 channel 5.8, 3.3 against 5.8, 3.1), 80 in x (6.9 and 2.8
// against 7.1 and 2.9 at 96).  The WENO face kernels' scattered stencils: 3 blocks (6.5 against
// 7.2 ms at 4) and 4 in FP32.
#ifndef MT_MAXT_D
#define MT_MAXT_D 512
#endif
#ifndef MT_MAXT_F
#define MT_MAXT_F 640
#endif
#ifndef XF_MINB_D
#define XF_MINB_D 4
#endif
#ifndef XF_MINB_F
#define XF_MINB_F 6
#endif
#ifndef WF_MINB_D
#define WF_MINB_D 3
#endif
// KEEP(n) (FS & 4) of order 8 in FP64, whose central flux holds eight values of eight points, takes 168
// registers: at 128 its passes spill up to 576 bytes (256x128x128 channel in noise, WENO7, ms per step
// for nkeep = -1, 1, 2: 15.0, 20.0, 25.1 at 128; 13.1, 18.6, 21.6 at 168; a marching form of 168
// registers 14.5, 21.3, 23.5).  Order 6 stays at 128: nkeep = 2 10.0 against 10.3 at 168.
template <class R, int LB, int FS>
constexpr bool wide_keep() { return sizeof(R) == sizeof(double) && LB == 4 && (FS & 4) != 0; }
template <class R, int LB, int FS>
constexpr int x_minb() { return sizeof(R) == sizeof(float) ? XF_MINB_F : (wide_keep<R, LB, FS>() ? 3 : XF_MINB_D); }
template <class R, int LB, int FS>
constexpr int march_maxt() { return sizeof(R) == sizeof(float) ? MT_MAXT_F : (wide_keep<R, LB, FS>() ? 384 : MT_MAXT_D); }
#ifndef WF_MINB_F
#define WF_MINB_F 4
#endif
// shared-memory carve-out (percent) preferred by the WENO face kernels: their listed faces'
// stencil loads are scattered and live on L1 hits (developed boundary layer 1024x256x192: 5.0
// against 8.1 ms per step of face kernels with the largest carve-out, which fits a fourth block)
#ifndef SB_WF_CARVEOUT
#define SB_WF_CARVEOUT 72
#endif
// the viscous pass: FP64 at 2 blocks of 256 threads per SM (4.2 ms per step on the 1024x256x192
// boundary layer; 5.8 at 3 blocks, whose 80 registers spill 140 bytes), FP32 at 4
#ifndef VISC_MINB
#define VISC_MINB 2
#endif
// resident threads per SM asked of the register allocator for the memory-bound pointwise passes:
// 2048 (32 registers, a little spilling in the update pass), for more loads in flight
// (1024x256x192 boundary layer, ms per step against the allocator's own choice: update 4.24
// against 5.02 at 60 registers, 4.51 at 1536 threads; aux 3.01 against 3.23; dt 1.12 against
// 1.27).  The update pass's blocks are 1024 threads (UPD_MINB of them; 4.63 at 64 registers and one
// block), the others 256.
#ifndef UPD_MINB
#define UPD_MINB 2
#endif
#ifndef AUX_MINB
#define AUX_MINB 8
#endif
#ifndef AUX_MINB_DT
#define AUX_MINB_DT 6
#endif
#ifndef DT_MINB
#define DT_MINB 8
#endif
#ifndef VISC_MINB_F
#define VISC_MINB_F 4
#endif
constexpr int FIN_NT = 1024;
// cells per block of the update and time-step passes: 1024 (the time-step pass: 4 per thread of
// 256), a quarter of the block partials for their one-block finishing reductions (1024x256x192:
// 0.43 -> 0.13 and 0.17 -> 0.05 ms per step)
#ifndef SB_PT_CELLS
#define SB_PT_CELLS 4
#endif
constexpr int PT_CELLS = SB_PT_CELLS;
// the update pass: one cell per thread in blocks of 1024 (the same count of block partials)
constexpr int UPD_NT = 256 * PT_CELLS;
inline unsigned pt_blocks(long long nint) { return (unsigned)((nint + 256 * PT_CELLS - 1) / (256 * PT_CELLS)); }

// Block coordinates seen by a kernel body (d_*): the hardware block index in a plain launch
// (k_*), the block's place in its own box's grid in a launch over a box table (kb_*)
struct Blk {
  unsigned x, y, z;
};

// Primitive state of an interior point recomputed from w in FP64, with the operations of
// eval_aux_subroutine (kernels_cpu.F90:6960-7011).
struct Prim {
  double rho, uu, vv, ww, tt;
};
template <bool TPA = true>
__device__ __forceinline__ Prim prim_from_w(const Geom& g, const double* __restrict__ w, long long c,
                                            double t_start) {
  const long long n = g.nvol;
  Prim p;
  p.rho = w[c];
  const double ri = 1.0 / p.rho;
  p.uu = w[n + c] * ri;
  p.vv = w[2 * n + c] * ri;
  p.ww = w[3 * n + c] * ri;
  const double qq = 0.5 * (p.uu * p.uu + p.vv * p.vv + p.ww * p.ww);
  p.tt = t_from_e<TPA>(g, w[4 * n + c] / p.rho - qq, t_start);
  return p;
}

// Conserved state at an interior or face-ghost point (i,j,k): the stored value, a periodic copy
// (bcswap, code/src/base_cpu.F90:1326-1435) or the staggered-wall mirror of
// bcwall_staggered_subroutine (kernels_cpu.F90:6612-6678); t_src is the start of the Newton
// iteration for the mirrored point's temperature (thermally perfect gas).
template <bool TPA = true>
__device__ __forceinline__ void point_state(const Geom& g, const double* __restrict__ w, int i, int j, int k,
                                            double (&st)[5], double t_src) {
  const long long n = g.nvol;
  const int ox = (i < 1 || i > g.nx), oy = (j < 1 || j > g.ny), oz = (k < 1 || k > g.nz);
  int si = i, sj = j, sk = k;
  int wall = 0;
  // periodic faces wrap, staggered walls mirror; any other face reads its stored ghost
  if (ox && g.periodic[0]) si = wrap(i, g.nx);
  if (oz && g.periodic[2]) sk = wrap(k, g.nz);
  if (oy) {
    if (j < 1) {
      if (g.periodic[1]) sj = j + g.ny;
      else if (g.wall_ymin) { sj = 1 - j; wall = 1; }
    } else {
      if (g.periodic[1]) sj = j - g.ny;
      else if (g.wall_ymax) { sj = 2 * g.ny + 1 - j; wall = 1; }
    }
  }
  const long long src = gidx(g, si, sj, sk);
  double rho = w[src], rhou = w[n + src], rhov = w[2 * n + src], rhow = w[3 * n + src], rhoe = w[4 * n + src];
  if (wall) {
    // mirror about the wall, T_g = 2 T_w - T, p_g = p, velocity reversed
    double uu = rhou / rho, vv = rhov / rho, ww = rhow / rho;
    double qq = 0.5 * (uu * uu + vv * vv + ww * ww);
    double ee = rhoe / rho - qq;
    double tt = t_from_e<TPA>(g, ee, t_src);
    double pp = rho * tt * g.rgas0;
    tt = 2.0 * g.t_wall - tt;
    ee = e_from_t<TPA>(g, tt);
    rho = pp / tt / g.rgas0;
    rhou = -rho * uu;
    rhov = -rho * vv;
    rhow = -rho * ww;
    rhoe = rho * (ee + qq);
  }
  st[0] = rho; st[1] = rhou; st[2] = rhov; st[3] = rhow; st[4] = rhoe;
}

// Inverse time scales of a cell (compute_dt_subroutine, kernels_cpu.F90:6814-6880): the largest of
// the nine, three convective, three viscous and three conductive ones.  Rounding is monotone, so the
// largest of the products with a metric is the product of the largest.
__device__ __forceinline__ double inverse_dt(const Geom& g, int i, int j, int k, double uu, double vv, double ww,
                                             double cs, double nu) {
  const double kr = nu / g.prandtl, nk = fmax(nu, kr);
  double m = fmax((fabs(uu) + cs) * g.dcsidx[i], fmax((fabs(vv) + cs) * g.detady[j], (fabs(ww) + cs) * g.dzitdz[k]));
  return fmax(m, nk * fmax(g.dcsidxs[i], fmax(g.detadys[j], g.dzitdzs[k])));
}
// largest of the block's values (non-negative) into out
__device__ __forceinline__ void block_max(double m, double* __restrict__ out) {
  __shared__ double sm[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) m = fmax(m, sm[q]);
    *out = m;
  }
}

// w -> aux at all interior and face-ghost points (eval_aux_subroutine, kernels_cpu.F90:6960-7011),
// computed in FP64 and stored as A; with write_ghost_w = 1 the ghost states are also stored into
// w, with write_ghost_w = 2 only they are (aux is left as it is).  With vel non-null the FP64
// velocities are stored too (the mixed form's stage-3 sensor reads them).  DT: the pass that starts
// a step also leaves the block maxima of the inverse time scales in red, for which a pass of its own
// read 48 (FP64) or 40 (mixed) bytes a cell: 1024x256x192, both passes 4.04 -> 3.21 ms per step,
// 1024x256x128 mixed 2.38 -> 1.76.  Memory bound (104 and 68 bytes a point); quotients by the density
// and by constants are products with reciprocals.
template <class A, bool TP, bool DT>
__device__ __forceinline__ void d_aux(const Geom& g, double* __restrict__ w, A* __restrict__ aux, int write_ghost_w,
                                      double* __restrict__ vel, double* __restrict__ red, const Blk blk) {
  const long long n = g.nvol;
  const long long q = (long long)blk.x * AUX_NT + threadIdx.x;
  double m = 0.0;
  auto point = [&]() {
    const unsigned qu = (unsigned)q, r = qu / (unsigned)g.sx;  // fewer than 2^32 points: more do not fit the memory
    const int ii = (int)(qu - r * (unsigned)g.sx);
    const int kk = (int)(r / (unsigned)g.sy), jj = (int)(r - (unsigned)kk * (unsigned)g.sy);
    const int i = ii - g.ng + 1, j = jj - g.ng + 1, k = kk - g.ng + 1;
    const int ox = (i < 1 || i > g.nx), oy = (j < 1 || j > g.ny), oz = (k < 1 || k > g.nz);
    if (ox + oy + oz > 1) return;  // halo edges and corners are never read
    if (write_ghost_w == 2 && !(ox | oy | oz)) return;
    const long long dst = gidx(g, i, j, k);
    // Newton starts (thermally perfect gas): the point's previous temperature, as eval_aux starts
    // from w_aux(6); for a wall ghost the mirror of it estimates the interior source point's
    double t_old = g.t0, t_src = g.t0;
    if constexpr (TP) {
      t_old = double(aux[5 * n + dst]);
      if (!(t_old > 0.0)) t_old = g.t0;
      t_src = 2.0 * g.t_wall - t_old;
      if (!(t_src > 0.0)) t_src = g.t0;
    }
    double st[5];
    point_state<TP>(g, w, i, j, k, st, t_src);
    const double rho = st[0], rhou = st[1], rhov = st[2], rhow = st[3], rhoe = st[4];
    if (write_ghost_w && (ox | oy | oz)) {
      w[dst] = rho; w[n + dst] = rhou; w[2 * n + dst] = rhov; w[3 * n + dst] = rhow; w[4 * n + dst] = rhoe;
    }
    if (write_ghost_w == 2) return;  // ghost layers of w only; aux keeps its values
    const double ri = rcp_pos(rho);
    const double uu = rhou * ri, vv = rhov * ri, ww = rhow * ri;
    const double qq = 0.5 * (uu * uu + vv * vv + ww * ww);
    const double ee = rhoe * ri - qq;
    const double tt = t_from_e<TP>(g, ee, t_old);
    const double pp = rho * tt * g.rgas0;
    if (vel) {  // FP64 velocities, as the sensor forms them from w
      vel[dst] = uu;
      vel[n + dst] = vv;
      vel[2 * n + dst] = ww;
    }
    aux[dst] = A(rho);
    aux[n + dst] = A(uu);
    aux[2 * n + dst] = A(vv);
    aux[3 * n + dst] = A(ww);
    aux[4 * n + dst] = A((rhoe + pp) * ri);
    aux[5 * n + dst] = A(tt);
    double mu = 0.0, cs = 0.0;
    if constexpr (DT || sizeof(A) == sizeof(double)) {
      mu = viscosity(g, tt);
      cs = sqrt((TP ? gamloc_of_t(g, tt) : g.gamloc) * g.rgas0 * tt);
    }
    // the mixed form's viscous arithmetic is FP32, and so is its viscosity law (with SB_FP32_FAST)
    if constexpr (sizeof(A) == sizeof(float) && SB_FP32_FAST != 0)
      aux[6 * n + dst] = viscosity_f(g, float(tt));
    else
      aux[6 * n + dst] = A(viscosity(g, tt));
    // FP64 form: the sound speed, which the WENO eigenvalue bound of every face reads at its
    // stencil points (the same expression the flux would form)
    if constexpr (sizeof(A) == sizeof(double)) aux[7 * n + dst] = cs;
    if constexpr (DT)
      if (!(ox | oy | oz)) m = inverse_dt(g, i, j, k, uu, vv, ww, cs, ri * mu);
  };
  if (q < n) point();
  if constexpr (DT) block_max(m, red + blk.x);
}
template <class A, bool TP = false, bool DT = false>
__global__ void __launch_bounds__(AUX_NT, DT ? AUX_MINB_DT : AUX_MINB)
    k_aux(Geom g, double* __restrict__ w, A* __restrict__ aux, int write_ghost_w, double* __restrict__ vel,
          double* __restrict__ red) {
  d_aux<A, TP, DT>(g, w, aux, write_ghost_w, vel, red, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// Ducros sensor in FP64 from w for the mixed form, so that the central/WENO switch is taken
// on the same values as in the FP64 form.  mode 0: initial sensor of run() (visflx(mode=2),
// kernels_cpu.F90:4680-4682); mode 1: sensor_subroutine of stage 3 (:4726-4744), which works
// from the stored |omega| and div/3 of visflx_reduced_ord2; mode 2: the same from the
// visc_order derivatives of visflx_nosensor_subroutine (conservative_viscous = 0); mode 3: the
// initial sensor of run() for conservative_viscous = 0 (visflx(mode=0), visflx_subroutine,
// kernels_cpu.F90:3598-3777: visc_order derivatives, theta from div and omega directly).
__device__ __forceinline__ void d_sensor64(const Geom& g, const double* __restrict__ w, double* __restrict__ out,
                                                  int mode, const Blk blk) {
  const long long q = (long long)blk.x * 256 + threadIdx.x;
  if (q >= g.nint) return;
  int i, j, k;
  cell_of(g, q, i, j, k);
  auto vel = [&](int a, int b, int c, double (&v)[3]) {
    double st[5];
    point_state(g, w, a, b, c, st, g.t_wall);
    const double ri = 1.0 / st[0];
    v[0] = st[1] * ri; v[1] = st[2] * ri; v[2] = st[3] * ri;
  };
  double ux, vx, wx, uy, vy, wy, uz, vz, wz;
  if (mode < 2) {
    double xp[3], xm[3], yp[3], ym[3], zp[3], zm[3];
    vel(i + 1, j, k, xp); vel(i - 1, j, k, xm);
    vel(i, j + 1, k, yp); vel(i, j - 1, k, ym);
    vel(i, j, k + 1, zp); vel(i, j, k - 1, zm);
    double dxl = 1.0 / (g.x[i + 1] - g.x[i - 1]);
    double dyl = 1.0 / (g.y[j + 1] - g.y[j - 1]);
    double dzl = 1.0 / (g.z[k + 1] - g.z[k - 1]);
    ux = dxl * (xp[0] - xm[0]); vx = dxl * (xp[1] - xm[1]); wx = dxl * (xp[2] - xm[2]);
    uy = dyl * (yp[0] - ym[0]); vy = dyl * (yp[1] - ym[1]); wy = dyl * (yp[2] - ym[2]);
    uz = dzl * (zp[0] - zm[0]); vz = dzl * (zp[1] - zm[1]); wz = dzl * (zp[2] - zm[2]);
  } else {
    // the derivatives of visflx_nosensor_subroutine (order visc_order, metric after the sum)
    const int lv = g.lmax_base;
    double d[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int l = 1; l <= lv; ++l) {
      const double ccl = g.coeff[lv - 1][l - 1];
      double p[3], m[3];
      vel(i + l, j, k, p); vel(i - l, j, k, m);
      for (int v = 0; v < 3; ++v) d[0][v] = d[0][v] + ccl * (p[v] - m[v]);
      vel(i, j + l, k, p); vel(i, j - l, k, m);
      for (int v = 0; v < 3; ++v) d[1][v] = d[1][v] + ccl * (p[v] - m[v]);
      vel(i, j, k + l, p); vel(i, j, k - l, m);
      for (int v = 0; v < 3; ++v) d[2][v] = d[2][v] + ccl * (p[v] - m[v]);
    }
    ux = d[0][0] * g.dcsidx[i]; vx = d[0][1] * g.dcsidx[i]; wx = d[0][2] * g.dcsidx[i];
    uy = d[1][0] * g.detady[j]; vy = d[1][1] * g.detady[j]; wy = d[1][2] * g.detady[j];
    uz = d[2][0] * g.dzitdz[k]; vz = d[2][1] * g.dzitdz[k]; wz = d[2][2] * g.dzitdz[k];
  }
  double div = ux + vy + wz;
  double omegax = wy - vz, omegay = uz - wx, omegaz = vx - uy;
  double omod2 = omegax * omegax + omegay * omegay + omegaz * omegaz;
  double u0l0 = g.u0 / g.l0;
  if (mode == 1 || mode == 2) {
    double div3l = div / 3.0;
    double om = sqrt(omod2);
    omod2 = om * om;
    div = 3.0 * div3l;
  }
  double t = fmax(-div / sqrt(omod2 + div * div + u0l0 * u0l0), 0.0);
  out[q] = t * t;
}
__global__ void __launch_bounds__(256) k_sensor64(Geom g, const double* __restrict__ w, double* __restrict__ out,
                                                  int mode) {
  d_sensor64(g, w, out, mode, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}
// The stage-3 Ducros sensor of the mixed form (k_sensor64 modes 1 and 2) from the FP64 velocities
// that the stage's aux pass stored at the interior and face-ghost points: the same quotients and
// the same arithmetic, without re-forming six neighbours' states per point.
__device__ __forceinline__ void d_sensor_vel(const Geom& g, const double* __restrict__ vel, double* __restrict__ out,
                                                    int mode, const Blk blk) {
  const long long q = (long long)blk.x * 256 + threadIdx.x;
  if (q >= g.nint) return;
  int i, j, k;
  cell_of(g, q, i, j, k);
  const long long n = g.nvol, c = gidx(g, i, j, k), sY = g.sx, sZ = (long long)g.sx * g.sy;
  auto V = [&](long long a, int m) { return vel[m * n + a]; };
  double ux, vx, wx, uy, vy, wy, uz, vz, wz;
  if (mode == 1) {
    double dxl = 1.0 / (g.x[i + 1] - g.x[i - 1]);
    double dyl = 1.0 / (g.y[j + 1] - g.y[j - 1]);
    double dzl = 1.0 / (g.z[k + 1] - g.z[k - 1]);
    ux = dxl * (V(c + 1, 0) - V(c - 1, 0)); vx = dxl * (V(c + 1, 1) - V(c - 1, 1)); wx = dxl * (V(c + 1, 2) - V(c - 1, 2));
    uy = dyl * (V(c + sY, 0) - V(c - sY, 0)); vy = dyl * (V(c + sY, 1) - V(c - sY, 1));
    wy = dyl * (V(c + sY, 2) - V(c - sY, 2));
    uz = dzl * (V(c + sZ, 0) - V(c - sZ, 0)); vz = dzl * (V(c + sZ, 1) - V(c - sZ, 1));
    wz = dzl * (V(c + sZ, 2) - V(c - sZ, 2));
  } else {
    const int lv = g.lmax_base;
    double d[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int l = 1; l <= lv; ++l) {
      const double ccl = g.coeff[lv - 1][l - 1];
      for (int v = 0; v < 3; ++v) d[0][v] = d[0][v] + ccl * (V(c + l, v) - V(c - l, v));
      for (int v = 0; v < 3; ++v) d[1][v] = d[1][v] + ccl * (V(c + l * sY, v) - V(c - l * sY, v));
      for (int v = 0; v < 3; ++v) d[2][v] = d[2][v] + ccl * (V(c + l * sZ, v) - V(c - l * sZ, v));
    }
    ux = d[0][0] * g.dcsidx[i]; vx = d[0][1] * g.dcsidx[i]; wx = d[0][2] * g.dcsidx[i];
    uy = d[1][0] * g.detady[j]; vy = d[1][1] * g.detady[j]; wy = d[1][2] * g.detady[j];
    uz = d[2][0] * g.dzitdz[k]; vz = d[2][1] * g.dzitdz[k]; wz = d[2][2] * g.dzitdz[k];
  }
  double div = ux + vy + wz;
  double omegax = wy - vz, omegay = uz - wx, omegaz = vx - uy;
  double omod2 = omegax * omegax + omegay * omegay + omegaz * omegaz;
  double u0l0 = g.u0 / g.l0;
  double div3l = div / 3.0;
  double om = sqrt(omod2);
  omod2 = om * om;
  div = 3.0 * div3l;
  double t = fmax(-div / sqrt(omod2 + div * div + u0l0 * u0l0), 0.0);
  out[q] = t * t;
}
__global__ void __launch_bounds__(256) k_sensor_vel(Geom g, const double* __restrict__ vel, double* __restrict__ out,
                                                    int mode) {
  d_sensor_vel(g, vel, out, mode, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// Pending energy shift on interior points only (before a download).  The Newton start of the
// thermally perfect gas is the point's temperature in aux, as force_var_1 starts from w_aux(6).
template <class A, bool TP = false>
__device__ __forceinline__ void d_apply_shift(const Geom& g, double* __restrict__ w, const A* __restrict__ aux,
                                                        const Scalars* __restrict__ sc, const Blk blk) {
  const long long q = (long long)blk.x * AUX_NT + threadIdx.x;
  if (q >= g.nint) return;
  int i, j, k;
  cell_of(g, q, i, j, k);
  const long long n = g.nvol, s = gidx(g, i, j, k);
  const double t_start = TP ? double(aux[5 * n + s]) : g.t0;
  w[4 * n + s] = shifted_rhoe<TP>(g, w[s], w[n + s], w[2 * n + s], w[3 * n + s], w[4 * n + s], sc->tbdiff, t_start);
}
template <class A, bool TP = false>
__global__ void __launch_bounds__(AUX_NT) k_apply_shift(Geom g, double* __restrict__ w, const A* __restrict__ aux,
                                                        const Scalars* __restrict__ sc) {
  d_apply_shift<A, TP>(g, w, aux, sc, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// Readers of the interior-only sensor and div/3 arrays at a stencil point that may be a ghost.
template <class R>
__device__ __forceinline__ R sensor_at(const Geom& g, const R* __restrict__ s, int i, int j, int k) {
  if (i < 1 || i > g.nx) { if (!g.periodic[0]) return R(0); i = wrap(i, g.nx); }
  if (j < 1 || j > g.ny) { if (!g.periodic[1]) return R(0); j = wrap(j, g.ny); }
  if (k < 1 || k > g.nz) { if (!g.periodic[2]) return R(0); k = wrap(k, g.nz); }
  return s[iidx(g, i, j, k)];
}
// bcextr_var (kernels_cpu.F90:6199-6254) then bcswap_var: periodic wrap, otherwise nearest interior
__device__ __forceinline__ long long div3_idx(const Geom& g, int i, int j, int k) {
  if (i < 1 || i > g.nx) i = g.periodic[0] ? wrap(i, g.nx) : (i < 1 ? 1 : g.nx);
  if (j < 1 || j > g.ny) j = g.periodic[1] ? wrap(j, g.ny) : (j < 1 ? 1 : g.ny);
  if (k < 1 || k > g.nz) k = g.periodic[2] ? wrap(k, g.nz) : (k < 1 ? 1 : g.nz);
  return iidx(g, i, j, k);
}
template <class R>
__device__ __forceinline__ R div3_at(const Geom& g, const R* __restrict__ d, int i, int j, int k) {
  return d[div3_idx(g, i, j, k)];
}

// 1/(x(i+1)-x(i-1)) of a line of direction d in R
template <class R>
__device__ __forceinline__ R line_r(const Geom& g, int d, int i) {
  if constexpr (sizeof(R) == sizeof(double)) return __ldg(g.vrl[d] + i);
  else return __ldg(g.vrlf[d] + i);
}

// Quotient by a value b that comes with its rounded reciprocal r: a product in FP64; in FP32 the
// rounded quotient itself (a r corrected by its remainder, Markstein), so that the mixed form's FP32
// results are those of a division.
template <class R>
struct Quot {
  R b, r;
};
__device__ __forceinline__ double quot(double a, const Quot<double>& q) { return a * q.r; }
__device__ __forceinline__ float quot(float a, const Quot<float>& q) {
  const float t = __fmul_rn(a, q.r);
  return __fmaf_rn(q.r, __fmaf_rn(-q.b, t, a), t);
}
// x(i+1)-x(i) of a face and its reciprocal, i = 0 .. n
template <class R>
__device__ __forceinline__ Quot<R> face_r(const Geom& g, int d, int i) {
  if constexpr (sizeof(R) == sizeof(double)) return Quot<R>{R(0), __ldg(g.vfr[d] + i)};
  else return Quot<R>{__ldg(g.vfdf[d] + i), __ldg(g.vfrf[d] + i)};
}

template <int DIR>
__device__ __forceinline__ int face_ep(const Geom& g, int p) {
  return DIR == 0 ? g.epx[p] : (DIR == 1 ? g.epy[p] : g.epz[p]);
}

// WENO faces apart (1) or always inside the hybrid passes (0).  Apart, the faces whose stencil
// sees the sensor are listed per direction once per step and computed by their own kernel at
// full occupancy; the hybrid passes read their fluxes from a face buffer.  A warp of the hybrid
// passes otherwise runs both branches whenever one of its faces is a WENO face.  The face kernels
// gather their stencils one sector a value and the buffer is written and read, so each direction
// chooses on the device from its list's length (weno_split): the x pass holds both branches, the y
// and z passes are launched in both forms and the one not chosen leaves at once.  The lists
// themselves are built only when a sample of every 16th plane is within the threshold, so a step
// that keeps its WENO faces in the hybrid passes pays for the sample and the unused launches
// (0.3 of 47.6 ms per step at 1024x256x192).  What either form costs: WENO_SPLIT_FRAC_DEFAULT.
#ifndef SB_WENO_SPLIT
#define SB_WENO_SPLIT 1
#endif

// Face index of the WENO face buffer of direction DIR for face p (0..n along DIR) of the line
// (a, b): x faces p fastest (a = j, b = k), y and z faces i fastest (a = i; b = k for y, j for z).
template <int DIR>
__host__ __device__ __forceinline__ long long wface_index(const Geom& g, int p, int a, int b) {
  if (DIR == 0) return ((long long)(b - 1) * g.ny + (a - 1)) * (g.nx + 1) + p;
  if (DIR == 1) return ((long long)(b - 1) * (g.ny + 1) + p) * g.nx + (a - 1);
  return ((long long)p * g.ny + (b - 1)) * g.nx + (a - 1);
}
template <int DIR>
__device__ __forceinline__ void wface_decode(const Geom& g, unsigned f, int& p, int& a, int& b) {
  // face counts per direction stay below 2^32 (checked at context creation)
  if (DIR == 0) {
    const unsigned n0 = g.nx + 1, r = f / n0;
    p = (int)(f - r * n0);
    a = (int)(r % (unsigned)g.ny) + 1;
    b = (int)(r / (unsigned)g.ny) + 1;
  } else if (DIR == 1) {
    const unsigned r = f / (unsigned)g.nx;
    a = (int)(f - r * (unsigned)g.nx) + 1;
    p = (int)(r % (unsigned)(g.ny + 1));
    b = (int)(r / (unsigned)(g.ny + 1)) + 1;
  } else {
    const unsigned r = f / (unsigned)g.nx;
    a = (int)(f - r * (unsigned)g.nx) + 1;
    b = (int)(r % (unsigned)g.ny) + 1;
    p = (int)(r / (unsigned)g.ny);
  }
}
// Whether the hybrid pass of direction DIR reads its WENO faces from the face buffer this step
// (the list, built at stage 1, holds at most wthr[DIR] faces) or computes them itself.
template <int DIR>
__device__ __forceinline__ bool weno_split(const Geom& g) {
  return SB_WENO_SPLIT && g.wsplit_on && *(volatile const unsigned*)(g.wcount + DIR) <= g.wthr[DIR];
}
template <int DIR>
__host__ __device__ __forceinline__ long long wface_count(const Geom& g) {
  return DIR == 0 ? (long long)(g.nx + 1) * g.ny * g.nz
                  : (DIR == 1 ? (long long)g.nx * (g.ny + 1) * g.nz : (long long)g.nx * g.ny * (g.nz + 1));
}

// Flux at a face in FP64 from its stencil in memory.  FS holds the flux variant flags of a
// kernel instantiation: bit 0 the component-wise (Rusanov) WENO splitting, bit 1 the thermally
// perfect gas, bit 2 a central flux with nkeep != 0 (otherwise nkeep = 0 at compile time), bit 3
// the WENO-Z weights (otherwise WENO-JS).  Options fixed per kernel instantiation keep the code
// of the branches a case does not take out of the register allocation of the ones it does
// (measured: nkeep 10-18 %, the WENO version 3-10 % of the flux passes).
// The WENO flux of face p (characteristic or component-wise splitting), order reduced near
// non-periodic boundaries as ep_ord_change says.
template <class R, int DIR, int LB, int WS, int S, int FS, class LN>
__device__ __forceinline__ void weno_face(const Geom& g, const LN& ln, int ep, double (&f)[5], const Scr<R>& scr) {
  const int ord = max(WS + ep, 1);
  auto flux = [&](auto full) {
    [[maybe_unused]] constexpr bool FULL = decltype(full)::value;
    if constexpr ((FS & 1) != 0) rusanov_flux<R, DIR, WS, S, (FS & 2) != 0, (FS & 8) != 0, FULL>(g, ln, ord, f);
    else if constexpr (sizeof(R) == sizeof(double)) weno_flux<DIR, WS, S, (FS & 2) != 0, (FS & 8) != 0, FULL>(g, ln, ord, f, scr);
    else weno_flux_f<DIR, WS, S, (FS & 8) != 0>(g, ln, ord, f, scr);
  };
  if (sizeof(R) != sizeof(double) || ord == WS) flux(std::true_type{});
  else flux(std::false_type{});
}

template <class R, int DIR, int LB, int WS, int S, int FS, class LN>
__device__ __forceinline__ void face_flux(const Geom& g, const LN& ln, bool ishk, int p, int ep, double (&f)[5],
                                          const Scr<R>& scr, bool split, int wa, int wb) {
  const int nd = DIR == 0 ? g.nx : (DIR == 1 ? g.ny : g.nz);
  if (!ishk) {
    const int lmax = max(g.lmax_base + ep, 1);
    const bool zf = (p == 0 && g.fzf[2 * DIR] == 1) || (p == nd && g.fzf[2 * DIR + 1] == 1);
    central_flux<R, DIR, LB, S, (FS & 4) != 0>(g, ln, lmax, g.nkeep, zf, f);
  } else if (SB_WENO_SPLIT && split) {
    // the WENO faces come from the face buffer
    const long long wf = wface_index<DIR>(g, p, wa, wb);
#pragma unroll
    for (int m = 0; m < 5; ++m) f[m] = __ldg(g.wface + m * g.nwface + wf);
  } else {
    weno_face<R, DIR, LB, WS, S, FS>(g, ln, ep, f, scr);
  }
}

// asynchronous copies of one value from global to shared memory
__device__ __forceinline__ void copy_async(unsigned dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async(unsigned dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// x faces.  The faces of all rows form one sequence (row (k-1) ny + (j-1), faces p = 0..nx in a row;
// fewer than 2^32 faces, checked at create), so that no lane idles at a row's end.  A warp takes
// ngrp groups of 32 consecutive faces one after another (its first face is the last of the warp
// before) and forms the cells below its faces, the lower face of a cell coming from the lane before
// by a shuffle and from the group before through shared memory.  A group's points are copied to the
// warp's own buffer while the group before is computed (no block barrier anywhere): 32 points and
// 2S - 1 more for every row that the group touches, and the sensor beside them.  1024x256x192
// boundary layer, ms per step: 16.7 with the stencil loaded by every face into registers, 13.7 read
// from L1 as often as used, 11.5 from the buffer (10.7 with the present weno_flux).
// fl is written (first contribution of the stage, euler_x after init_flux).
constexpr int XG_MAX = 8, X_SMEM_MAX = 96 * 1024;  // rows of 4 cells, WENO7 in FP64: 78 KB
struct XShape {
  int ngrp, slots;
  unsigned nblk;
};
__host__ __device__ __forceinline__ int x_slots(int nx, int S) { return 32 + (2 * S - 1) * ((31 + nx) / (nx + 1) + 1); }
template <class R, int WS>
__host__ __device__ __forceinline__ size_t x_warp_bytes(int slots) {
  return 2 * (size_t)((slots * XS * (int)sizeof(R) + 7) / 8 * 8 + slots * 8) + 5 * 8 + scr_vals<R, WS>() * 32 * sizeof(R);
}
template <class R, int LB, int WS, int FS = 0>
__device__ __forceinline__ void d_xflux(const Geom& g, const R* __restrict__ aux, const double* __restrict__ sensor,
                                        double* __restrict__ fl, int ngrp, const Blk blk) {
  constexpr int S = LB > WS ? LB : WS, W2 = 2 * S - 1, RF = ring_fields<R>();
  extern __shared__ __align__(16) unsigned char sb_dyn_smem[];
  const int lane = threadIdx.x, nfr = g.nx + 1, slots = x_slots(g.nx, S);
  const unsigned long long nface = (unsigned long long)nfr * g.ny * g.nz;
  const unsigned long long fw0 = (unsigned long long)(blk.x * XF_TY + threadIdx.y) * (unsigned)(32 * ngrp - 1);
  if (fw0 >= nface) return;  // whole warp leaves together
  const unsigned nmine = (unsigned)min((unsigned long long)(32 * ngrp), nface - fw0);  // this warp's faces
  unsigned char* wm = sb_dyn_smem + threadIdx.y * x_warp_bytes<R, WS>(slots);
  const Scr<R> scr{reinterpret_cast<R*>(wm) + lane, 32};
  wm += scr_vals<R, WS>() * 32 * sizeof(R);
  double* carry = reinterpret_cast<double*>(wm);  // the group before's last face
  const unsigned pb = (unsigned)((slots * XS * (int)sizeof(R) + 7) / 8 * 8);  // bytes of a buffer's points
  unsigned char* buf0 = wm + 5 * 8;
  // a group's first face (p0 of the row j0, k0); the faces of a group in its first row
  struct Pos {
    int p, j, k;
  };
  auto forward = [&](Pos q, int n) {  // n faces on
    q.p += n;
    while (q.p >= nfr) {
      q.p -= nfr;
      if (++q.j > g.ny) {
        q.j = 1;
        ++q.k;
      }
    }
    return q;
  };
  // rows between the row of a group's first face and that of the face n after the row's face 0 (a
  // group touches two rows at most unless the rows are shorter than a warp)
  auto rows_on = [&](int n) { return n < nfr ? 0 : (n < 2 * nfr ? 1 : n / nfr); };
  auto fetch = [&](const Pos& q0, int nf, int bi) {  // the points of the nf faces from q0 on
    unsigned char* pts = buf0 + bi * (pb + slots * 8);
    double* sen = reinterpret_cast<double*>(pts + pb);
    const int n0 = nfr - q0.p;  // faces left in the first row
    const int total = nf + W2 * (rows_on(q0.p + nf - 1) + 1);
    for (int s = lane; s < total; s += 32) {
      Pos q = q0;
      int t = s;
      if (t < n0 + W2) {
        t += q.p;
      } else {
        t -= n0 + W2;
        q = forward(Pos{0, q.j, q.k}, nfr);
        while (t >= nfr + W2) {
          t -= nfr + W2;
          q = forward(q, nfr);
        }
      }
      const int i = t - (S - 1);
      const unsigned dst = (unsigned)__cvta_generic_to_shared(pts) + s * (XS * (unsigned)sizeof(R));
      const R* src = aux + gidx(g, i, q.j, q.k);
#pragma unroll
      for (int f = 0; f < RF; ++f) copy_async(dst + f * (unsigned)sizeof(R), src + (f == F_C ? 7 : f) * g.nvol);
      int is = i;
      if (i < 1 || i > g.nx) is = g.periodic[0] ? wrap(i, g.nx) : 0;
      if (is > 0) copy_async((unsigned)__cvta_generic_to_shared(sen + s), sensor + iidx(g, is, q.j, q.k));
      else sen[s] = 0.0;  // no sensor beyond a boundary
    }
  };
  Pos q0;
  {
    const unsigned fu = (unsigned)fw0, row = fu / (unsigned)nfr;
    q0.p = (int)(fu - row * (unsigned)nfr);
    q0.k = (int)(row / (unsigned)g.ny) + 1;
    q0.j = (int)(row - (unsigned)(q0.k - 1) * (unsigned)g.ny) + 1;
  }
  const bool split = weno_split<0>(g);
  fetch(q0, (int)min(32u, nmine), 0);
  copy_commit();
  for (unsigned b = 0; b < nmine; b += 32) {
    const int nf = (int)min(32u, nmine - b), bi = (b >> 5) & 1;
    const Pos qn = forward(q0, 32);
    // this lane's face (between the points p and p+1) and its first stencil point
    const Pos q = forward(q0, lane);
    const int s0 = lane + W2 * rows_on(q0.p + lane);
    const int p = q.p;
    const bool in = lane < nf;
    const int ep = in ? face_ep<0>(g, p) : 0;
    if (b + 32 < nmine) fetch(qn, (int)min(32u, nmine - b - 32), bi ^ 1);
    copy_commit();
    copy_wait<1>();
    __syncwarp();
    unsigned char* pts = buf0 + bi * (pb + slots * 8);
    const double* sen = reinterpret_cast<const double*>(pts + pb);
    double f[5] = {0, 0, 0, 0, 0};
    if (in && p >= g.eul_imin - 1 && p <= g.eul_imax) {
      bool ishk = false;
#pragma unroll
      for (int o = S - WS; o < S + WS; ++o) ishk = ishk | (sen[s0 + o] > g.sensor_threshold);
      const RowPts<R> ln{(unsigned)__cvta_generic_to_shared(pts) + s0 * (XS * (unsigned)sizeof(R))};
      face_flux<R, 0, LB, WS, S, FS>(g, ln, ishk, p, ep, f, scr, split, q.j, q.k);
    }
    // the cell i = p between the faces p-1 and p
    const bool cell = in && p >= 1 && b + lane > 0;
    const bool upd = cell && p >= g.eul_imin && p <= g.eul_imax;
    const double met = upd ? g.dcsidx[p] : 0.0;
    const long long ic = iidx(g, p, q.j, q.k);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      double lo = __shfl_up_sync(0xffffffffu, f[m], 1);
      if (lane == 0 && b > 0) lo = carry[m];
      if (cell) fl[m * g.nint + ic] = upd ? (f[m] - lo) * met : 0.0;
    }
    __syncwarp();  // the buffer and the carry have been read
    if (lane == 31)
#pragma unroll
      for (int m = 0; m < 5; ++m) carry[m] = f[m];
    q0 = qn;
  }
}
template <class R, int LB, int WS, int FS = 0>
__global__ void __launch_bounds__(XF_NT, x_minb<R, LB, FS>())
    k_xflux(Geom g, const R* __restrict__ aux, const double* __restrict__ sensor, double* __restrict__ fl, int ngrp) {
  d_xflux<R, LB, WS, FS>(g, aux, sensor, fl, ngrp, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// y or z faces: a block owns a tile of 32 lines (consecutive i of the lines' plane, so that every
// load is a coalesced row) over a segment of cells, and its warps take consecutive faces of the
// segment, one each per round.  The points sit in a ring in shared memory, copied once per block
// while the round before is computed, so that a face reads its stencil as often as it likes without
// the address arithmetic and the latency of global loads; the warps' fluxes meet in shared memory,
// where the cells between them find both faces.  A face is a chain of about a thousand FP64
// operations, most of them dependent: what bounds the pass is how many are in flight (22 % of the
// warp slots at 128 registers, FP64 pipe 60 % in y and 54 % in z).
// Against a thread marching alone along its line with the stencil in registers (168 of them, and
// 51 KB of scratch per block), 1024x256x192 boundary layer: y 17.0 -> 11.0, z 20.5 -> 12.5 ms per
// step; and since a segment takes a round per block of faces instead of a face at a time, a
// 32x24x16 channel's z pass 93 -> 17 us, its y pass 66 -> 19 us.  What a cell adds to is read before
// the barrier after the fluxes, which hides it behind the other warps' faces (in an earlier form:
// read after it y 12.6, z 16.1; copied to shared memory a round ahead 13.6, 17.3, the copies' own
// instructions; read before it 12.2, 13.6).
// The z pass also applies the grad(mu div/3) term of visflx_div_ord2_subroutine
// (kernels_cpu.F90:3446-3480) and emits the force_rhs block partials (:3157-3193).
//
// Dynamic shared memory: the fluxes of a round ((warps + 1) x 5 x 32, slot 0 the previous round's
// last face), the threads' scratch, the ring of points (the nw + 2S - 1 of a round and the nw of the
// next, which are copied while the round's fluxes are formed), the sensor flags of the segment's
// points (a word of 32 lanes each).
constexpr int MARCH_SMEM_MAX = 220 * 1024;
__host__ __device__ __forceinline__ int ring_slots(int nw, int S) { return 2 * nw + 2 * S - 1; }
template <class R, int LB, int WS>
size_t march_smem(int nwarps, int seglen, bool split = false) {
  constexpr int S = LB > WS ? LB : WS;
  return (size_t)(nwarps + 1) * 5 * 32 * 8 + (split ? 0 : (size_t)nwarps * 32 * scr_vals<R, WS>() * sizeof(R)) +
         (size_t)ring_slots(nwarps, S) * ring_fields<R>() * 32 * sizeof(R) + ((size_t)seglen + 2 * WS) * 4;
}
template <class R, int DIR, int LB, int WS, bool CH = false, int FS = 0, bool SPLIT = false>
__device__ __forceinline__ void d_march(const Geom& g, const R* __restrict__ aux,
                                                 const double* __restrict__ sensor, double* __restrict__ fl,
                                                 const R* __restrict__ div3,
                                                 const double* __restrict__ w, const double* __restrict__ fl_prev,
                                                 const Scalars* __restrict__ sc, double rhork, double gamrk,
                                                 int istep, int seglen, double* __restrict__ red, const Blk blk) {
  static_assert(DIR == 1 || DIR == 2, "march kernel handles y and z");
  constexpr int S = LB > WS ? LB : WS;
  extern __shared__ __align__(16) unsigned char sb_dyn_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* xch = reinterpret_cast<double*>(sb_dyn_smem);
  constexpr int RF = ring_fields<R>();
  const int nslot = ring_slots(nw, S);
  R* scd = reinterpret_cast<R*>(xch + (nw + 1) * 5 * 32);
  const Scr<R> scr{scd + threadIdx.x, (int)blockDim.x};
  R* ring = (scd + (SPLIT ? 0 : scr_vals<R, WS>() * blockDim.x));  // no WENO face is computed in the split form
  unsigned* flag = reinterpret_cast<unsigned*>(ring + nslot * RF * 32);
  const unsigned ring_a = (unsigned)__cvta_generic_to_shared(ring) + lane * (unsigned)sizeof(R);
  const int n1 = g.nx;
  const int n2 = DIR == 1 ? g.nz : g.ny;
  const int nd = DIR == 1 ? g.ny : g.nz;
  const int emin = DIR == 1 ? g.eul_jmin : g.eul_kmin;
  const int emax = DIR == 1 ? g.eul_jmax : g.eul_kmax;
  const long long nlines = (long long)n1 * n2;
  // both forms are launched; the one that the list length does not select leaves at once
  if (weno_split<DIR>(g) != SPLIT) return;
  const unsigned tiles = (unsigned)((nlines + 31) / 32);
  const unsigned sgi = blk.x / tiles;
  const long long line = (long long)(blk.x - sgi * tiles) * 32 + lane;
  const bool in = line < nlines;
  const unsigned lu = in ? (unsigned)line : 0u, lb = lu / (unsigned)n1;
  const int i = (int)(lu - lb * (unsigned)n1) + 1;
  const int b = (int)lb + 1;  // k for y lines, j for z lines
  const int c0 = emin + (int)sgi * seglen;
  const int c1 = min(c0 + seglen - 1, emax);
  const long long n = g.nvol, nI = g.nint;
  const long long sd = DIR == 1 ? (long long)g.sx : (long long)g.sx * g.sy;
  const long long base0 = DIR == 1 ? gidx(g, i, 0, b) : gidx(g, i, b, 0);  // address of c = 0
  constexpr unsigned PB = RF * 32 * (unsigned)sizeof(R);  // bytes of a point of the ring
  // points c0-S .. c1+S of the segment's stencils, point c in slot (c - c0 + S) mod nslot, which is
  // s0 for ca; a warp copies a point at a time
  auto fetch = [&](int ca, int cb, int s0) {
    for (int c = ca + wid; c <= cb; c += nw)
      if (in) {
        int sl = s0 + (c - ca);
        if (sl >= nslot) sl -= nslot;
        const unsigned dst = ring_a + sl * PB;
        const R* src = aux + base0 + (long long)c * sd;
#pragma unroll
        for (int q = 0; q < RF; ++q) copy_async(dst + q * 32 * (unsigned)sizeof(R), src + (q == F_C ? 7 : q) * n);
      }
  };
  fetch(c0 - S, min(c0 - 2 + nw + S, c1 + S), 0);
  copy_commit();
  // the sensor flags of the points c0-WS .. c1+WS (word q: point c0-WS+q)
  for (int q = wid; q < c1 - c0 + 1 + 2 * WS; q += nw) {
    int c = c0 - WS + q;
    bool on = in;
    if (c < 1 || c > nd) {
      on = on && g.periodic[DIR];
      c = on ? wrap(c, nd) : 1;
    }
    if (on) on = (DIR == 1 ? sensor[iidx(g, i, c, b)] : sensor[iidx(g, i, b, c)]) > g.sensor_threshold;
    const unsigned bal = __ballot_sync(0xffffffffu, on);
    if (lane == 0) flag[q] = bal;
  }
  double part[5] = {0, 0, 0, 0, 0};
  double f[5] = {0, 0, 0, 0, 0};
  int sr = 0;  // slot of the round's first point, cr - S + 1
  for (int cr = c0 - 1; cr <= c1; cr += nw) {
    const int c = cr + wid;  // this warp's face (between the cells c and c+1)
    const bool face = in && c <= c1;
    const int ep = face ? face_ep<DIR>(g, c) : 0;
    // the next round's points: their slots were last read before the barrier after the fluxes
    {
      int sn = sr + nw + 2 * S - 1;
      if (sn >= nslot) sn -= nslot;
      fetch(cr + nw + S, min(cr + 2 * nw - 1 + S, c1 + S), sn);
    }
    copy_commit();
    copy_wait<1>();
    __syncthreads();  // this round's points and (first round) the flags are there
    if (wid == nw - 1)  // the previous round's last face
#pragma unroll
      for (int m = 0; m < 5; ++m) xch[m * 32 + lane] = f[m];
    Ring<R, 2 * S> ln;
    {
      int sl = sr + wid;
      if (sl >= nslot) sl -= nslot;
#pragma unroll
      for (int q = 0; q < 2 * S; ++q) ln.o[q] = ring_a + (sl + q >= nslot ? sl + q - nslot : sl + q) * PB;
    }
    sr += nw;
    if (sr >= nslot) sr -= nslot;
    if (face) {
      unsigned any = 0;  // points c-WS+1 .. c+WS
#pragma unroll
      for (int q = 0; q < 2 * WS; ++q) any |= flag[c + 1 - c0 + q];
      face_flux<R, DIR, LB, WS, S, FS>(g, ln, (any >> lane) & 1u, c, ep, f, scr, SPLIT, i, b);
    }
    double* own = xch + (wid + 1) * 5 * 32 + lane;
#pragma unroll
    for (int m = 0; m < 5; ++m) own[m * 32] = f[m];
    // what the cell c between the faces c-1 and c adds to, read before the barrier
    const bool cell = face && c >= c0;
    const long long ic = DIR == 1 ? iidx(g, i, c, b) : iidx(g, i, b, c);
    double r[5] = {0, 0, 0, 0, 0}, met = 0;
    R uu = 0, vv = 0, ww = 0, tt0 = 0, rh0 = 0, mu = 0, dv[6] = {0, 0, 0, 0, 0, 0};
    if (cell) {
#pragma unroll
      for (int m = 0; m < 5; ++m) r[m] = fl[m * nI + ic];
      met = DIR == 1 ? g.detady[c] : g.dzitdz[c];
      if constexpr (DIR == 2) {
        mu = __ldg(aux + 6 * n + base0 + (long long)c * sd);
        if (g.conservative_viscous) {
          dv[0] = __ldg(div3 + div3_idx(g, i + 1, b, c));
          dv[1] = __ldg(div3 + div3_idx(g, i - 1, b, c));
          dv[2] = __ldg(div3 + div3_idx(g, i, b + 1, c));
          dv[3] = __ldg(div3 + div3_idx(g, i, b - 1, c));
          dv[4] = __ldg(div3 + div3_idx(g, i, b, c + 1));
          dv[5] = __ldg(div3 + div3_idx(g, i, b, c - 1));
        }
        uu = ln(1, S - 1); vv = ln(2, S - 1); ww = ln(3, S - 1);  // the face's lower point
        if constexpr (CH && sizeof(R) == sizeof(double)) {
          rh0 = ln(0, S - 1);
          tt0 = ln(5, S - 1);
        }
      }
    }
    __syncthreads();
    if (cell) {
      // the lower face: the warp before, or the previous round's last
#pragma unroll
      for (int m = 0; m < 5; ++m) r[m] = r[m] + (f[m] - own[m * 32 - 5 * 32]) * met;
      if (DIR == 2) {
        const int j = b, k = c;
        R sigx, sigy, sigz;
        if (g.conservative_viscous) {
          // mu/(x(i+1)-x(i-1)): in FP64 by the per-line reciprocals, in FP32 the rounded quotient
          R dxl, dyl, dzl;
          if constexpr (sizeof(R) == sizeof(double)) {
            dxl = mu * line_r<R>(g, 0, i); dyl = mu * line_r<R>(g, 1, j); dzl = mu * line_r<R>(g, 2, k);
          } else {
            dxl = mu / R(g.x[i + 1] - g.x[i - 1]);
            dyl = mu / R(g.y[j + 1] - g.y[j - 1]);
            dzl = mu / R(g.z[k + 1] - g.z[k - 1]);
          }
          sigx = dxl * (dv[0] - dv[1]);
          sigy = dyl * (dv[2] - dv[3]);
          sigz = dzl * (dv[4] - dv[5]);
        } else {
          // visflx_div_subroutine (kernels_cpu.F90:3484-3532): order visc_order
          const int lv = g.lmax_base;
          R dx3 = R(0), dy3 = R(0), dz3 = R(0);
          for (int l = 1; l <= lv; ++l) {
            const R ccl = R(g.coeff[lv - 1][l - 1]);
            dx3 = dx3 + ccl * (div3_at(g, div3, i + l, j, k) - div3_at(g, div3, i - l, j, k));
            dy3 = dy3 + ccl * (div3_at(g, div3, i, j + l, k) - div3_at(g, div3, i, j - l, k));
            dz3 = dz3 + ccl * (div3_at(g, div3, i, j, k + l) - div3_at(g, div3, i, j, k - l));
          }
          sigx = mu * (dx3 * R(g.dcsidx[i]));
          sigy = mu * (dy3 * R(g.detady[j]));
          sigz = mu * (dz3 * R(g.dzitdz[k]));
        }
        const R sigq = sigx * uu + sigy * vv + sigz * ww;
        r[1] = r[1] - double(sigx);
        r[2] = r[2] - double(sigy);
        r[3] = r[3] - double(sigz);
        r[4] = r[4] - double(sigq);
        if constexpr (CH) {
          const double dt = sc->dt;
          const double rhodt = rhork * dt, gamdt = gamrk * dt;
          const double fln1 = (istep > 1 ? -(rhodt * fl_prev[ic]) : 0.0) - gamdt * r[0];
          const double fln2 = (istep > 1 ? -(rhodt * fl_prev[nI + ic]) : 0.0) - gamdt * r[1];
          const double dy = g.yn[j + 1] - g.yn[j];
          // density, momentum and temperature of the stage's state: the ring's in FP64, else from w
          double rho, rhou, tt;
          if constexpr (sizeof(R) == sizeof(double)) {
            rho = rh0;
            rhou = rho * uu;
            tt = tt0;
          } else {
            const long long a = base0 + (long long)c * sd;
            const Prim pr = prim_from_w<false>(g, w, a, g.t0);
            rho = pr.rho;
            rhou = w[n + a];
            tt = pr.tt;
          }
          part[0] += fln1 * dy;
          part[1] += fln2 * dy;
          part[2] += rho * dy;
          part[3] += rhou * dy;
          part[4] += rhou * dy * tt;
        }
      }
#pragma unroll
      for (int m = 0; m < 5; ++m) fl[m * nI + ic] = r[m];
    }
  }
  if constexpr (DIR == 2 && CH) {
    // lanes, then the block's warps in order (the flux exchange is done with: reuse it)
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part[r] += __shfl_down_sync(0xffffffffu, part[r], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
      for (int r = 0; r < 5; ++r) xch[r * 32 + wid] = part[r];
    __syncthreads();
    if (threadIdx.x < 5) {
      double a = 0.0;
      for (int q = 0; q < nw; ++q) a += xch[threadIdx.x * 32 + q];
      red[(long long)blk.x * 5 + threadIdx.x] = a;
    }
  }
}
template <class R, int DIR, int LB, int WS, bool CH = false, int FS = 0, bool SPLIT = false>
__global__ void __launch_bounds__(march_maxt<R, LB, FS>(), 1) k_march(Geom g, const R* __restrict__ aux,
                                                 const double* __restrict__ sensor, double* __restrict__ fl,
                                                 const R* __restrict__ div3,
                                                 const double* __restrict__ w, const double* __restrict__ fl_prev,
                                                 const Scalars* __restrict__ sc, double rhork, double gamrk,
                                                 int istep, int seglen, double* __restrict__ red) {
  d_march<R, DIR, LB, WS, CH, FS, SPLIT>(g, aux, sensor, fl, div3, w, fl_prev, sc, rhork, gamrk, istep, seglen, red, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// The viscous pass: visflx_reduced_ord2_subroutine (kernels_cpu.F90:4623-4721, update_sensor = 0)
// followed by visflx_x/y/z_subroutine (:4779-4999); at stage 3 also sensor_subroutine (:4726-4744)
// into the next sensor buffer.  Arithmetic in R, accumulation into the FP64 register.
// A block of 32 x 8 threads owns a 32 x 8 column of cells and marches vk cells along z; the five
// fields the pass reads (u, v, w, T, mu) sit in a ring of four tiles of 34 x 10 points (the column and
// its x / y halo): the planes k-1, k, k+1 that the cells of plane k read, and k+2, which is copied
// (cp.async, with the cells' fl of the next plane) while plane k is computed.  Every point is loaded
// once per block, the x / y / z neighbours come from shared memory, the flux of a cell's upper z face
// is the next cell's lower one, and the grid's and the gas's quotients come from tables and constants
// of the context: of the divisions of a cell (6 by face distances, 6 by the Prandtl number, one by
// 3) none is left.
// 1024x256x192 boundary layer, FP64: 7.4 -> 4.2 ms per step (its 112 algorithmic bytes a cell take
// 2.5 at the copy rate); 1024x256x128 mixed: 3.4 -> 2.1; a 32x24x16 channel, whose segments were
// 16 cells: 57 -> 9 us a pass.
constexpr int VT_X = 32, VT_Y = 8, VT_NT = VT_X * VT_Y, VT_KMAX = 16;
constexpr int VT_PX = VT_X + 2, VT_PY = VT_Y + 2, VT_PP = VT_PX * VT_PY;
template <class R>
constexpr size_t visc_smem() { return (size_t)VT_NT * 4 * 8 + (size_t)4 * 5 * VT_PP * sizeof(R); }
// blocks: 32 x 8 columns x segments of vk cells in z, VT_KMAX of them (two more planes are loaded per
// segment) or as few as give each SM three blocks (two are resident in FP64, four in FP32)
inline int visc_k(const Geom& g) {
  const long long tiles = (long long)((g.nx + VT_X - 1) / VT_X) * ((g.ny + VT_Y - 1) / VT_Y);
  return (int)std::min<long long>(VT_KMAX, std::max<long long>(1, tiles * g.nz / (148 * 3)));
}
inline unsigned visc_tiled_blocks(const Geom& g) {
  const int vk = visc_k(g);
  return (unsigned)((g.nx + VT_X - 1) / VT_X) * (unsigned)((g.ny + VT_Y - 1) / VT_Y) * (unsigned)((g.nz + vk - 1) / vk);
}
template <class R, bool TP = false>
__device__ __forceinline__ void d_visc_tiled(const Geom& g, const R* __restrict__ aux, double* __restrict__ fl,
                                             R* __restrict__ div3, double* __restrict__ sensor_next,
                                             double* __restrict__ wallprop, int do_sensor, int vk, const Blk blk) {
  extern __shared__ __align__(16) unsigned char sb_dyn_smem[];
  double* flb = reinterpret_cast<double*>(sb_dyn_smem) + threadIdx.x;  // this thread's fl(2:5), VT_NT apart
  R* pl = reinterpret_cast<R*>(sb_dyn_smem + VT_NT * 4 * 8);           // [4][5][VT_PP]
  const unsigned nbx = (unsigned)(g.nx + VT_X - 1) / VT_X, nby = (unsigned)(g.ny + VT_Y - 1) / VT_Y;
  const unsigned bx = blk.x % nbx, rest = blk.x / nbx, by = rest % nby, bk = rest / nby;
  const int tx = (int)threadIdx.x % VT_X, ty = (int)threadIdx.x / VT_X;
  const int i0 = (int)bx * VT_X, j0 = (int)by * VT_Y;  // the tile's points are i0 .. i0+VT_X+1
  const int i = i0 + 1 + tx, j = j0 + 1 + ty;
  const bool own = i <= g.nx && j <= g.ny;
  const int k0 = (int)bk * vk + 1, k1 = min(k0 + vk - 1, g.nz);
  const long long n = g.nvol, nI = g.nint, sZ = (long long)g.sx * g.sy, cz = (long long)g.nx * g.ny;
  // this thread's points of a tile: t = threadIdx.x and t + VT_NT (points beyond the face ghosts are
  // left unread: no cell of the column uses them)
  const int t1 = threadIdx.x + VT_NT;
  const int ia = i0 + (int)threadIdx.x % VT_PX, ja = j0 + (int)threadIdx.x / VT_PX;
  const int ib = i0 + t1 % VT_PX, jb = j0 + t1 / VT_PX;
  const bool ga = ia <= g.nx + 1 && ja <= g.ny + 1, gb = t1 < VT_PP && ib <= g.nx + 1 && jb <= g.ny + 1;
  const R* pa = aux + n + gidx(g, ia, ja, 0);
  const long long dab = gidx(g, ib, jb, 0) - gidx(g, ia, ja, 0);
  const unsigned da = (unsigned)__cvta_generic_to_shared(pl + threadIdx.x);
  auto load_plane = [&](int k) {
    const unsigned d = da + (k & 3) * (unsigned)(5 * VT_PP * sizeof(R));
    const R* s = pa + k * sZ;
#pragma unroll
    for (int f = 0; f < 5; ++f) {  // u, v, w, T, mu
      const R* q = s + (f < 3 ? f : f + 1) * n;
      if (ga) copy_async(d + f * (unsigned)(VT_PP * sizeof(R)), q);
      if (gb) copy_async(d + (f * VT_PP + VT_NT) * (unsigned)sizeof(R), q + dab);
    }
  };
  const long long q0 = own ? iidx(g, i, j, 0) : 0;  // interior index of the column's plane 0
  auto load_fl = [&](int k) {
    if (own)
#pragma unroll
      for (int m = 0; m < 4; ++m)
        copy_async((unsigned)__cvta_generic_to_shared(flb + m * VT_NT), fl + (m + 1) * nI + q0 + k * cz);
  };
  load_plane(k0 - 1);
  load_plane(k0);
  load_plane(k0 + 1);
  load_fl(k0);
  copy_commit();
  const R cpp = R(g.cpp), rpr = sizeof(R) == sizeof(double) ? R(g.rpr) : R(1) / R(g.prandtl);
  R zlo[4] = {R(0), R(0), R(0), R(0)};  // flux of the lower z face
  for (int k = k0; k <= k1; ++k) {
    copy_wait<0>();
    __syncthreads();  // plane k+1 is there, and every thread is done with plane k-2
    double f2 = flb[0], f3 = flb[VT_NT], f4 = flb[2 * VT_NT], f5 = flb[3 * VT_NT];
    if (k < k1) {
      load_plane(k + 2);
      load_fl(k + 1);
    }
    copy_commit();
    if (own) {
      const R* pm = pl + ((k - 1) & 3) * 5 * VT_PP + (tx + 1) + (ty + 1) * VT_PX;
      const R* p0 = pl + (k & 3) * 5 * VT_PP + (tx + 1) + (ty + 1) * VT_PX;
      const R* pp = pl + ((k + 1) & 3) * 5 * VT_PP + (tx + 1) + (ty + 1) * VT_PX;
      // field f (0 u, 1 v, 2 w, 3 T, 4 mu) at the point o of a plane
      auto F = [&](const R* p, int o, int f) -> R { return p[f * VT_PP + o]; };
      const long long q = q0 + k * cz;
      const R dxl = line_r<R>(g, 0, i), dyl = line_r<R>(g, 1, j), dzl = line_r<R>(g, 2, k);
      const R c0[5] = {F(p0, 0, 0), F(p0, 0, 1), F(p0, 0, 2), F(p0, 0, 3), F(p0, 0, 4)};
      const R qc = R(0.5) * (c0[0] * c0[0] + c0[1] * c0[1] + c0[2] * c0[2]);
      // conservative face Laplacian: flux at the face between the cell and its neighbour o of plane
      // p at distance 1/rd, for the cell below (sgn = 1) or above (-1) the face
      auto face = [&](const R* p, int o, const Quot<R>& rd, R sgn, R (&s)[4]) {
        const R u = F(p, o, 0), v = F(p, o, 1), w = F(p, o, 2), t = F(p, o, 3);
        const R muf = quot(R(0.5) * (F(p, o, 4) + c0[4]), rd) * sgn;
        const R qn = R(0.5) * (u * u + v * v + w * w);
        s[0] = (u - c0[0]) * muf;
        s[1] = (v - c0[1]) * muf;
        s[2] = (w - c0[2]) * muf;
        R heat;  // (T - T0) cp/Pr
        if constexpr (TP) heat = (t - c0[3]) * (R(cp_of_t(g, double(R(0.5) * (t + c0[3])))) * rpr);
        else if constexpr (sizeof(R) == sizeof(double)) heat = (t - c0[3]) * cpp;
        else heat = quot((t - c0[3]) * R(g.cp0), Quot<R>{R(g.prandtl), rpr});
        s[3] = (heat + (qn - qc)) * muf;
      };
      R lo[4], hi[4];
      // x: fl += dxhl*(fhat(i) - fhat(i-1)), fhat = -sigma
      face(p0, -1, face_r<R>(g, 0, i - 1), R(-1), lo);
      face(p0, 1, face_r<R>(g, 0, i), R(1), hi);
      const double dxhl = __ldg(g.vhl[0] + i);
      f2 = f2 + dxhl * (double(lo[0]) - double(hi[0]));
      f3 = f3 + dxhl * (double(lo[1]) - double(hi[1]));
      f4 = f4 + dxhl * (double(lo[2]) - double(hi[2]));
      f5 = f5 + dxhl * (double(lo[3]) - double(hi[3]));
      face(p0, -VT_PX, face_r<R>(g, 1, j - 1), R(-1), lo);
      face(p0, VT_PX, face_r<R>(g, 1, j), R(1), hi);
      const double dyhl = __ldg(g.vhl[1] + j);
      f2 = f2 + dyhl * (double(lo[0]) - double(hi[0]));
      f3 = f3 + dyhl * (double(lo[1]) - double(hi[1]));
      f4 = f4 + dyhl * (double(lo[2]) - double(hi[2]));
      f5 = f5 + dyhl * (double(lo[3]) - double(hi[3]));
      if (k == k0) face(pm, 0, face_r<R>(g, 2, k - 1), R(-1), zlo);
      face(pp, 0, face_r<R>(g, 2, k), R(1), hi);
      const double dzhl = __ldg(g.vhl[2] + k);
      f2 = f2 + dzhl * (double(zlo[0]) - double(hi[0]));
      f3 = f3 + dzhl * (double(zlo[1]) - double(hi[1]));
      f4 = f4 + dzhl * (double(zlo[2]) - double(hi[2]));
      f5 = f5 + dzhl * (double(zlo[3]) - double(hi[3]));
#pragma unroll
      for (int m = 0; m < 4; ++m) zlo[m] = hi[m];
      // reduced second-order terms
      R ux = dxl * (F(p0, 1, 0) - F(p0, -1, 0));
      R vx = dxl * (F(p0, 1, 1) - F(p0, -1, 1));
      R wx = dxl * (F(p0, 1, 2) - F(p0, -1, 2));
      R mux = dxl * (F(p0, 1, 4) - F(p0, -1, 4));
      R uy = dyl * (F(p0, VT_PX, 0) - F(p0, -VT_PX, 0));
      R vy = dyl * (F(p0, VT_PX, 1) - F(p0, -VT_PX, 1));
      R wy = dyl * (F(p0, VT_PX, 2) - F(p0, -VT_PX, 2));
      R muy = dyl * (F(p0, VT_PX, 4) - F(p0, -VT_PX, 4));
      R uz = dzl * (F(pp, 0, 0) - F(pm, 0, 0));
      R vz = dzl * (F(pp, 0, 1) - F(pm, 0, 1));
      R wz = dzl * (F(pp, 0, 2) - F(pm, 0, 2));
      R muz = dzl * (F(pp, 0, 4) - F(pm, 0, 4));
      if (j == 1) {
        const R ty_ = dyl * (F(p0, VT_PX, 3) - F(p0, -VT_PX, 3));
        const R cploc = TP ? R(cp_of_t(g, double(c0[3]))) : R(g.cp0);
        const long long wp = (long long)(k - 1) * g.nx + (i - 1);
        const long long nw = (long long)g.nx * g.nz;
        wallprop[wp] = double(c0[4] * uy);
        wallprop[nw + wp] = double(c0[4] * wy);
        wallprop[2 * nw + wp] = double(c0[4] * ty_ * cploc / R(g.prandtl));
      }
      R div;  // with the rounding of the mixed form fixed: du/dx fused with the first sum only
      if constexpr (sizeof(R) == sizeof(double)) div = ux + vy + wz;
      else div = __fadd_rn(__fmaf_rn(dxl, F(p0, 1, 0) - F(p0, -1, 0), vy), wz);
      const R div3l = quot(div, Quot<R>{R(3), R(1.0 / 3.0)});
      div3[q] = div3l;
      if (do_sensor) {
        // sensor_subroutine works from the stored |omega| and div/3
        const R omegax = wy - vz, omegay = uz - wx, omegaz = vx - uy;
        const R om = sqrt(omegax * omegax + omegay * omegay + omegaz * omegaz);
        const R om2 = om * om;
        const R dv = R(3) * div3l;
        const R u0l0 = R(g.u0 / g.l0);
        const R t = fmax(-dv / sqrt(om2 + dv * dv + u0l0 * u0l0), R(0));
        sensor_next[q] = double(t * t);
      }
      const R sig11 = ux - R(2) * div3l, sig12 = vx, sig13 = wx;
      const R sig21 = uy, sig22 = vy - R(2) * div3l, sig23 = wy;
      const R sig31 = uz, sig32 = vz, sig33 = wz - R(2) * div3l;
      const R sigx = mux * sig11 + muy * sig12 + muz * sig13;
      const R sigy = mux * sig21 + muy * sig22 + muz * sig23;
      const R sigz = mux * sig31 + muy * sig32 + muz * sig33;
      const R sigah = (sig11 * ux + sig12 * uy + sig13 * uz + sig21 * vx + sig22 * vy + sig23 * vz + sig31 * wx +
                       sig32 * wy + sig33 * wz) * c0[4];
      const R sigq = sigx * c0[0] + sigy * c0[1] + sigz * c0[2] + sigah;
      fl[nI + q] = f2 - double(sigx);
      fl[2 * nI + q] = f3 - double(sigy);
      fl[3 * nI + q] = f4 - double(sigz);
      fl[4 * nI + q] = f5 - double(sigq);
    }
  }
}
template <class R, bool TP = false>
__global__ void __launch_bounds__(VT_NT, sizeof(R) == 8 ? VISC_MINB : VISC_MINB_F)
    k_visc_tiled(Geom g, const R* __restrict__ aux, double* __restrict__ fl, R* __restrict__ div3,
                 double* __restrict__ sensor_next, double* __restrict__ wallprop, int do_sensor, int vk) {
  d_visc_tiled<R, TP>(g, aux, fl, div3, sensor_next, wallprop, do_sensor, vk, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// visflx_nosensor_subroutine (kernels_cpu.F90:3996-4180), the non-conservative viscous form of
// conservative_viscous = 0: first and second derivatives of u, v, w, T (and first of mu) with the
// central stencil of order visc_order, the full stress divergence and dissipation, heat flux;
// div/3 and |omega| for the div term and the stage-3 sensor (sensor_subroutine,
// kernels_cpu.F90:4726-4744, from |omega| and div/3), wall shear at j = 1.  Arithmetic in R,
// accumulation into the FP64 register.
template <class R, bool TP = false>
__device__ __forceinline__ void d_visc_ns(const Geom& g, const R* __restrict__ aux, double* __restrict__ fl,
                                                 R* __restrict__ div3, double* __restrict__ sensor_next,
                                                 double* __restrict__ wallprop, int do_sensor, const Blk blk) {
  const long long q = (long long)blk.x * 256 + threadIdx.x;
  if (q >= g.nint) return;
  int i, j, k;
  cell_of(g, q, i, j, k);
  const long long n = g.nvol, nI = g.nint;
  const long long c = gidx(g, i, j, k);
  const long long st[3] = {1, g.sx, (long long)g.sx * g.sy};
  auto A = [&](long long a, int m) -> R { return __ldg(aux + (m - 1) * n + a); };
  const int lmax = g.lmax_base;
  const R uu = A(c, 2), vv = A(c, 3), ww = A(c, 4), tt = A(c, 6), mu = A(c, 7);
  // d[dir][var]: first derivative of u, v, w, T, mu; lap[dir][var]: second derivative of u, v, w, T
  R d1[3][5], lap[3][4];
  const R c20 = R(g.coeff2[lmax - 1][0]);
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
#pragma unroll
    for (int v = 0; v < 5; ++v) d1[dir][v] = R(0);
    lap[dir][0] = c20 * uu; lap[dir][1] = c20 * vv; lap[dir][2] = c20 * ww; lap[dir][3] = c20 * tt;
    for (int l = 1; l <= lmax; ++l) {
      const R ccl = R(g.coeff[lmax - 1][l - 1]);
      const R clapl = R(g.coeff2[lmax - 1][l]);
      const long long ap = c + l * st[dir], am = c - l * st[dir];
      const int ms[5] = {2, 3, 4, 6, 7};
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const R fp = A(ap, ms[v]), fm = A(am, ms[v]);
        d1[dir][v] = d1[dir][v] + ccl * (fp - fm);
        if (v < 4) lap[dir][v] = lap[dir][v] + clapl * (fp + fm);
      }
    }
  }
  const R m1[3] = {R(g.dcsidx[i]), R(g.detady[j]), R(g.dzitdz[k])};
  const R ms2[3] = {R(g.dcsidxs[i]), R(g.detadys[j]), R(g.dzitdzs[k])};
  const R m2[3] = {R(g.dcsidx2[i]), R(g.detady2[j]), R(g.dzitdz2[k])};
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
#pragma unroll
    for (int v = 0; v < 5; ++v) d1[dir][v] = d1[dir][v] * m1[dir];
#pragma unroll
    for (int v = 0; v < 4; ++v) lap[dir][v] = lap[dir][v] * ms2[dir] + d1[dir][v] * m2[dir];
  }
  const R ux = d1[0][0], vx = d1[0][1], wx = d1[0][2], tx = d1[0][3], mux = d1[0][4];
  const R uy = d1[1][0], vy = d1[1][1], wy = d1[1][2], ty = d1[1][3], muy = d1[1][4];
  const R uz = d1[2][0], vz = d1[2][1], wz = d1[2][2], tz = d1[2][3], muz = d1[2][4];
  const R ulap = lap[0][0] + lap[1][0] + lap[2][0];
  const R vlap = lap[0][1] + lap[1][1] + lap[2][1];
  const R wlap = lap[0][2] + lap[1][2] + lap[2][2];
  const R tlap = lap[0][3] + lap[1][3] + lap[2][3];
  const R div = ux + vy + wz;
  const R div3l = div / R(3);
  div3[q] = div3l;
  const R omegax = wy - vz, omegay = uz - wx, omegaz = vx - uy;
  const R omod2 = omegax * omegax + omegay * omegay + omegaz * omegaz;
  if (do_sensor) {
    const R om = sqrt(omod2);
    const R om2 = om * om;
    const R dv = R(3) * div3l;
    const R u0l0 = R(g.u0 / g.l0);
    const R t = fmax(-dv / sqrt(om2 + dv * dv + u0l0 * u0l0), R(0));
    sensor_next[q] = double(t * t);
  }
  const R cploc = TP ? R(cp_of_t(g, double(A(c, 6)))) : R(g.cp0), prandtl = R(g.prandtl);
  const R sig11 = R(2) * (ux - div3l), sig12 = uy + vx, sig13 = uz + wx;
  const R sig22 = R(2) * (vy - div3l), sig23 = vz + wy, sig33 = R(2) * (wz - div3l);
  const R sigx = mux * sig11 + muy * sig12 + muz * sig13 + mu * ulap;
  const R sigy = mux * sig12 + muy * sig22 + muz * sig23 + mu * vlap;
  const R sigz = mux * sig13 + muy * sig23 + muz * sig33 + mu * wlap;
  const R sigqt = (mux * tx + muy * ty + muz * tz + mu * tlap) * cploc / prandtl;
  const R sigah = (sig11 * ux + sig12 * uy + sig13 * uz + sig12 * vx + sig22 * vy + sig23 * vz + sig13 * wx +
                   sig23 * wy + sig33 * wz) * mu;
  const R sigq = sigx * uu + sigy * vv + sigz * ww + sigah + sigqt;
  fl[nI + q] = fl[nI + q] - double(sigx);
  fl[2 * nI + q] = fl[2 * nI + q] - double(sigy);
  fl[3 * nI + q] = fl[3 * nI + q] - double(sigz);
  fl[4 * nI + q] = fl[4 * nI + q] - double(sigq);
  if (j == 1) {
    const long long wp = (long long)(k - 1) * g.nx + (i - 1);
    const long long nw = (long long)g.nx * g.nz;
    wallprop[wp] = double(mu * uy);
    wallprop[nw + wp] = double(mu * wy);
    wallprop[2 * nw + wp] = double(mu * ty * cploc / prandtl);
  }
}
template <class R, bool TP = false>
__global__ void __launch_bounds__(256) k_visc_ns(Geom g, const R* __restrict__ aux, double* __restrict__ fl,
                                                 R* __restrict__ div3, double* __restrict__ sensor_next,
                                                 double* __restrict__ wallprop, int do_sensor) {
  d_visc_ns<R, TP>(g, aux, fl, div3, sensor_next, wallprop, do_sensor, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// Initial Ducros sensor of run() (visflx(mode=2), singleideal_cpu.F90:1550-1555):
// visflx_reduced_ord2 with update_sensor = 1 (kernels_cpu.F90:4680-4682)
template <class R>
__device__ __forceinline__ void d_init_sensor(const Geom& g, const R* __restrict__ aux,
                                                     double* __restrict__ sensor, const Blk blk) {
  const long long q = (long long)blk.x * 256 + threadIdx.x;
  if (q >= g.nint) return;
  int i, j, k;
  cell_of(g, q, i, j, k);
  const long long n = g.nvol, c = gidx(g, i, j, k), sY = g.sx, sZ = (long long)g.sx * g.sy;
  auto A = [&](long long a, int m) -> R { return aux[(m - 1) * n + a]; };
  R dxl = R(1) / R(g.x[i + 1] - g.x[i - 1]);
  R dyl = R(1) / R(g.y[j + 1] - g.y[j - 1]);
  R dzl = R(1) / R(g.z[k + 1] - g.z[k - 1]);
  R ux = dxl * (A(c + 1, 2) - A(c - 1, 2));
  R vx = dxl * (A(c + 1, 3) - A(c - 1, 3));
  R wx = dxl * (A(c + 1, 4) - A(c - 1, 4));
  R uy = dyl * (A(c + sY, 2) - A(c - sY, 2));
  R vy = dyl * (A(c + sY, 3) - A(c - sY, 3));
  R wy = dyl * (A(c + sY, 4) - A(c - sY, 4));
  R uz = dzl * (A(c + sZ, 2) - A(c - sZ, 2));
  R vz = dzl * (A(c + sZ, 3) - A(c - sZ, 3));
  R wz = dzl * (A(c + sZ, 4) - A(c - sZ, 4));
  R div = ux + vy + wz;
  R omegax = wy - vz, omegay = uz - wx, omegaz = vx - uy;
  R omod2 = omegax * omegax + omegay * omegay + omegaz * omegaz;
  R u0l0 = R(g.u0 / g.l0);
  R t = fmax(-div / sqrt(omod2 + div * div + u0l0 * u0l0), R(0));
  sensor[q] = double(t * t);
}
template <class R>
__global__ void __launch_bounds__(256) k_init_sensor(Geom g, const R* __restrict__ aux,
                                                     double* __restrict__ sensor) {
  d_init_sensor<R>(g, aux, sensor, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// The time step where the aux pass does not run (aux is current): block maxima of the inverse time
// scales.  The FP64 form reads the primitive fields; the mixed form recomputes them from w in FP64.
template <class R>
__device__ __forceinline__ void d_dt(const Geom& g, const double* __restrict__ w, const R* __restrict__ aux,
                                            double* __restrict__ red, const Blk blk) {
  double m = 0.0;
#pragma unroll 1
  for (int cq = 0; cq < PT_CELLS; ++cq) {
    const long long q = (long long)blk.x * (256 * PT_CELLS) + cq * 256 + threadIdx.x;
    if (q >= g.nint) break;
    int i, j, k;
    cell_of(g, q, i, j, k);
    const long long n = g.nvol, c = gidx(g, i, j, k);
    const double ri = rcp_pos(w[c]);
    double uu, vv, ww, tt, mu;
    if constexpr (sizeof(R) == sizeof(double)) {
      uu = aux[n + c]; vv = aux[2 * n + c]; ww = aux[3 * n + c]; tt = aux[5 * n + c]; mu = aux[6 * n + c];
    } else {
      const Prim p = prim_from_w<false>(g, w, c, g.t0);  // mixed form only: calorically perfect
      uu = p.uu; vv = p.vv; ww = p.ww; tt = p.tt; mu = viscosity(g, tt);
    }
    const double cs = sqrt(gamloc_of_t(g, tt) * g.rgas0 * tt);
    m = fmax(m, inverse_dt(g, i, j, k, uu, vv, ww, cs, ri * mu));
  }
  block_max(m, red + blk.x);
}
template <class R>
__global__ void __launch_bounds__(256, DT_MINB) k_dt(Geom g, const double* __restrict__ w, const R* __restrict__ aux,
                                            double* __restrict__ red) {
  d_dt<R>(g, w, aux, red, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

__device__ __forceinline__ void d_dt_finish(const double* __restrict__ red, long long nblk, double cfl,
                                                      Scalars* __restrict__ sc, const Blk blk) {
  __shared__ double sm[FIN_NT / 32];
  double m = 0.0;
  for (long long b = threadIdx.x; b < nblk; b += FIN_NT) m = fmax(m, red[b]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    for (int wq = 0; wq < FIN_NT / 32; ++wq) a = fmax(a, sm[wq]);
    double dt_min = 1.0 / a;
    sc->dt = cfl * dt_min;
  }
}
__global__ void __launch_bounds__(FIN_NT) k_dt_finish(const double* __restrict__ red, long long nblk, double cfl,
                                                      Scalars* __restrict__ sc) {
  d_dt_finish(red, nblk, cfl, sc, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// Sum NR partials per block in a fixed order (thread-strided, then tree).
template <int NR>
__device__ __forceinline__ void finish_sums(const double* __restrict__ red, long long nblk, double (&out)[NR],
                                            double* sm) {
  double v[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) v[r] = 0.0;
  for (long long b = threadIdx.x; b < nblk; b += FIN_NT)
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = v[r] + red[b * NR + r];
  block_reduce_sum<NR, FIN_NT>(v, sm);
#pragma unroll
  for (int r = 0; r < NR; ++r) out[r] = v[r];
}

// force_rhs (singleideal_cpu.F90:845-889): bulk values from the partials
__device__ __forceinline__ void d_finish_rhs(const Geom& g, const double* __restrict__ red, long long nblk,
                                                       int first_stage, Scalars* __restrict__ sc, const Blk blk) {
  __shared__ double sm[5 * (FIN_NT / 32)];
  double b[5];
  finish_sums<5>(red, nblk, b, sm);
  if (threadIdx.x == 0) {
    for (int r = 0; r < 5; ++r) b[r] = b[r] / g.volchan;
    double dpdx = first_stage ? 0.0 : sc->dpdx;
    sc->dpdx = dpdx + b[1];
    sc->rhobulk = b[2];
    sc->ubulk = b[3] / sc->rhobulk;
    sc->tbulk = b[4] / sc->rhobulk / sc->ubulk;
    for (int r = 0; r < 5; ++r) sc->bulk[r] = b[r];
  }
}
__global__ void __launch_bounds__(FIN_NT) k_finish_rhs(Geom g, const double* __restrict__ red, long long nblk,
                                                       int first_stage, Scalars* __restrict__ sc) {
  d_finish_rhs(g, red, nblk, first_stage, sc, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// update_flux + force_rhs_2 + update_field (kernels_cpu.F90:3400-3442, 3092-3116) and the
// partials of force_var_1 (:3241-3282) and of compute_residual / minmax (:6682-6810).  All FP64;
// the primitive values of the stage's starting state are recomputed from w as eval_aux does.
// MODE: 0 the update alone, 1 with the bulk temperature's partials (force_var), 2 with the residual
// and extrema too (the last stage of a step).  Memory bound (160 bytes a cell) while the registers
// hold a cell's loads: a pass with what its stage needs only spills 8, 28 and 44 bytes (MODE 0, 1, 2; the
// thermally perfect gas 8, 108 and 284) at 32 registers where one for all spilled 48 and loaded w twice
// (1024x256x192 4.54 -> 4.14 ms per step, 512x256x256 channel 4.14 -> 2.97).  The quotients stay divisions: the series of rcp_pos keeps more
// values alive (4.93 and 3.56 ms).
template <class R, bool TP, int MODE>
__device__ __forceinline__ void d_update(const Geom& g, double* __restrict__ w, const double* __restrict__ fl_prev,
                                                const double* __restrict__ fl_new, const Scalars* __restrict__ sc,
                                                double rhork, double gamrk, int istep,
                                                double* __restrict__ red, const double* __restrict__ sensor_next,
                                                double* __restrict__ sensor, R* __restrict__ aux, const Blk blk) {
  double sv = 0.0, sr = 0.0;
  double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX};
  double mx[3] = {-100.0, -100.0, -100.0};
  const long long q = (long long)blk.x * UPD_NT + threadIdx.x;
  if (q < g.nint) {
    int i, j, k;
    cell_of(g, q, i, j, k);
    const long long n = g.nvol, nI = g.nint, c = gidx(g, i, j, k);
    const double dt = sc->dt;
    const double rhodt = rhork * dt, gamdt = gamrk * dt;
    // the stage's starting temperature is in aux (Newton start of the thermally perfect gas)
    const double t_aux = TP ? double(aux[5 * n + c]) : g.t0;
    double wo[5], wn[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) wo[m] = w[m * n + c];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double a = istep > 1 ? -(rhodt * fl_prev[m * nI + q]) : 0.0;
      wn[m] = a - gamdt * fl_new[m * nI + q];  // fln
    }
    if (g.channel_case) {
      const double b1 = sc->bulk[0], b2 = sc->bulk[1];
      wn[0] = wn[0] - b1;
      wn[1] = wn[1] - b2;
      wn[4] = wn[4] - wo[1] * (1.0 / wo[0]) * b2;
    }
    const double fln1 = wn[1];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      wn[m] = wo[m] + wn[m];
      w[m * n + c] = wn[m];
    }
    // the stage-3 sensor becomes current once every flux of the stage has used the old one
    if (istep == 3) sensor[q] = sensor_next[q];
    // temperature of a state
    auto temp = [&](const double (&s)[5]) {
      const double ri = 1.0 / s[0];
      const double uu = s[1] * ri, vv = s[2] * ri, ww = s[3] * ri;
      return t_from_e<TP>(g, s[4] * ri - 0.5 * (uu * uu + vv * vv + ww * ww), t_aux);
    };
    double tt = 0.0;
    if (MODE >= 1 && g.force_var) {
      tt = temp(wn);
      sv = wn[1] * tt * (g.yn[j + 1] - g.yn[j]);
      // force_var_1 leaves this temperature in w_aux(6), where the statistics read it
      if (istep == 3) aux[5 * n + c] = R(tt);
    }
    if constexpr (MODE == 2) {
      if (!g.force_var) tt = temp(wo);
      const double r = fln1 / dt;
      sr = r * r;
      const double pp = wo[0] * tt * g.rgas0;
      mn[0] = mx[0] = wo[0];
      mn[1] = mx[1] = tt;
      mn[2] = mx[2] = pp;
    }
  }
  if constexpr (MODE == 0) return;
  constexpr int NW = UPD_NT / 32;
  __shared__ double sm[2 * NW], smn[3 * NW], smx[3 * NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* o = red + (long long)blk.x * NRED_UPD;
  if constexpr (MODE == 1) {
    double s1[1] = {sv};
    block_reduce_sum<1, UPD_NT>(s1, sm);
    if (threadIdx.x == 0) o[0] = s1[0];
    return;
  }
  double s2[2] = {sv, sr};
  block_reduce_sum<2, UPD_NT>(s2, sm);
  // min / max (exact, order independent)
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int of = 16; of > 0; of >>= 1) {
      mn[r] = fmin(mn[r], __shfl_down_sync(0xffffffffu, mn[r], of));
      mx[r] = fmax(mx[r], __shfl_down_sync(0xffffffffu, mx[r], of));
    }
  if (lane == 0)
#pragma unroll
    for (int r = 0; r < 3; ++r) { smn[r * NW + warp] = mn[r]; smx[r * NW + warp] = mx[r]; }
  __syncthreads();
  if (threadIdx.x == 0) {
    o[0] = s2[0];
    o[1] = s2[1];
    for (int r = 0; r < 3; ++r) {
      double a = DBL_MAX, b = -100.0;
      for (int wq = 0; wq < NW; ++wq) { a = fmin(a, smn[r * NW + wq]); b = fmax(b, smx[r * NW + wq]); }
      o[2 + r] = a;
      o[5 + r] = b;
    }
  }
}
template <class R, bool TP, int MODE>
__global__ void __launch_bounds__(UPD_NT, UPD_MINB) k_update(Geom g, double* __restrict__ w, const double* __restrict__ fl_prev,
                                                const double* __restrict__ fl_new, const Scalars* __restrict__ sc,
                                                double rhork, double gamrk, int istep,
                                                double* __restrict__ red, const double* __restrict__ sensor_next,
                                                double* __restrict__ sensor, R* __restrict__ aux) {
  d_update<R, TP, MODE>(g, w, fl_prev, fl_new, sc, rhork, gamrk, istep, red, sensor_next, sensor, aux, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

// force_var (singleideal_cpu.F90:890-933): energy shift for the next pass; residual and extrema
__device__ __forceinline__ void d_finish_upd(const Geom& g, const double* __restrict__ red, long long nblk,
                                                       int stats, int add_time, Scalars* __restrict__ sc, const Blk blk) {
  __shared__ double sm[2 * (FIN_NT / 32)];
  __shared__ double smn[3 * (FIN_NT / 32)], smx[3 * (FIN_NT / 32)];
  double v[2] = {0.0, 0.0};
  double mn[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, mx[3] = {-100.0, -100.0, -100.0};
  // k_update wrote all block partials for a stats sample, the first alone for the forcing, else none
  const long long nb = (g.force_var || stats) ? nblk : 0;
  for (long long b = threadIdx.x; b < nb; b += FIN_NT) {
    const double* o = red + b * NRED_UPD;
    v[0] = v[0] + o[0];
    if (stats) {
      v[1] = v[1] + o[1];
      for (int r = 0; r < 3; ++r) { mn[r] = fmin(mn[r], o[2 + r]); mx[r] = fmax(mx[r], o[5 + r]); }
    }
  }
  block_reduce_sum<2, FIN_NT>(v, sm);
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn[r] = fmin(mn[r], __shfl_down_sync(0xffffffffu, mn[r], o));
      mx[r] = fmax(mx[r], __shfl_down_sync(0xffffffffu, mx[r], o));
    }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int r = 0; r < 3; ++r) { smn[r * (FIN_NT / 32) + warp] = mn[r]; smx[r * (FIN_NT / 32) + warp] = mx[r]; }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (g.force_var) {
      double bulktg = v[0] / g.volchan;
      bulktg = bulktg / sc->rhobulk / sc->ubulk;
      sc->tbdiff = g.t_bulk_target - bulktg;
      sc->pending_shift = 1;
    }
    if (stats) {
      sc->residual_sum = v[1];
      double a[3], b[3];
      for (int r = 0; r < 3; ++r) {
        a[r] = DBL_MAX; b[r] = -100.0;
        for (int wq = 0; wq < FIN_NT / 32; ++wq) {
          a[r] = fmin(a[r], smn[r * (FIN_NT / 32) + wq]);
          b[r] = fmax(b[r], smx[r * (FIN_NT / 32) + wq]);
        }
      }
      sc->rhomin = a[0]; sc->tmin = a[1]; sc->pmin = a[2];
      sc->rhomax = b[0]; sc->tmax = b[1]; sc->pmax = b[2];
      if (!(v[1] == v[1])) sc->nan_flag = 1;
    }
    if (add_time) sc->time = sc->time + sc->dt;
  }
}
__global__ void __launch_bounds__(FIN_NT) k_finish_upd(Geom g, const double* __restrict__ red, long long nblk,
                                                       int stats, int add_time, Scalars* __restrict__ sc) {
  d_finish_upd(g, red, nblk, stats, add_time, sc, Blk{blockIdx.x, blockIdx.y, blockIdx.z});
}

__global__ void k_add_time(Scalars* sc) { sc->time = sc->time + sc->dt; }

// count_weno_subroutine (kernels_cpu.F90:52-113): number of faces whose stencil sees the sensor
__global__ void __launch_bounds__(256) k_count_weno(Geom g, const double* __restrict__ sensor, double* red) {
  __shared__ double sm[3 * 8];
  const long long q = (long long)blockIdx.x * 256 + threadIdx.x;
  double v[3] = {0.0, 0.0, 0.0};
  if (q < g.nint) {
    int i, j, k;
    cell_of(g, q, i, j, k);
    const int ws = g.weno_scheme;
    const double thr = g.sensor_threshold;
    if (i >= g.eul_imin && i <= g.eul_imax) {
      bool s = false;
      for (int o = -ws + 1; o <= ws; ++o) s = s || sensor_at(g, sensor, i + o, j, k) > thr;
      v[0] = s ? 1.0 : 0.0;
    }
    if (j >= g.eul_jmin && j <= g.eul_jmax) {
      bool s = false;
      for (int o = -ws + 1; o <= ws; ++o) s = s || sensor_at(g, sensor, i, j + o, k) > thr;
      v[1] = s ? 1.0 : 0.0;
    }
    if (k >= g.eul_kmin && k <= g.eul_kmax) {
      bool s = false;
      for (int o = -ws + 1; o <= ws; ++o) s = s || sensor_at(g, sensor, i, j, k + o) > thr;
      v[2] = s ? 1.0 : 0.0;
    }
  }
  block_reduce_sum<3, 256>(v, sm);
  if (threadIdx.x == 0)
    for (int r = 0; r < 3; ++r) red[(long long)blockIdx.x * 3 + r] = v[r];
}

// Face (p, a, b) of direction DIR as wface_index numbers it (x (p, j, k), y (p, i, k), z (p, i, j))
// from the list kernels' thread coordinates: t0 the fastest index of that numbering (x faces: p;
// y and z faces: i), t1 the second, t2 the third.
template <int DIR>
__device__ __forceinline__ void list_face(int t0, int t1, int t2, int& p, int& a, int& b) {
  p = DIR == 0 ? t0 : (DIR == 1 ? t1 : t2);
  a = DIR == 0 ? t1 + 1 : t0 + 1;
  b = DIR == 2 ? t1 + 1 : t2 + 1;
}

// Block-aggregated append: one atomic per block reserves the entries of its faces with shk set
// (the order of a list does not matter, every entry is computed independently).  Returns the
// entry of this thread (any value when !shk).  All threads of the block call it; successive
// calls alternate between the two halves of wsum (2 x warps) and base (2), so that a call
// needs no barrier after its last read.
__device__ __forceinline__ unsigned block_append(bool shk, unsigned* counter, unsigned* wsum, unsigned* base,
                                                 int par) {
  const int nw = (int)(blockDim.x >> 5);
  unsigned* ws = wsum + par * nw;
  const unsigned bal = __ballot_sync(0xffffffffu, shk);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) ws[wid] = (unsigned)__popc(bal);
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned tot = 0;
    for (int q = 0; q < nw; ++q) {
      const unsigned cq = ws[q];
      ws[q] = tot;
      tot += cq;
    }
    base[par] = tot ? atomicAdd(counter, tot) : 0u;
  }
  __syncthreads();
  return base[par] + ws[wid] + (unsigned)__popc(bal & ((1u << lane) - 1u));
}

constexpr int WL_NT = 256;  // list kernels: 32 faces along t0 x 8 along t1

// The sample count of direction DIR: the WENO faces (stencil sees the sensor, eul range) of the
// planes t2 = 0, WSAMPLE, 2 WSAMPLE, ... read from the sensor itself, into wcount[4 + DIR].
template <int DIR, int WS>
__global__ void __launch_bounds__(WL_NT) k_weno_sample(Geom g, const double* __restrict__ sensor) {
  __shared__ unsigned wsum[2 * (WL_NT / 32)];
  __shared__ unsigned base[2];
  const int t0 = blockIdx.x * 32 + (threadIdx.x & 31), t1 = blockIdx.y * 8 + (threadIdx.x >> 5);
  const int t2 = blockIdx.z * WSAMPLE;
  int p, a, b;
  list_face<DIR>(t0, t1, t2, p, a, b);
  const int n0 = DIR == 0 ? g.nx + 1 : g.nx, n1 = DIR == 1 ? g.ny + 1 : g.ny;
  const int emin = DIR == 0 ? g.eul_imin : (DIR == 1 ? g.eul_jmin : g.eul_kmin);
  const int emax = DIR == 0 ? g.eul_imax : (DIR == 1 ? g.eul_jmax : g.eul_kmax);
  bool shk = false;
  if (t0 < n0 && t1 < n1 && p >= emin - 1 && p <= emax) {
#pragma unroll
    for (int o = -WS + 1; o <= WS; ++o) {
      const double th = DIR == 0 ? sensor_at(g, sensor, p + o, a, b)
                                 : (DIR == 1 ? sensor_at(g, sensor, a, p + o, b) : sensor_at(g, sensor, a, b, p + o));
      shk = shk || th > g.sensor_threshold;
    }
  }
  block_append(shk, g.wcount + 4 + DIR, wsum, base, 0);
}

// Whether the lists of direction DIR are built this step (its sample is within the threshold).
template <int DIR>
__device__ __forceinline__ bool list_wanted(const Geom& g) {
  return *(volatile const unsigned*)(g.wcount + 4 + DIR) <= g.wthr_s[DIR];
}

// The sensor flags of a step on the ghosted grid: sensor > threshold at interior points, the
// periodic image at the ghosts of periodic directions and 0 at the others (sensor_at).  Only
// when some direction builds its list; grid-stride over tiles of 32 x 8 points of a z plane.
__global__ void __launch_bounds__(256) k_weno_bits(Geom g, const double* __restrict__ sensor) {
  if (!list_wanted<0>(g) && !list_wanted<1>(g) && !list_wanted<2>(g)) return;
  const unsigned tx = (g.sx + 31) / 32, ty = (g.sy + 7) / 8;
  const unsigned ntile = tx * ty * (unsigned)g.sz;
  for (unsigned tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const unsigned r = tile / tx;
    const int i = (int)(tile - r * tx) * 32 + (threadIdx.x & 31) + 1 - g.ng;
    const int j = (int)(r % ty) * 8 + (threadIdx.x >> 5) + 1 - g.ng;
    const int k = (int)(r / ty) + 1 - g.ng;
    if (i <= g.nx + g.ng && j <= g.ny + g.ng)
      g.wbits[gidx(g, i, j, k)] = sensor_at(g, sensor, i, j, k) > g.sensor_threshold ? 1 : 0;
  }
}

// The WENO faces of direction DIR: the faces the hybrid pass computes (eul range) whose stencil
// sees a sensor flag, appended to the direction's list; grid-stride over tiles of 32 faces along
// t0 x 8 along t1 of one t2 plane.  A direction whose sample is above its threshold builds no
// list and marks its count as above every threshold (its hybrid pass computes the WENO faces).
template <int DIR, int WS>
__global__ void __launch_bounds__(WL_NT) k_weno_list(Geom g) {
  __shared__ unsigned wsum[2 * (WL_NT / 32)];
  __shared__ unsigned base[2];
  if (!list_wanted<DIR>(g)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) g.wcount[DIR] = 0xffffffffu;
    return;
  }
  const int n0 = DIR == 0 ? g.nx + 1 : g.nx, n1 = DIR == 1 ? g.ny + 1 : g.ny;
  const int n2 = DIR == 2 ? g.nz + 1 : g.nz;
  const unsigned tx = (unsigned)(n0 + 31) / 32, ty = (unsigned)(n1 + 7) / 8;
  const unsigned ntile = tx * ty * (unsigned)n2;
  const int emin = DIR == 0 ? g.eul_imin : (DIR == 1 ? g.eul_jmin : g.eul_kmin);
  const int emax = DIR == 0 ? g.eul_imax : (DIR == 1 ? g.eul_jmax : g.eul_kmax);
  const long long sd = DIR == 0 ? 1 : (DIR == 1 ? (long long)g.sx : (long long)g.sx * g.sy);
  int par = 0;
  for (unsigned tile = blockIdx.x; tile < ntile; tile += gridDim.x, par ^= 1) {
    const unsigned r = tile / tx;
    const int t0 = (int)(tile - r * tx) * 32 + (threadIdx.x & 31);
    const int t1 = (int)(r % ty) * 8 + (threadIdx.x >> 5);
    const int t2 = (int)(r / ty);
    int p, a, b;
    list_face<DIR>(t0, t1, t2, p, a, b);
    bool shk = false;
    if (t0 < n0 && t1 < n1 && p >= emin - 1 && p <= emax) {
      // the stencil points p-WS+1 .. p+WS of the face, all inside the ghosted grid (ng >= WS)
      const long long c = DIR == 0 ? gidx(g, p, a, b) : (DIR == 1 ? gidx(g, a, p, b) : gidx(g, a, b, p));
      const unsigned char* f = g.wbits + c;
      unsigned any = 0;
#pragma unroll
      for (int o = -WS + 1; o <= WS; ++o) any |= f[o * sd];
      shk = any != 0;
    }
    const unsigned e = block_append(shk, g.wcount + DIR, wsum, base, par);
    if (shk) g.wlist[DIR][e] = (unsigned)wface_index<DIR>(g, p, a, b);
  }
}

// The fluxes of the listed WENO faces of direction DIR into the face buffer (grid-stride over the
// list; each thread loads its face's stencil as the hybrid pass would hold it).
constexpr int WF_NT = 128;
template <class R, int DIR, int LB, int WS, int FS>
__global__ void __launch_bounds__(WF_NT, sizeof(R) == 8 ? WF_MINB_D : WF_MINB_F) k_weno_faces(Geom g, const R* __restrict__ aux) {
  constexpr int S = LB > WS ? LB : WS;
  const unsigned cnt = g.wcount[DIR];
  if (cnt > g.wthr[DIR]) return;  // the hybrid pass computes the WENO faces itself
  const long long n = g.nvol;
  const long long sd = DIR == 0 ? 1 : (DIR == 1 ? (long long)g.sx : (long long)g.sx * g.sy);
  for (unsigned e = blockIdx.x * WF_NT + threadIdx.x; e < cnt; e += gridDim.x * WF_NT) {
    const unsigned f = g.wlist[DIR][e];
    int p, a, b;
    wface_decode<DIR>(g, f, p, a, b);
    const long long base = DIR == 0 ? gidx(g, p, a, b) : (DIR == 1 ? gidx(g, a, p, b) : gidx(g, a, b, p));
    const Line<R> ln{aux + base - (S - 1) * sd, n, sd};
    double fw[5];
    __shared__ R wsc[scr_vals<R, WS>() * WF_NT];
    const Scr<R> scr{wsc + threadIdx.x, WF_NT};
    weno_face<R, DIR, LB, WS, S, FS>(g, ln, face_ep<DIR>(g, p), fw, scr);
#pragma unroll
    for (int m = 0; m < 5; ++m) g.wface[m * g.nwface + f] = fw[m];
  }
}

inline unsigned nblocks(long long n, int nt) { return (unsigned)((n + nt - 1) / nt); }
// Launch shape of the x pass: XF_TY warps a block, each of ngrp groups of 32 faces with one face
// shared between neighbouring warps; as many groups as leave four waves of resident warps (a group
// more saves a face in 32 and hides the copy of its points, a wave less leaves SMs idle at the end)
inline XShape x_shape(const Geom& g) {
  const int S = std::max(g.lmax_base, g.weno_scheme);
  const long long nface = (long long)(g.nx + 1) * g.ny * g.nz;
  XShape x;
  x.ngrp = (int)std::min<long long>(XG_MAX, std::max<long long>(1, nface / (32LL * 148 * 16 * 4)));
  x.slots = x_slots(g.nx, S);
  const long long per = 32LL * x.ngrp - 1;
  x.nblk = nblocks((std::max<long long>(1, nface - 1) + per - 1) / per, XF_TY);
  return x;
}

// Launch shape of a y or z pass: segments of seglen cells of a line and the warps
// of a block.  The segments are at least minseg cells and at most as many as bring the pass to
// about target threads; among the counts allowed, the one with the least estimated time is taken:
// rounds of a segment's seglen + 1 faces over the block's warps times the blocks an SM works
// through, of which up to MT_FREE run beside one another at no cost (a face is a long dependent
// chain).  Blocks have LW warps; when they are fewer than the SMs can hold, up to MT_MAXW of them
// (a function of the box alone, so that a box has the same partition in every form it runs in).
constexpr int LW = 4, MT_FREE = 4;
struct MarchShape {
  int seglen, nwarps;
  unsigned nblk;
};
inline MarchShape march_shape_with(const Geom& g, int dir, long long target, int minseg) {
  const int emin = dir == 1 ? g.eul_jmin : g.eul_kmin, emax = dir == 1 ? g.eul_jmax : g.eul_kmax;
  const int ncell = emax - emin + 1;
  if (ncell < 1) return MarchShape{1, LW, 0};
  const long long lines = (long long)g.nx * (dir == 1 ? g.nz : g.ny);
  const long long tiles = (lines + 31) / 32;
  const long long most = std::min<long long>(std::max(1, ncell / minseg), (target + lines * LW - 1) / (lines * LW));
  // a segment's flags sit in shared memory: at most MT_SEG cells
  const long long least = (ncell + MT_SEG - 1) / MT_SEG;
  double best = 0.0;
  int bn = 1;
  for (long long ns = least; ns <= std::max(least, most); ++ns) {
    const int sl = (int)((ncell + ns - 1) / ns);
    const double rounds = (sl + 1 + LW - 1) / LW;
    const double perSM = (double)((tiles * ns + 147) / 148);
    const double cost = rounds * std::max(1.0, perSM / MT_FREE);
    if (ns == least || cost < best) {
      best = cost;
      bn = (int)ns;
    }
  }
  MarchShape m;
  m.seglen = (ncell + bn - 1) / bn;
  const long long blocks = tiles * ((ncell + m.seglen - 1) / m.seglen);
  m.nblk = (unsigned)blocks;
  const int room = (int)std::min<long long>(MT_MAXW, 148LL * MT_MAXW / std::max<long long>(1, blocks));
  m.nwarps = LW;
  if (room > LW) {
    const int rounds = (m.seglen + 1 + room - 1) / room;
    m.nwarps = std::max(LW, (m.seglen + 1 + rounds - 1) / rounds);
  }
  return m;
}
inline MarchShape march_shape(const Geom& g, int dir) {
  return march_shape_with(g, dir, g.march_threads, g.march_minseg);
}

// typed views of the precision-dependent buffers
template <class R> R* aux_of(DevState& d);
template <> double* aux_of<double>(DevState& d) { return d.aux; }
template <> float* aux_of<float>(DevState& d) { return d.auxf; }
template <class R> R* div3_of(DevState& d);
template <> double* div3_of<double>(DevState& d) { return d.div3; }
template <> float* div3_of<float>(DevState& d) { return d.div3f; }

}  // namespace

}  // namespace sb200
