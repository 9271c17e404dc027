// Device functions of the hybrid convective flux at one cell face: energy-preserving split-form
// central flux (KEEP variants) and characteristic WENO where the Ducros sensor fires.
// Restates euler_{x,y,z}_*hybrid_kernel, compute_roe_average, eigenvectors_{x,y,z} and
// wenorec_1d of code/src/singleideal/kernels_cpu.F90 (lines cited per function).
#pragma once

#include "common.cuh"

// quotients and square roots of the mixed form's FP32 flux arithmetic: IEEE (0), the hardware
// approximations (1), or the hardware approximations refined by one Newton step (2)
#ifndef SB_FP32_FAST
#define SB_FP32_FAST 2
#endif

namespace sb200 {

// Quotient and square root (of a positive value) in the flux arithmetic: IEEE in FP64, where the
// reference's operations are kept; with SB_FP32_FAST the FP32 form takes the hardware reciprocal
// and reciprocal square root (at most 2 ulp: the mixed form's error is set by FP32 rounding).
// With SB_FP32_FAST = 2 the approximate reciprocal r of b is refined by one Newton-Raphson step
// (e = 1 - b r, r += r e) and the quotient q = a r corrected by its remainder (Markstein:
// q += r (a - b q)); the approximate reciprocal square root y of x gives s = x y, corrected by one
// Newton step for the square root (s += (x - s s) y / 2).  Without the refinement the errors of
// the raw approximations do not average out over many steps (the transverse momenta of a
// WENO-only channel drifted twice as far from the FP64 oracle in 100 steps).
template <class R>
__device__ __forceinline__ R fdiv(R a, R b) {
  if constexpr (sizeof(R) == sizeof(double) || !SB_FP32_FAST) {
    return a / b;
  } else if constexpr (SB_FP32_FAST == 1) {
    return __fdividef(a, b);
  } else {
    float r = __fdividef(1.0f, b);
    const float e = __fmaf_rn(-b, r, 1.0f);
    r = __fmaf_rn(r, e, r);
    const float q = a * r;
    return __fmaf_rn(r, __fmaf_rn(-b, q, a), q);
  }
}
template <class R>
__device__ __forceinline__ R fsqrt_pos(R x) {
  if constexpr (sizeof(R) == sizeof(double) || !SB_FP32_FAST) {
    return sqrt(x);
  } else if constexpr (SB_FP32_FAST == 1) {
    return x * rsqrtf(x);
  } else {
    const float y = rsqrtf(x);
    const float sx = x * y;
    return __fmaf_rn(__fmaf_rn(-sx, sx, x), 0.5f * y, sx);
  }
}

__device__ __forceinline__ float rcp_pos(float b) { return fdiv(1.0f, b); }
__device__ __forceinline__ float rsqrt_pos(float x) { return rsqrt(x); }
// maximum that keeps b when a is not a number (as fmax does for the running maxima here), without
// fmax's handling of two of them in FP64
__device__ __forceinline__ double max_of(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ float max_of(float a, float b) { return fmaxf(a, b); }

// The stencil of a face: point q = 0 .. 2S-1 (offsets -(S-1) .. S from the face's lower point) of
// field f (rho, u, v, w, H, T and, in the FP64 form, F_C, the sound speed).
constexpr int F_C = 6;
// in global memory
template <class R>
struct Line {
  const R* p;        // field 0 at point 0
  long long n, sd;   // strides of the fields and of the points
  __device__ __forceinline__ R operator()(int f, int q) const { return __ldg(p + (f == F_C ? 7 : f) * n + q * sd); }
};
// in a ring of points in shared memory, 32 lanes of a field in a row, RF fields a point.  The reads
// are volatile: the compiler would otherwise keep the stencil in registers from its first use to
// its last (36 values in 72 registers), where a second read costs one instruction.
template <class R>
constexpr int ring_fields() { return sizeof(R) == sizeof(double) ? 7 : 6; }
template <class R, int NP>
struct Ring {
  unsigned o[NP];    // shared address of this lane's field 0 at point q
  __device__ __forceinline__ R operator()(int f, int q) const {
    R v;
    if constexpr (sizeof(R) == sizeof(double)) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(o[q] + f * 256));
    else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(o[q] + f * 128));
    return v;
  }
};

// in a row of points in shared memory, XS values a point (an odd count: lanes at consecutive points
// meet no bank twice), lane by lane from its own first point
constexpr int XS = 7;
template <class R>
struct RowPts {
  unsigned o;        // shared address of field 0 at point 0
  __device__ __forceinline__ R operator()(int f, int q) const {
    R v;
    if constexpr (sizeof(R) == sizeof(double)) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(o + (q * XS + f) * 8));
    else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(o + (q * XS + f) * 4));
    return v;
  }
};

// Stencil of a face in registers: NP = 2*S points.
template <class R, int S>
struct Stencil {
  R rho[2 * S], u[2 * S], v[2 * S], w[2 * S], h[2 * S], t[2 * S];
};

// One side of wenorec_1d (kernels_cpu.F90:2526-2724): v[0 .. 2WS-2] in upwind order (the upwind
// cell of the face at v[WS-1]) scaled so that its smoothness indicators are divided by the
// reference's scale, eps2 = 1e-6 in that scaling.  The side's value is base + num/den.
// The indicators and candidates are written in first and second differences d, s of the points:
// beta_k = 13/12 s_k^2 + 1/4 b_k^2 with b_k = 3 d - d', d + d', d' - 3 d, and candidate k minus the
// upwind cell is (3 d + 2 s)/6 or (3 d - s)/6; the weights' common factors (1/4 of the indicators,
// 1/10 of the weights) cancel.  With the projection of weno_flux a face of the FP64 y pass executes
// 880 FP64 instructions (central faces of its warp included) where the point values, with the fluxes
// projected beside the states and IEEE quotients, took 1415.
template <class R, int WS, bool WZ>
__device__ __forceinline__ void weno_side(const R (&v)[2 * WS - 1], int ord, R eps2, R& base, R& num, R& den) {
  constexpr int c = WS - 1;
  base = v[c];
  num = R(0);
  den = R(1);
  if (ord == 1) return;
  if constexpr (WS >= 3) {
    if (ord == 3) {
      const R d0 = v[c - 1] - v[c - 2], d1 = v[c] - v[c - 1], d2 = v[c + 1] - v[c], d3 = v[c + 2] - v[c + 1];
      const R s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2;
      const R b0 = R(3) * d1 - d0, b1 = d1 + d2, b2 = d3 - R(3) * d2;
      const R k = R(13.0 / 3.0);
      const R t3 = R(3) * d1;
      const R r0 = R(2) * s0 + t3, r1 = R(2) * s1 + t3, r2 = R(3) * d2 - s2;  // 6 (candidate - base)
      R n0, n1, n2;
      if constexpr (!WZ) {
        const R eps = R(4) * eps2;
        const R e0 = b0 * b0 + ((k * s0) * s0 + eps), e1 = b1 * b1 + ((k * s1) * s1 + eps),
                e2 = b2 * b2 + ((k * s2) * s2 + eps);
        // omega_k = (d_k/e_k^2) / sum, written over the common denominator
        const R p12 = e1 * e2, p02 = e0 * e2, p01 = e0 * e1;
        n0 = p12 * p12;
        n1 = R(6) * (p02 * p02);
        n2 = R(3) * (p01 * p01);
      } else {
        // WENO-Z, omega_k = d_k (beta_k + tau)/(beta_k + eps); eps is a single-precision literal in
        // the reference
        const R eps = R(4.0 * static_cast<double>(1.e-35f) / 0.000001) * eps2;
        const R e0 = b0 * b0 + (k * s0) * s0, e1 = b1 * b1 + (k * s1) * s1, e2 = b2 * b2 + (k * s2) * s2;
        const R tau = fabs(e0 - e2) + eps;
        if constexpr (sizeof(R) == sizeof(double)) {
          const R f0 = e0 + eps, f1 = e1 + eps, f2 = e2 + eps;
          n0 = (e0 + tau) * (f1 * f2);
          n1 = R(6) * ((e1 + tau) * (f0 * f2));
          n2 = R(3) * ((e2 + tau) * (f0 * f1));
        } else {  // the products of two eps leave the FP32 range
          n0 = R(1) / ((e0 + eps) / (e0 + tau));
          n1 = R(6) / ((e1 + eps) / (e1 + tau));
          n2 = R(3) / ((e2 + eps) / (e2 + tau));
        }
      }
      den = n0 + n1 + n2;
      num = (n0 * r0 + n1 * r1 + n2 * r2) * R(1.0 / 6.0);
      return;
    }
  }
  if constexpr (WS >= 2) {
    if (ord == 2) {
      const R d1 = v[c] - v[c - 1], d2 = v[c + 1] - v[c];
      const R e0 = d1 * d1 + eps2, e1 = d2 * d2 + eps2;
      const R n0 = e1 * e1, n1 = R(2) * (e0 * e0);
      den = n0 + n1;
      num = R(0.5) * (n0 * d1 + n1 * d2);
      return;
    }
  }
  if constexpr (WS >= 4) {
    const R k1 = R(1.0 / 36.0), k2 = R(13.0 / 12.0), k3 = R(781.0 / 720.0);
    auto sq = [](R a) { return a * a; };
    const R a0 = v[c - 3], a1 = v[c - 2], a2 = v[c - 1], a3 = v[c], a4 = v[c + 1], a5 = v[c + 2], a6 = v[c + 3];
    R b[4];
    b[3] = k1 * sq(-11 * a3 + 18 * a4 - 9 * a5 + 2 * a6) + k2 * sq(2 * a3 - 5 * a4 + 4 * a5 - a6) +
           k3 * sq(-a3 + 3 * a4 - 3 * a5 + a6);
    b[2] = k1 * sq(-2 * a2 - 3 * a3 + 6 * a4 - a5) + k2 * sq(a2 - 2 * a3 + a4) + k3 * sq(-a2 + 3 * a3 - 3 * a4 + a5);
    b[1] = k1 * sq(a1 - 6 * a2 + 3 * a3 + 2 * a4) + k2 * sq(a2 - 2 * a3 + a4) + k3 * sq(-a1 + 3 * a2 - 3 * a3 + a4);
    b[0] = k1 * sq(-2 * a0 + 9 * a1 - 18 * a2 + 11 * a3) + k2 * sq(-a0 + 4 * a1 - 5 * a2 + 2 * a3) +
           k3 * sq(-a0 + 3 * a1 - 3 * a2 + a3);
    const R dw[4] = {R(1), R(12), R(18), R(4)};
    // with the indicators relative to eps in FP32, whose range is too narrow for the weights' squares
    const R sc = sizeof(R) == sizeof(double) ? R(1) : R(1) / eps2;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const R e = sc * (b[l] + eps2);
      b[l] = dw[l] / (e * e);
    }
    den = b[0] + b[1] + b[2] + b[3];
    base = R(0);
    num = (b[3] * (6 * a3 + 26 * a4 - 10 * a5 + 2 * a6) + b[2] * (-2 * a2 + 14 * a3 + 14 * a4 - 2 * a5) +
           b[1] * (2 * a1 - 10 * a2 + 26 * a3 + 6 * a4) + b[0] * (-6 * a0 + 26 * a1 - 46 * a2 + 50 * a3)) *
          R(1.0 / 24.0);
  }
}
// wenorec_1d of one variable: the two sides of the face, p in upwind order from the left, m from the
// right.  FP64 takes one reciprocal for both (the denominators are positive and stay far inside the
// exponent range); the FP32 range is too narrow for their product.
template <class R, int WS, bool WZ>
__device__ __forceinline__ R weno_rec(const R (&p)[2 * WS - 1], const R (&m)[2 * WS - 1], int ord, R eps2) {
  R bp, np, dp, bm, nm, dm;
  weno_side<R, WS, WZ>(p, ord, eps2, bp, np, dp);
  weno_side<R, WS, WZ>(m, ord, eps2, bm, nm, dm);
  if constexpr (sizeof(R) == sizeof(double)) return (bp + bm) + (np * dm + nm * dp) * rcp_pos(dp * dm);
  else return (bp + bm) + (fdiv(np, dp) + fdiv(nm, dm));
}

// Central energy-preserving split-form flux (kernels_cpu.F90:462-612 for x; same in y, z).
// DIR: 0 x, 1 y, 2 z.  The general form: KEEP(n) (nkeep != 0), and the default nkeep = 0 in FP32.
// The sums over the stencil are formed in R, those over their orders l and the flux in FP64: face
// fluxes leave in FP64, so that the differences of neighbouring faces do not lose the mixed form's
// digits to the FP32 rounding of their final sums.
template <class R, int DIR, int LB, int S, bool KG, class LN>
__device__ __forceinline__ void central_flux_general(const Geom& g, const LN& ln, int lmax, int nkeep_in,
                                                     bool zero_flux, double (&f)[5]) {
  const int nkeep = KG ? nkeep_in : 0;
  const R rgas0 = R(g.rgas0);
  Stencil<R, S> st;
  R pp[2 * S], ee[2 * S];
#pragma unroll
  for (int q = S - LB; q < S + LB; ++q) {
    st.rho[q] = ln(0, q); st.u[q] = ln(1, q); st.v[q] = ln(2, q); st.w[q] = ln(3, q);
    st.h[q] = ln(4, q); st.t[q] = ln(5, q);
    pp[q] = st.t[q] * st.rho[q] * rgas0;
    // e = H - p/rho - |u|^2/2 with p/rho = R T taken directly (the reference divides p by rho;
    // the two differ in the last bit only and the division is the costliest operation here)
    ee[q] = st.h[q] - st.t[q] * rgas0 - R(0.5) * (st.u[q] * st.u[q] + st.v[q] * st.v[q] + st.w[q] * st.w[q]);
  }
  double ft[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int l = 1; l <= LB; ++l) {
    if (l <= lmax) {
      R uvs1 = 0, uvs2 = 0, uvs3 = 0, uvs4 = 0, uvs5 = 0, uvs5_i = 0, uvs5_k = 0, uvs5_p = 0, uvs6 = 0;
#pragma unroll
      for (int m = 0; m < LB; ++m) {
        if (m <= l - 1) {
          const int a = -m + S - 1, b = -m + l + S - 1;
          const R vna = DIR == 0 ? st.u[a] : (DIR == 1 ? st.v[a] : st.w[a]);
          const R vnb = DIR == 0 ? st.u[b] : (DIR == 1 ? st.v[b] : st.w[b]);
          R rhom = st.rho[a] + st.rho[b];
          if (nkeep >= 0) {
            R eem = ee[a] + ee[b];
            R drhof = R(1), deef = R(1);
            if (nkeep != 0) {
              R drho = R(2) * (st.rho[b] - st.rho[a]) / rhom;
              R dee = R(2) * (ee[b] - ee[a]) / eem;
              R t_sumdenrho = (R(0.5) * drho) * (R(0.5) * drho);
              R t_sumdenee = (R(0.5) * dee) * (R(0.5) * dee);
              R t2r = t_sumdenrho, t2e = t_sumdenee;
              R sumdenrho = R(1) + t_sumdenrho / R(3);
              R sumdenee = R(1) + t_sumdenee;
              R sumnumee = R(1) + t_sumdenee / R(3);
              for (int n = 2; n <= nkeep; ++n) {
                R n21 = R(1) + R(2 * n);
                t_sumdenrho = t2r * t_sumdenrho;
                t_sumdenee = t2e * t_sumdenee;
                sumdenrho = sumdenrho + t_sumdenrho / n21;
                sumdenee = sumdenee + t_sumdenee;
                sumnumee = sumnumee + t_sumdenee / n21;
              }
              drhof = R(1) / sumdenrho;
              deef = sumnumee / sumdenee;
            }
            R uv_part = (vna + vnb) * rhom * drhof;
            uvs1 = uvs1 + uv_part * R(2);
            uvs2 = uvs2 + uv_part * (st.u[a] + st.u[b]);
            uvs3 = uvs3 + uv_part * (st.v[a] + st.v[b]);
            uvs4 = uvs4 + uv_part * (st.w[a] + st.w[b]);
            uvs5_i = uvs5_i + uv_part * eem * deef;
            uvs5_k = uvs5_k + uv_part * (st.u[a] * st.u[b] + st.v[a] * st.v[b] + st.w[a] * st.w[b]);
            uvs5_p = uvs5_p + R(4) * (vna * pp[b] + vnb * pp[a]);
            uvs6 = uvs6 + R(2) * (pp[a] + pp[b]);
          } else {
            R uv_part = (vna + vnb) * rhom;
            uvs1 = uvs1 + uv_part * R(2);
            uvs2 = uvs2 + uv_part * (st.u[a] + st.u[b]);
            uvs3 = uvs3 + uv_part * (st.v[a] + st.v[b]);
            uvs4 = uvs4 + uv_part * (st.w[a] + st.w[b]);
            uvs5 = uvs5 + uv_part * (st.h[a] + st.h[b]);
            uvs6 = uvs6 + R(2) * (pp[a] + pp[b]);
          }
        }
      }
      const double cl = g.coeff[lmax - 1][l - 1];
      ft[0] = ft[0] + cl * double(uvs1);
      ft[1] = ft[1] + cl * double(uvs2);
      ft[2] = ft[2] + cl * double(uvs3);
      ft[3] = ft[3] + cl * double(uvs4);
      ft[4] = ft[4] + cl * double(nkeep >= 0 ? (uvs5_i + uvs5_k + uvs5_p) : uvs5);
      ft[5] = ft[5] + cl * double(uvs6);
    }
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) f[m] = zero_flux ? 0.0 : 0.25 * ft[m];
  f[1 + DIR] = f[1 + DIR] + 0.5 * ft[5];
}

// nkeep = 0 in FP64, pair by pair: the sum over the orders l and the pairs (a, b) of an order is
// one over all pairs with the coefficient of l = b - a on each, taken lower point by lower point,
// so that LB + 1 points are held instead of 2 LB (the registers of a flux kernel are set by this
// branch and the characteristic one: see XF_MINB_D).
template <int DIR, int LB, int S, class LN>
__device__ __forceinline__ void central_flux_pairs(const Geom& g, const LN& ln, int lmax, bool zero_flux,
                                                   double (&f)[5]) {
  const double rgas0 = g.rgas0;
  struct Pt {
    double rho, v[3], pp, ee;
  };
  auto load = [&](int q) {
    Pt a;
    a.rho = ln(0, q);
    a.v[0] = ln(1, q); a.v[1] = ln(2, q); a.v[2] = ln(3, q);
    const double rt = ln(5, q) * rgas0;
    a.pp = rt * a.rho;
    // e = H - p/rho - |u|^2/2 with p/rho = R T
    a.ee = ln(4, q) - rt - 0.5 * (a.v[0] * a.v[0] + a.v[1] * a.v[1] + a.v[2] * a.v[2]);
    return a;
  };
  const double* cf = g.coeff[lmax - 1];
  double f1 = 0, fv[3] = {0, 0, 0}, fe = 0, fp = 0;
  Pt up[LB];
#pragma unroll
  for (int u = 0; u < LB; ++u) up[u] = load(S + u);
#pragma unroll
  for (int m = 0; m < LB; ++m) {  // lower point S-1-m with the upper points S .. S+LB-1-m
    const Pt a = load(S - 1 - m);
#pragma unroll
    for (int u = 0; u < LB; ++u) {
      const int l = m + u + 1;
      if (l <= LB && l <= lmax) {
        const Pt& b = up[u];
        const double cl = cf[l - 1];
        const double uv = cl * ((a.v[DIR] + b.v[DIR]) * (a.rho + b.rho));
        f1 = f1 + uv;
#pragma unroll
        for (int d = 0; d < 3; ++d) fv[d] = fv[d] + uv * (a.v[d] + b.v[d]);
        fe = fe + uv * ((a.ee + b.ee) + (a.v[0] * b.v[0] + a.v[1] * b.v[1] + a.v[2] * b.v[2]));
        fe = fe + (4.0 * cl) * (a.v[DIR] * b.pp + b.v[DIR] * a.pp);
        fp = fp + cl * (a.pp + b.pp);
      }
    }
  }
  f[0] = zero_flux ? 0.0 : 0.5 * f1;
#pragma unroll
  for (int d = 0; d < 3; ++d) f[1 + d] = zero_flux ? 0.0 : 0.25 * fv[d];
  f[4] = zero_flux ? 0.0 : 0.25 * fe;
  f[1 + DIR] = f[1 + DIR] + fp;
}

// KG = false: nkeep = 0 fixed at compile time (the KEEP(n) divisions would otherwise shape the
// register allocation of the whole flux kernel).
template <class R, int DIR, int LB, int S, bool KG, class LN>
__device__ __forceinline__ void central_flux(const Geom& g, const LN& ln, int lmax, int nkeep, bool zero_flux,
                                             double (&f)[5]) {
  if constexpr (sizeof(R) == sizeof(double) && !KG) central_flux_pairs<DIR, LB, S>(g, ln, lmax, zero_flux, f);
  else central_flux_general<R, DIR, LB, S, KG>(g, ln, lmax, nkeep, zero_flux, f);
}

// A thread's own values in shared memory, for the FP64 form (st apart; a = 0: in registers).  They
// are volatile for the same reason as the ring's.
template <class R>
struct Scr {
  unsigned a, st;
  __device__ __forceinline__ void put(int q, R v) const {
    if constexpr (sizeof(R) == sizeof(double)) asm volatile("st.shared.f64 [%0], %1;" ::"r"(a + q * st), "d"(v));
  }
  __device__ __forceinline__ R get(int q) const {
    R v = R(0);
    if constexpr (sizeof(R) == sizeof(double)) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a + q * st));
    return v;
  }
};

// Characteristic WENO flux: compute_roe_average (kernels_cpu.F90:3013-3089), eigenvectors_{x,y,z}
// (:2728-2782, :2842-2896, :2956-3010), local Lax-Friedrichs splitting with the stencil maximum
// of |u_n -+ c| (:614-675) and wenorec_1d; back-projection with the right eigenvectors (:677-683),
// accumulated in FP64 in both forms.
// TP: thermally perfect gas (Newton for the Roe-averaged temperature, gamma(T) per point; FP64).
// WZ: WENO-Z weights (weno_version = 1) instead of WENO-JS, fixed at compile time.
//
// The stencil is read point by point, again where it is needed again, and the fields are taken one
// after another: what a thread holds between them are the projections of its points' states and
// fluxes on the two acoustic fields, in its scratch (against the projections of the states only, the
// fluxes formed again per field: 1024x256x192, FP64, 50.4 -> 49.0 ms per step; 1024x256x128 mixed
// 26.8 -> 25.8).
template <class R, int DIR, int WS, int S, bool TP, bool WZ, class LN>
__device__ __forceinline__ void weno_flux(const Geom& g, const LN& ln, int ord, double (&f)[5], const Scr<R>& scr) {
  static_assert(!TP || sizeof(R) == sizeof(double), "the thermally perfect gas is an FP64 path");
  constexpr int NP = 2 * WS - 1;
  const R rgas0 = R(g.rgas0);
  constexpr int t1 = DIR == 0 ? 1 : 0;
  constexpr int t2 = DIR == 2 ? 1 : 2;
  constexpr int q0 = S - WS;  // the first point used
  // Roe average of the two points adjacent to the face
  R vel[3], h, r, rp1;
  {
    const R ra = ln(0, S - 1), rb = ln(0, S);
    if constexpr (sizeof(R) == sizeof(double)) r = rb * rsqrt_pos(ra * rb);  // sqrt(rb/ra)
    else r = fsqrt_pos(fdiv(rb, ra));
    rp1 = rcp_pos(r + R(1));
#pragma unroll
    for (int d = 0; d < 3; ++d) vel[d] = (r * ln(1 + d, S) + ln(1 + d, S - 1)) * rp1;
    h = (r * ln(4, S) + ln(4, S - 1)) * rp1;
  }
  const R qq = R(0.5) * (vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
  const R hbar = h - qq - R(g.cp_last) * R(g.t0);
  R c, ci, b1, b2, b3;
  if constexpr (TP) {
    // Newton on h(T) from the Roe average of the two temperatures (compute_roe_average)
    const R t_start = (r * ln(5, S) + ln(5, S - 1)) * rp1;
    const R tt = tp_newton(g, g.cpc, hbar, t_start);
    const R gamloc = gamloc_of_t(g, tt);
    const R cc = gamloc * tt * rgas0;
    const R rho = r * ln(0, S - 1), p_rho = tt * rgas0, etot = h - tt * rgas0;
    const R gm1loc = gamloc - R(1);
    c = sqrt(cc);
    ci = R(1) / c;
    const R p_e = rho * gm1loc;
    b3 = etot - rho * p_rho / p_e;
    b2 = p_e / (rho * cc);
    b1 = p_rho / cc - b2 * (etot - R(2) * qq);
  } else {
    // constant gamma: p_e = rho (gamma - 1), so b2 = (gamma - 1)/c^2 and rho p_rho/p_e =
    // p_rho/(gamma - 1); one reciprocal square root gives c and 1/c (the reference forms three
    // quotients and a square root here: the results differ in the last bits)
    const R tt = sizeof(R) == sizeof(double) ? R(g.t0) + hbar * R(g.rcp0) : R(g.t0) + fdiv(hbar, R(g.cp0));
    const R p_rho = tt * rgas0, cc = R(g.gamloc) * p_rho, etot = h - p_rho;
    ci = rsqrt_pos(cc);
    c = cc * ci;
    const R ci2 = ci * ci;
    b2 = R(g.gm1) * ci2;
    b1 = p_rho * ci2 - b2 * (etot - R(2) * qq);
    b3 = etot - p_rho * R(g.rgm1);
  }
  // stencil maximum of the characteristic speeds (offsets -WS+1 .. WS)
  R ev0 = R(-1), ev1 = R(-1), ev4 = R(-1);
#pragma unroll
  for (int l = 0; l < 2 * WS; ++l) {
    const R vnq = ln(1 + DIR, q0 + l);
    R cs;
    if constexpr (sizeof(R) == sizeof(double)) cs = ln(F_C, q0 + l);  // the aux pass's sound speed (FP64 form)
    else cs = fsqrt_pos(R(g.gamloc) * rgas0 * ln(5, q0 + l));
    ev0 = max_of(fabs(vnq - cs), ev0);
    ev1 = max_of(fabs(vnq), ev1);
    ev4 = max_of(fabs(vnq + cs), ev4);
  }
  // Projection from the structure of the left eigenvectors and of the flux: with
  // U = rho (1, u, v, w, E) and F = u_n U + p (0, n, u_n), P(F) = u_n P(U) + p P(0, n, u_n), so that
  // only U is projected.  s = rho (b1 + b2 (E - u_Roe.u)), a = rho ci (vn - u_n) give
  //   P1 = (s + a)/2, P2 = rho - s, P3 = rho (u_t1 - v_t1), P4 = rho (u_t2 - v_t2), P5 = (s - a)/2
  // and the split values are (u_n +- lambda_m) P_m(U) + p P_m(0, n, u_n), kept as 4 (m = 1, 5) and 2
  // times the reference's g+-, exactly, undone after weno_rec.  wenorec_1d reads g+ at the points
  // 1 .. 2WS-1 and g- at 2 .. 2WS whatever its order; the g- side is kept in upwind order from the
  // right.  sg scales FP32 densities (a power of two near 1/(rho0 u0)).
  constexpr bool D = sizeof(R) == sizeof(double);
  const R sg = D ? R(1) : R(g.wsg_a), isg = D ? R(1) : R(g.wsg_ai);
  auto rho_at = [&](int q) { return D ? ln(0, q) : ln(0, q) * sg; };
  R fi[5];
  // the two shear fields
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int t = m == 0 ? t1 : t2;
    R gp[NP], gm[NP];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const R P = rho_at(q0 + l) * (ln(1 + t, q0 + l) - vel[t]), T = ln(1 + DIR, q0 + l) * P;
      if (l < 2 * WS - 1) gp[l] = T + ev1 * P;
      if (l > 0) gm[2 * WS - 1 - l] = T - ev1 * P;
    }
    fi[2 + m] = weno_rec<R, WS, WZ>(gp, gm, ord, R(D ? g.weps_b : g.wepsf_ab) * R(4)) * (R(0.5) * isg);
  }
  // the entropy field, and P_m(U) and T_m = P_m(F) of the two acoustic ones (g+- = T +- lambda P)
  const R epsa = R(D ? g.weps_a : g.wepsf_a);
  R hold[D ? 1 : 8 * WS];
  auto put = [&](int q, R v) {
    if constexpr (D) scr.put(q, v);
    else hold[q] = v;
  };
  auto get = [&](int q) -> R {
    if constexpr (D) return scr.get(q);
    else return hold[q];
  };
  {
    R gp[NP], gm[NP];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const int q = q0 + l;
      const R rr = rho_at(q), rt = ln(5, q) * rgas0;
      const R vq[3] = {ln(1, q), ln(2, q), ln(3, q)};
      const R un = vq[DIR], dn = vel[DIR] - un, pp = rr * rt;
      const R de = (ln(4, q) - rt) - (vel[0] * vq[0] + vel[1] * vq[1] + vel[2] * vq[2]);
      const R sv = rr * (b2 * de + b1);
      const R av = ci * (rr * dn);
      const R ps = (pp * b2) * dn, pc = pp * ci;
      const R A = sv + av, B = sv - av, E = rr - sv;
      put(4 * l, A);
      put(4 * l + 1, un * A - (ps + pc));
      put(4 * l + 2, B);
      put(4 * l + 3, un * B + (pc - ps));
      const R T = un * E + ps;
      if (l < 2 * WS - 1) gp[l] = T + ev1 * E;
      if (l > 0) gm[2 * WS - 1 - l] = T - ev1 * E;
    }
    fi[1] = weno_rec<R, WS, WZ>(gp, gm, ord, epsa * R(4)) * (R(0.5) * isg);
  }
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const R lam = m == 0 ? ev0 : ev4;
    R gp[NP], gm[NP];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const R P = get(4 * l + 2 * m), T = get(4 * l + 2 * m + 1);
      if (l < 2 * WS - 1) gp[l] = T + lam * P;
      if (l > 0) gm[2 * WS - 1 - l] = T - lam * P;
    }
    fi[4 * m] = weno_rec<R, WS, WZ>(gp, gm, ord, epsa * R(16)) * (R(0.25) * isg);
  }
  // back-projection with the right eigenvectors, er(m,:) = (1, u - c n, h - vn c) for m = 1,
  // (1, u, b3) for m = 2, (0, e_t, v_t) for m = 3, 4, (1, u + c n, h + vn c) for m = 5
  const double F0 = fi[0], F1 = fi[1], F2 = fi[2], F3 = fi[3], F4 = fi[4];
  const double vd[3] = {double(vel[0]), double(vel[1]), double(vel[2])};
  const double fa = F0 + F4, fd = double(c) * (F4 - F0);
  f[0] = fa + F1;
#pragma unroll
  for (int d = 0; d < 3; ++d) f[1 + d] = vd[d] * f[0] + (d == DIR ? fd : (d == t1 ? F2 : F3));
  f[4] = double(h) * fa + vd[DIR] * fd + double(b3) * F1 + vd[t1] * F2 + vd[t2] * F3;
}

// Rusanov (component-wise local Lax-Friedrichs) WENO flux of the *_hybrid_rusanov kernels
// (kernels_cpu.F90:692-941 for x, same in y and z): stencil maximum of |u_n -+ c|, split
// values of the conserved fluxes, wenorec with the scales of wenorec_1d_rusanov (:2325-2523).
template <class R, int DIR, int WS, int S, bool TP, bool WZ, class LN>
__device__ __forceinline__ void rusanov_flux(const Geom& g, const LN& ln, int ord, double (&f)[5]) {
  static_assert(!TP || sizeof(R) == sizeof(double), "the thermally perfect gas is an FP64 path");
  constexpr int NP = 2 * WS - 1;
  constexpr int q0 = S - WS;
  const R rgas0 = R(g.rgas0);
  R evmax = R(-1);
#pragma unroll
  for (int l = 0; l < 2 * WS; ++l) {
    const R un = ln(1 + DIR, q0 + l);
    R c;
    if constexpr (sizeof(R) == sizeof(double)) c = ln(F_C, q0 + l);
    else c = fsqrt_pos(R(g.gamloc) * rgas0 * ln(5, q0 + l));
    evmax = max_of(max_of(fabs(un - c), fabs(un + c)), evmax);
  }
#pragma unroll 1
  for (int m = 0; m < 5; ++m) {
    // FP32 values are scaled by a power of two near the square root of the indicators' scale
    R sg = R(1), isg = R(1), eps;
    if constexpr (sizeof(R) == sizeof(double)) {
      eps = m == 0 ? g.weps_a : (m == 4 ? g.weps_c : g.weps_b);
    } else {
      sg = m == 0 ? R(g.wsg_a) : (m == 4 ? R(g.wsg_c) : R(g.wsg_b));
      isg = m == 0 ? R(g.wsg_ai) : (m == 4 ? R(g.wsg_ci) : R(g.wsg_bi));
      eps = m == 0 ? R(g.wepsf_a) : (m == 4 ? R(g.wepsf_c) : R(g.wepsf_b));
    }
    R gp[NP], gm[NP];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const int q = q0 + l;
      const R rho = ln(0, q);
      const R un = ln(1 + DIR, q);
      const R rhou = rho * un;
      R evm, c;
      if (m == 0) {
        evm = rhou;
        c = R(0.5) * (evm + rho * evmax);
      } else if (m == 4) {
        const R h = ln(4, q);
        evm = h * rhou;
        c = R(0.5) * (evm + evmax * (rho * h - rho * ln(5, q) * rgas0));
      } else {
        const R vd = ln(m, q);
        evm = vd * rhou;
        if (m == 1 + DIR) evm = evm + rho * ln(5, q) * rgas0;
        c = R(0.5) * (evm + rho * evmax * vd);
      }
      if (l < 2 * WS - 1) gp[l] = sg * c;
      if (l > 0) gm[2 * WS - 1 - l] = sg * (evm - c);
    }
    const R v = weno_rec<R, WS, WZ>(gp, gm, ord, eps) * isg;
#pragma unroll
    for (int mm = 0; mm < 5; ++mm)
      if (mm == m) f[mm] = double(v);
  }
}

}  // namespace sb200
