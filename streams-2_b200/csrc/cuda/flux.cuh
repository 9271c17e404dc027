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

// Quotient and square root (of a positive value) of the mixed form's FP32 flux arithmetic: with
// SB_FP32_FAST the hardware reciprocal and reciprocal square root (at most 2 ulp: the form's error is
// set by FP32 rounding) instead of the IEEE routines.
// With SB_FP32_FAST = 2 the approximate reciprocal r of b is refined by one Newton-Raphson step
// (e = 1 - b r, r += r e) and the quotient q = a r corrected by its remainder (Markstein:
// q += r (a - b q)); the approximate reciprocal square root y of x gives s = x y, corrected by one
// Newton step for the square root (s += (x - s s) y / 2).  Without the refinement the errors of
// the raw approximations do not average out over many steps (the transverse momenta of a
// WENO-only channel drifted twice as far from the FP64 oracle in 100 steps).
__device__ __forceinline__ float fdiv(float a, float b) {
#if !SB_FP32_FAST
  return a / b;
#elif SB_FP32_FAST == 1
  return __fdividef(a, b);
#else
  float r = __fdividef(1.0f, b);
  const float e = __fmaf_rn(-b, r, 1.0f);
  r = __fmaf_rn(r, e, r);
  const float q = a * r;
  return __fmaf_rn(r, __fmaf_rn(-b, q, a), q);
#endif
}
__device__ __forceinline__ float fsqrt_pos(float x) {
#if !SB_FP32_FAST
  return sqrtf(x);
#elif SB_FP32_FAST == 1
  return x * rsqrtf(x);
#else
  const float y = rsqrtf(x);
  const float sx = x * y;
  return __fmaf_rn(__fmaf_rn(-sx, sx, x), 0.5f * y, sx);
#endif
}

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

// wenorec_1d (kernels_cpu.F90:2526-2724) for one variable in the mixed form's FP32, from the point
// values as the reference writes it: the difference form below rounds differently, and one point
// whose sensor then crosses its threshold another way changes a face by O(1).  The nonlinear weights
// are normalised by one reciprocal of their sum (the reference divides each weight by the sum;
// the results differ in the last bit only).
// vp[l-1], vm[l-1] hold the reference's vp(m,l), vm(m,l), l = 1..2*WS; i = iweno = WS.
template <int WS>
__device__ __forceinline__ float wenorec(const float (&vp)[2 * WS], const float (&vm)[2 * WS], int ord,
                                         int version, float betascale) {
  using R = float;
  auto VP = [&](int l) -> R { return vp[l - 1]; };
  auto VM = [&](int l) -> R { return vm[l - 1]; };
  constexpr int i = WS;
  const R eps6 = R(0.000001);
  if (ord == 1) {
    return VP(i) + VM(i + 1);
  }
  if constexpr (WS >= 2) {
    if (ord == 2) {
      const R dwe0 = R(1.0) / R(3.0), dwe1 = R(2.0) / R(3.0);
      R a = VP(i) - VP(i - 1), b = VP(i + 1) - VP(i);
      R bp0 = betascale * (a * a), bp1 = betascale * (b * b);
      R c = VM(i + 2) - VM(i + 1), d = VM(i + 1) - VM(i);
      R bm0 = betascale * (c * c), bm1 = betascale * (d * d);
      R tp0 = eps6 + bp0, tp1 = eps6 + bp1, tm0 = eps6 + bm0, tm1 = eps6 + bm1;
      bp0 = dwe0 / (tp0 * tp0);
      bm0 = dwe0 / (tm0 * tm0);
      bp1 = dwe1 / (tp1 * tp1);
      bm1 = dwe1 / (tm1 * tm1);
      const R rsp = fdiv(R(1), (R(0) + bp0) + bp1), rsm = fdiv(R(1), (R(0) + bm0) + bm1);
      bp0 = bp0 * rsp; bp1 = bp1 * rsp; bm0 = bm0 * rsm; bm1 = bm1 * rsm;
      R vminus = bp0 * (-VP(i - 1) + R(3) * VP(i)) + bp1 * (VP(i) + VP(i + 1));
      R vplus = bm0 * (-VM(i + 2) + R(3) * VM(i + 1)) + bm1 * (VM(i) + VM(i + 1));
      return R(0.5) * (vminus + vplus);
    }
  }
  if constexpr (WS >= 3) {
    if (ord == 3) {
      const R dwe[3] = {R(1.0) / R(10.0), R(6.0) / R(10.0), R(3.0) / R(10.0)};
      const R d0 = R(13.0) / R(12.0), d1 = R(1.0) / R(4.0);
      const R c0 = R(1.0) / R(3.0), c1 = R(5.0) / R(6.0), c2 = R(-1.0) / R(6.0), c3 = R(-7.0) / R(6.0),
              c4 = R(11.0) / R(6.0);
      R bp[3], bm[3];
      {
        R a = VP(i) - R(2) * VP(i + 1) + VP(i + 2), b = R(3) * VP(i) - R(4) * VP(i + 1) + VP(i + 2);
        bp[2] = d0 * (a * a) + d1 * (b * b);
        a = VP(i - 1) - R(2) * VP(i) + VP(i + 1);
        b = VP(i - 1) - VP(i + 1);
        bp[1] = d0 * (a * a) + d1 * (b * b);
        a = VP(i) - R(2) * VP(i - 1) + VP(i - 2);
        b = R(3) * VP(i) - R(4) * VP(i - 1) + VP(i - 2);
        bp[0] = d0 * (a * a) + d1 * (b * b);
        a = VM(i + 1) - R(2) * VM(i) + VM(i - 1);
        b = R(3) * VM(i + 1) - R(4) * VM(i) + VM(i - 1);
        bm[2] = d0 * (a * a) + d1 * (b * b);
        a = VM(i + 2) - R(2) * VM(i + 1) + VM(i);
        b = VM(i + 2) - VM(i);
        bm[1] = d0 * (a * a) + d1 * (b * b);
        a = VM(i + 1) - R(2) * VM(i + 2) + VM(i + 3);
        b = R(3) * VM(i + 1) - R(4) * VM(i + 2) + VM(i + 3);
        bm[0] = d0 * (a * a) + d1 * (b * b);
      }
#pragma unroll
      for (int l = 2; l >= 0; --l) {
        bp[l] = betascale * bp[l];
        bm[l] = betascale * bm[l];
      }
      if (version == 0) {
        // omega_l = (d_l / t_l) / sum_k (d_k / t_k), t_l = (eps + beta_l)^2, formed with one
        // division per side: omega_l = d_l prod_{m != l} t_m / sum_k d_k prod_{m != k} t_m
        // (the same weights; the products stay far inside the exponent range for eps = 1e-6)
        R tp[3], tm[3];
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          const R a = eps6 + bp[l], b = eps6 + bm[l];
          tp[l] = a * a;
          tm[l] = b * b;
        }
        const R np0 = dwe[0] * (tp[1] * tp[2]), np1 = dwe[1] * (tp[0] * tp[2]), np2 = dwe[2] * (tp[0] * tp[1]);
        const R nm0 = dwe[0] * (tm[1] * tm[2]), nm1 = dwe[1] * (tm[0] * tm[2]), nm2 = dwe[2] * (tm[0] * tm[1]);
        const R rsp = fdiv(R(1), (np0 + np1) + np2), rsm = fdiv(R(1), (nm0 + nm1) + nm2);
        bp[0] = np0 * rsp; bp[1] = np1 * rsp; bp[2] = np2 * rsp;
        bm[0] = nm0 * rsm; bm[1] = nm1 * rsm; bm[2] = nm2 * rsm;
      } else {
        // eps40 is a single-precision literal in the reference
        const R eps40 = R(static_cast<double>(1.e-35f));
        R tau5p = fabs(bp[0] - bp[2]) + eps40;
        R tau5m = fabs(bm[0] - bm[2]) + eps40;
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          bp[l] = (bp[l] + eps40) / (bp[l] + tau5p);
          bm[l] = (bm[l] + eps40) / (bm[l] + tau5m);
        }
        R sump = R(0), summ = R(0);
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          bp[l] = dwe[l] / bp[l];
          bm[l] = dwe[l] / bm[l];
          sump = sump + bp[l];
          summ = summ + bm[l];
        }
        const R rsp = fdiv(R(1), sump), rsm = fdiv(R(1), summ);
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          bp[l] = bp[l] * rsp;
          bm[l] = bm[l] * rsm;
        }
      }
      R vminus = bp[2] * (c0 * VP(i) + c1 * VP(i + 1) + c2 * VP(i + 2)) +
                 bp[1] * (c2 * VP(i - 1) + c1 * VP(i) + c0 * VP(i + 1)) +
                 bp[0] * (c0 * VP(i - 2) + c3 * VP(i - 1) + c4 * VP(i));
      R vplus = bm[2] * (c0 * VM(i + 1) + c1 * VM(i) + c2 * VM(i - 1)) +
                bm[1] * (c2 * VM(i + 2) + c1 * VM(i + 1) + c0 * VM(i)) +
                bm[0] * (c0 * VM(i + 3) + c3 * VM(i + 2) + c4 * VM(i + 1));
      return vminus + vplus;
    }
  }
  if constexpr (WS >= 4) {
    if (ord == 4) {
      const R dwe[4] = {R(1.0) / R(35.0), R(12.0) / R(35.0), R(18.0) / R(35.0), R(4.0) / R(35.0)};
      const R d1 = R(1.0) / R(36.0), d2 = R(13.0) / R(12.0), d3 = R(781.0) / R(720.0);
      auto sq = [](R a) { return a * a; };
      R bp[4], bm[4];
      bp[3] = d1 * sq(-11 * VP(i) + 18 * VP(i + 1) - 9 * VP(i + 2) + 2 * VP(i + 3)) +
              d2 * sq(2 * VP(i) - 5 * VP(i + 1) + 4 * VP(i + 2) - VP(i + 3)) +
              d3 * sq(-VP(i) + 3 * VP(i + 1) - 3 * VP(i + 2) + VP(i + 3));
      bp[2] = d1 * sq(-2 * VP(i - 1) - 3 * VP(i) + 6 * VP(i + 1) - VP(i + 2)) +
              d2 * sq(VP(i - 1) - 2 * VP(i) + VP(i + 1)) + d3 * sq(-VP(i - 1) + 3 * VP(i) - 3 * VP(i + 1) + VP(i + 2));
      bp[1] = d1 * sq(VP(i - 2) - 6 * VP(i - 1) + 3 * VP(i) + 2 * VP(i + 1)) +
              d2 * sq(VP(i - 1) - 2 * VP(i) + VP(i + 1)) + d3 * sq(-VP(i - 2) + 3 * VP(i - 1) - 3 * VP(i) + VP(i + 1));
      bp[0] = d1 * sq(-2 * VP(i - 3) + 9 * VP(i - 2) - 18 * VP(i - 1) + 11 * VP(i)) +
              d2 * sq(-VP(i - 3) + 4 * VP(i - 2) - 5 * VP(i - 1) + 2 * VP(i)) +
              d3 * sq(-VP(i - 3) + 3 * VP(i - 2) - 3 * VP(i - 1) + VP(i));
      bm[3] = d1 * sq(-11 * VM(i + 1) + 18 * VM(i) - 9 * VM(i - 1) + 2 * VM(i - 2)) +
              d2 * sq(2 * VM(i + 1) - 5 * VM(i) + 4 * VM(i - 1) - VM(i - 2)) +
              d3 * sq(-VM(i + 1) + 3 * VM(i) - 3 * VM(i - 1) + VM(i - 2));
      bm[2] = d1 * sq(-2 * VM(i + 2) - 3 * VM(i + 1) + 6 * VM(i) - VM(i - 1)) +
              d2 * sq(VM(i + 2) - 2 * VM(i + 1) + VM(i)) + d3 * sq(-VM(i + 2) + 3 * VM(i + 1) - 3 * VM(i) + VM(i - 1));
      bm[1] = d1 * sq(VM(i + 3) - 6 * VM(i + 2) + 3 * VM(i + 1) + 2 * VM(i)) +
              d2 * sq(VM(i + 2) - 2 * VM(i + 1) + VM(i)) + d3 * sq(-VM(i + 3) + 3 * VM(i + 2) - 3 * VM(i + 1) + VM(i));
      bm[0] = d1 * sq(-2 * VM(i + 4) + 9 * VM(i + 3) - 18 * VM(i + 2) + 11 * VM(i + 1)) +
              d2 * sq(-VM(i + 4) + 4 * VM(i + 3) - 5 * VM(i + 2) + 2 * VM(i + 1)) +
              d3 * sq(-VM(i + 4) + 3 * VM(i + 3) - 3 * VM(i + 2) + VM(i + 1));
      R sump = R(0), summ = R(0);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        bp[l] = betascale * bp[l];
        bm[l] = betascale * bm[l];
      }
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        R tp = eps6 + bp[l], tm = eps6 + bm[l];
        bp[l] = dwe[l] / (tp * tp);
        bm[l] = dwe[l] / (tm * tm);
        sump = sump + bp[l];
        summ = summ + bm[l];
      }
      const R rsp = fdiv(R(1), sump), rsm = fdiv(R(1), summ);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        bp[l] = bp[l] * rsp;
        bm[l] = bm[l] * rsm;
      }
      R vminus = bp[3] * (6 * VP(i) + 26 * VP(i + 1) - 10 * VP(i + 2) + 2 * VP(i + 3)) +
                 bp[2] * (-2 * VP(i - 1) + 14 * VP(i) + 14 * VP(i + 1) - 2 * VP(i + 2)) +
                 bp[1] * (2 * VP(i - 2) - 10 * VP(i - 1) + 26 * VP(i) + 6 * VP(i + 1)) +
                 bp[0] * (-6 * VP(i - 3) + 26 * VP(i - 2) - 46 * VP(i - 1) + 50 * VP(i));
      R vplus = bm[3] * (6 * VM(i + 1) + 26 * VM(i) - 10 * VM(i - 1) + 2 * VM(i - 2)) +
                bm[2] * (-2 * VM(i + 2) + 14 * VM(i + 1) + 14 * VM(i) - 2 * VM(i - 1)) +
                bm[1] * (2 * VM(i + 3) - 10 * VM(i + 2) + 26 * VM(i + 1) + 6 * VM(i)) +
                bm[0] * (-6 * VM(i + 4) + 26 * VM(i + 3) - 46 * VM(i + 2) + 50 * VM(i + 1));
      return (vminus + vplus) / R(24);
    }
  }
  return R(0);
}

// One side of wenorec_1d (kernels_cpu.F90:2526-2724): v[0 .. 2WS-2] in upwind order (the upwind cell
// of the face at v[WS-1]), eps2 = 1e-6 over the reference's scale of the smoothness indicators, zs as
// weno_rec says.  The side's value is base + num/den.
// The indicators and candidates are written in first and second differences d, s of the points:
// beta_k = 13/12 s_k^2 + 1/4 b_k^2 with b_k = 3 d - d', d + d', d' - 3 d, and the candidates share
// the upwind cell and d1/2; the weights' common factors (1/4 of the indicators, 1/10 of the weights)
// cancel.  With the projection of weno_flux a face of the FP64 y pass executes 880 FP64 instructions
// (central faces of its warp included) where the point values, with the fluxes projected beside the
// states and IEEE quotients, took 1415.
// FULL: order WS, in straight-line code that the two sides and the fields share the schedule of
// (1024x256x192, ms per step: 48.1 against 49.0 with the order chosen at run time in every side);
// otherwise a lower one, ord, next to a boundary.
template <int WS, bool WZ, bool FULL>
__device__ __forceinline__ void weno_side(const double (&v)[2 * WS - 1], int ord, double eps2, double zs, double& base,
                                          double& num, double& den) {
  using R = double;
  constexpr int c = WS - 1;
  base = v[c];
  num = R(0);
  den = R(1);
  if (!FULL && ord == 1) return;
  if constexpr (FULL ? WS == 3 : WS > 3) {
    if (FULL || ord == 3) {
      const R d0 = v[c - 1] - v[c - 2], d1 = v[c] - v[c - 1], d2 = v[c + 1] - v[c], d3 = v[c + 2] - v[c + 1];
      const R s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2;
      const R b0 = R(3) * d1 - d0, b1 = d1 + d2, b2 = d3 - R(3) * d2;
      const R k = R(13.0 / 3.0);
      R n0, n1, n2;
      if constexpr (!WZ) {
        const R eps = R(4) * eps2;
        const R e0 = b0 * b0 + ((k * s0) * s0 + eps), e1 = b1 * b1 + ((k * s1) * s1 + eps),
                e2 = b2 * b2 + ((k * s2) * s2 + eps);
        // omega_k = (d_k/e_k^2) / sum, written over the common denominator
        const R p12 = e1 * e2, p02 = e0 * e2, p01 = e0 * e1;
        n0 = p12 * p12;
        n1 = R(6) * (p02 * p02);
        n2 = p01 * p01;
      } else {
        // WENO-Z, omega_k = d_k (beta_k + tau)/(beta_k + eps); eps is a single-precision literal in
        // the reference.  The factors are scaled by zs where they are summed, which costs and rounds nothing.
        const R eps = R(4.0 * static_cast<double>(1.e-35f) / 0.000001) * eps2 * zs;
        const R e0 = b0 * b0 + (k * s0) * s0, e1 = b1 * b1 + (k * s1) * s1, e2 = b2 * b2 + (k * s2) * s2;
        const R tau = fma(fabs(e0 - e2), zs, eps);
        const R f0 = fma(e0, zs, eps), f1 = fma(e1, zs, eps), f2 = fma(e2, zs, eps);
        n0 = fma(e0, zs, tau) * (f1 * f2);
        n1 = R(6) * (fma(e1, zs, tau) * (f0 * f2));
        n2 = fma(e2, zs, tau) * (f0 * f1);
      }
      // sum of the weights (n2's factor 3 apart), and of the candidates less base = v[c] + d1/2, which
      // are s0/3, s1/3 and s1/2 - s2/6
      den = R(3) * n2 + (n0 + n1);
      num = (n0 * s0 + n1 * s1) + (R(1.5) * n2) * (R(3) * s1 - s2);
      base = R(0.5) * d1 + base;
      num = num * R(1.0 / 3.0);
      return;
    }
  }
  if constexpr (FULL ? WS == 2 : WS > 2) {
    if (FULL || ord == 2) {
      const R d1 = v[c] - v[c - 1], d2 = v[c + 1] - v[c];
      const R e0 = d1 * d1 + eps2, e1 = d2 * d2 + eps2;
      const R n0 = e1 * e1, n1 = R(2) * (e0 * e0);
      den = n0 + n1;
      num = R(0.5) * (n0 * d1 + n1 * d2);
      return;
    }
  }
  if constexpr (FULL && WS == 4) {
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
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const R e = b[l] + eps2;
      b[l] = dw[l] / (e * e);
    }
    den = b[0] + b[1] + b[2] + b[3];
    base = R(0);
    num = (b[3] * (6 * a3 + 26 * a4 - 10 * a5 + 2 * a6) + b[2] * (-2 * a2 + 14 * a3 + 14 * a4 - 2 * a5) +
           b[1] * (2 * a1 - 10 * a2 + 26 * a3 + 6 * a4) + b[0] * (-6 * a0 + 26 * a1 - 46 * a2 + 50 * a3)) *
          R(1.0 / 24.0);
  }
}
// wenorec_1d of one variable in FP64: the two sides of the face, p in upwind order from the left, m
// from the right, with one reciprocal for both.  The product of the denominators must stay above 2.2e-308
// where neither side has differences: it is then 100 e^8 for WENO-JS, e = 4 eps2, and 100 e^6 for WENO-Z,
// e = 4e-29 eps2 zs.  With eps2 = 1e-6 rho0^2 u0^2 (the mass flux, entropy and acoustic fields; rho0 = 1)
// that holds for u0 above 3e-9; with u0^4 (momentum fluxes, shear fields) it holds for WENO-JS above 5e-9,
// and for WENO-Z by the power of two zs next to 1/(rho0^2 u0^4) (without it above 5e-5 only); an energy
// flux (u0^6) comes scaled to order 1 by a power of two (else above 3e-6 and 1.4e-3 only).
template <int WS, bool WZ, bool FULL>
__device__ __forceinline__ double weno_rec(const double (&p)[2 * WS - 1], const double (&m)[2 * WS - 1], int ord,
                                           double eps2, double zs) {
  double bp, np, dp, bm, nm, dm;
  weno_side<WS, WZ, FULL>(p, ord, eps2, zs, bp, np, dp);
  weno_side<WS, WZ, FULL>(m, ord, eps2, zs, bm, nm, dm);
  return (bp + bm) + (np * dm + nm * dp) * rcp_pos(dp * dm);
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
      const double cl = double(R(g.coeff[lmax - 1][l - 1]));
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

// A thread's own values in shared memory, st values apart.  FP64 goes by volatile accesses, for the
// same reason as the ring's.
template <class R>
struct Scr {
  R* p;
  int st;
};
__device__ __forceinline__ void scr_put(const Scr<double>& s, int q, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(s.p + q * s.st)), "d"(v));
}
__device__ __forceinline__ double scr_get(const Scr<double>& s, int q) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"((unsigned)__cvta_generic_to_shared(s.p + q * s.st)));
  return v;
}
// values of a thread's scratch: state and flux of the stencil's points on the two acoustic fields
// (FP64), the split values of all fields (FP32)
template <class R, int WS>
constexpr int scr_vals() { return sizeof(R) == sizeof(double) ? 8 * WS : 10 * (2 * WS - 1); }

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
template <int DIR, int WS, int S, bool TP, bool WZ, bool FULL, class LN>
__device__ __forceinline__ void weno_flux(const Geom& g, const LN& ln, int ord, double (&f)[5], const Scr<double>& scr) {
  using R = double;
  constexpr int NP = 2 * WS - 1;
  const R rgas0 = R(g.rgas0);
  constexpr int t1 = DIR == 0 ? 1 : 0;
  constexpr int t2 = DIR == 2 ? 1 : 2;
  constexpr int q0 = S - WS;  // the first point used
  // Roe average of the two points adjacent to the face
  R vel[3], h, r, rp1;
  {
    const R ra = ln(0, S - 1), rb = ln(0, S);
    r = rb * rsqrt_pos(ra * rb);  // sqrt(rb/ra)
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
    const R tt = g.t0 + hbar * g.rcp0;
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
    const R cs = ln(F_C, q0 + l);  // the aux pass's sound speed
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
  // right.
  R fi[5];
  // the two shear fields
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int t = m == 0 ? t1 : t2;
    R gp[NP], gm[NP];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const R P = ln(0, q0 + l) * (ln(1 + t, q0 + l) - vel[t]), T = ln(1 + DIR, q0 + l) * P;
      if (l < 2 * WS - 1) gp[l] = T + ev1 * P;
      if (l > 0) gm[2 * WS - 1 - l] = T - ev1 * P;
    }
    fi[2 + m] = weno_rec<WS, WZ, FULL>(gp, gm, ord, g.weps_b * 4.0, g.wzs_b) * 0.5;
  }
  // the entropy field, and P_m(U) and T_m = P_m(F) of the two acoustic ones (g+- = T +- lambda P)
  const R epsa = g.weps_a;
  {
    R gp[NP], gm[NP];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const int q = q0 + l;
      const R rr = ln(0, q), rt = ln(5, q) * rgas0;
      const R vq[3] = {ln(1, q), ln(2, q), ln(3, q)};
      const R un = vq[DIR], dn = vel[DIR] - un, pp = rr * rt;
      const R de = (ln(4, q) - rt) - (vel[0] * vq[0] + vel[1] * vq[1] + vel[2] * vq[2]);
      const R sv = rr * (b2 * de + b1);
      const R av = ci * (rr * dn);
      const R ps = (pp * b2) * dn, pc = pp * ci;
      const R A = sv + av, B = sv - av, E = rr - sv;
      scr_put(scr, 4 * l, A);
      scr_put(scr, 4 * l + 1, un * A - (ps + pc));
      scr_put(scr, 4 * l + 2, B);
      scr_put(scr, 4 * l + 3, un * B + (pc - ps));
      const R T = un * E + ps;
      if (l < 2 * WS - 1) gp[l] = T + ev1 * E;
      if (l > 0) gm[2 * WS - 1 - l] = T - ev1 * E;
    }
    fi[1] = weno_rec<WS, WZ, FULL>(gp, gm, ord, epsa * 4.0, 1.0) * 0.5;
  }
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const R lam = m == 0 ? ev0 : ev4;
    R gp[NP], gm[NP];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const R P = scr_get(scr, 4 * l + 2 * m), T = scr_get(scr, 4 * l + 2 * m + 1);
      if (l < 2 * WS - 1) gp[l] = T + lam * P;
      if (l > 0) gm[2 * WS - 1 - l] = T - lam * P;
    }
    fi[4 * m] = weno_rec<WS, WZ, FULL>(gp, gm, ord, epsa * 16.0, 1.0) * 0.25;
  }
  // back-projection with the right eigenvectors, er(m,:) = (1, u - c n, h - vn c) for m = 1,
  // (1, u, b3) for m = 2, (0, e_t, v_t) for m = 3, 4, (1, u + c n, h + vn c) for m = 5
  const double fa = fi[0] + fi[4], fd = c * (fi[4] - fi[0]);
  f[0] = fa + fi[1];
#pragma unroll
  for (int d = 0; d < 3; ++d) f[1 + d] = vel[d] * f[0] + (d == DIR ? fd : (d == t1 ? fi[2] : fi[3]));
  f[4] = h * fa + vel[DIR] * fd + b3 * fi[1] + vel[t1] * fi[2] + vel[t2] * fi[3];
}

// The same flux in the mixed form's FP32: the states and the fluxes projected separately and the
// point-value reconstruction (wenorec), the field loop rolled over the split values in the thread's
// scratch; the back-projection in FP64.
template <int DIR, int WS, int S, bool WZ, class LN>
__device__ __forceinline__ void weno_flux_f(const Geom& g, const LN& ln, int ord, double (&f)[5], const Scr<float>& scr) {
  using R = float;
  R* gs = scr.p;
  const int gstride = scr.st;
  const R rgas0 = R(g.rgas0);
  const int o0 = S - 1, o1 = S;  // the two points adjacent to the face
  // Roe average
  R uu = ln(1, o0), vv = ln(2, o0), ww = ln(3, o0), h = ln(4, o0);
  R r = fdiv(ln(0, o1), ln(0, o0));
  r = fsqrt_pos(r);
  R rho = r * ln(0, o0);
  R rp1 = fdiv(R(1), r + R(1));
  uu = (r * ln(1, o1) + uu) * rp1;
  vv = (r * ln(2, o1) + vv) * rp1;
  ww = (r * ln(3, o1) + ww) * rp1;
  h = (r * ln(4, o1) + h) * rp1;
  R qq = R(0.5) * (uu * uu + vv * vv + ww * ww);
  R hbar = h - qq - R(g.cp_last) * R(g.t0);
  const R tt = R(g.t0) + fdiv(hbar, R(g.cp0));
  const R gamloc = R(g.gamloc);
  R cc = gamloc * tt * rgas0;
  R c, ci, b1, b2, b3;
  const R p_rho = tt * rgas0;
  const R etot = h - tt * rgas0;
  ci = rsqrt(cc);
  c = cc * ci;
  const R ci2 = ci * ci;
  b2 = R(g.gm1) * ci2;
  b1 = p_rho * ci2 - b2 * (etot - R(2) * qq);
  b3 = etot - p_rho * R(g.rgm1);
  const R vn = DIR == 0 ? uu : (DIR == 1 ? vv : ww);
  constexpr int t1 = DIR == 0 ? 1 : 0;
  constexpr int t2 = DIR == 2 ? 1 : 2;
  // stencil maximum of the characteristic speeds (offsets -WS+1 .. WS)
  R ev0 = R(-1), ev1 = R(-1), ev4 = R(-1);
#pragma unroll
  for (int l = 0; l < 2 * WS; ++l) {
    const int q = l + S - WS;
    const R vnq = ln(1 + DIR, q);
    const R gq = R(g.gamloc);
    const R cs = fsqrt_pos(gq * R(g.rgas0) * ln(5, q));
    ev0 = fmax(fabs(vnq - cs), ev0);
    ev1 = fmax(fabs(vnq), ev1);
    ev4 = fmax(fabs(vnq + cs), ev4);
  }
  const R betascale_a = R(g.wbs_a), betascale_b = R(g.wbs_b);
  // Projection of the stencil's conserved states U and fluxes F onto the five characteristic
  // fields, point by point, using the structure of the left eigenvectors (the reference forms
  // the five dot products el(:,m).U one field at a time): with dq = Roe velocity . X(2:4),
  // s = b1 X1 + b2 (X5 - dq) and a = ci (vn X1 - X(normal momentum)),
  //   P1 = (s + a)/2, P2 = X1 - s, P3 = X(t1) - v_t1 X1, P4 = X(t2) - v_t2 X1, P5 = (s - a)/2.
  // The split values g+- = (P(F) +- lambda_m P(U))/2 of every point and field go to this
  // thread's scratch.  wenorec_1d reads g+ at the points l = 1 .. 2WS-1 and g- at l = 2 .. 2WS
  // whatever its order (vp(i-WS+1 .. i+WS-1), vm(i-WS+2 .. i+WS) with i = WS), so each side keeps
  // 2WS-1 values: gs[((m*(2WS-1) + l)*2 + side) * gstride], l counted from the first point used.
  const R lam[5] = {ev0, ev1, ev1, ev1, ev4};
  const R vel[3] = {uu, vv, ww};
#pragma unroll
  for (int l = 0; l < 2 * WS; ++l) {
    const int q = l + S - WS;
    const R rr = ln(0, q), u1 = ln(1, q), v1 = ln(2, q), w1 = ln(3, q), h1 = ln(4, q);
    const R vq[3] = {u1, v1, w1};
    const R rhovn = rr * vq[DIR];
    const R pp = rr * ln(5, q) * rgas0;
    R U[5], F[5];
    U[0] = rr; U[1] = rr * u1; U[2] = rr * v1; U[3] = rr * w1; U[4] = rr * h1 - pp;
    F[0] = rhovn; F[1] = u1 * rhovn; F[2] = v1 * rhovn; F[3] = w1 * rhovn; F[4] = h1 * rhovn;
    F[1 + DIR] = F[1 + DIR] + pp;
    R PU[5], PF[5];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const R* X = side == 0 ? U : F;
      R* P = side == 0 ? PU : PF;
      const R dq = uu * X[1] + vv * X[2] + ww * X[3];
      const R sv = b1 * X[0] + b2 * (X[4] - dq);
      const R av = ci * (vn * X[0] - X[1 + DIR]);
      P[0] = R(0.5) * (sv + av);
      P[1] = X[0] - sv;
      P[2] = X[1 + t1] - vel[t1] * X[0];
      P[3] = X[1 + t2] - vel[t2] * X[0];
      P[4] = R(0.5) * (sv - av);
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const R cm = R(0.5) * (PF[m] + lam[m] * PU[m]);
      if (l < 2 * WS - 1) gs[((m * (2 * WS - 1) + l) * 2) * gstride] = cm;
      if (l > 0) gs[((m * (2 * WS - 1) + l - 1) * 2 + 1) * gstride] = PF[m] - cm;
    }
  }
  // reconstruction, one characteristic field per iteration (rolled: one copy of wenorec)
  R fi[5];
#pragma unroll 1
  for (int m = 0; m < 5; ++m) {
    R gp[2 * WS], gm[2 * WS];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      gp[l] = l < 2 * WS - 1 ? gs[((m * (2 * WS - 1) + l) * 2) * gstride] : R(0);
      gm[l] = l > 0 ? gs[((m * (2 * WS - 1) + l - 1) * 2 + 1) * gstride] : R(0);
    }
    const R bs = (m == 2 || m == 3) ? betascale_b : betascale_a;
    const R f = wenorec<WS>(gp, gm, ord, WZ ? 1 : 0, bs);
#pragma unroll
    for (int mm = 0; mm < 5; ++mm)
      if (mm == m) fi[mm] = f;
  }
  const double F0 = fi[0], F1 = fi[1], F2 = fi[2], F3 = fi[3], F4 = fi[4];
  f[0] = (F0 + F4) + F1;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    f[1 + d] = double(vel[d]) * f[0] + (d == DIR ? double(c) * (F4 - F0) : (d == t1 ? F2 : F3));
  f[4] = double(h - vn * c) * F0 + double(b3) * F1 + double(vel[t1]) * F2 + double(vel[t2]) * F3 + double(h + vn * c) * F4;
}

// Rusanov (component-wise local Lax-Friedrichs) WENO flux of the *_hybrid_rusanov kernels
// (kernels_cpu.F90:692-941 for x, same in y and z): stencil maximum of |u_n -+ c|, split
// values of the conserved fluxes, wenorec with the scales of wenorec_1d_rusanov (:2325-2523).
template <class R, int DIR, int WS, int S, bool TP, bool WZ, bool FULL, class LN>
__device__ __forceinline__ void rusanov_flux(const Geom& g, const LN& ln, int ord, double (&f)[5]) {
  static_assert(!TP || sizeof(R) == sizeof(double), "the thermally perfect gas is an FP64 path");
  constexpr int q0 = S - WS;
  const R rgas0 = R(g.rgas0);
  R evmax = R(-1);
#pragma unroll
  for (int l = 0; l < 2 * WS; ++l) {
    const R un = ln(1 + DIR, q0 + l);
    R c;
    if constexpr (sizeof(R) == sizeof(double)) {
      c = ln(F_C, q0 + l);
    } else {
      const R gq = R(g.gamloc);
      c = fsqrt_pos(gq * rgas0 * ln(5, q0 + l));
    }
    evmax = max_of(max_of(fabs(un - c), fabs(un + c)), evmax);
  }
#pragma unroll 1
  for (int m = 0; m < 5; ++m) {
    R gp[2 * WS], gm[2 * WS];
#pragma unroll
    for (int l = 0; l < 2 * WS; ++l) {
      const int q = q0 + l;
      const R rho = ln(0, q), h = ln(4, q);
      const R vel[3] = {ln(1, q), ln(2, q), ln(3, q)};
      const R rhou = rho * vel[DIR];
      const R pp = rho * ln(5, q) * rgas0;
      const R rhoevm = rho * evmax;
      R evm, c;
      if (m == 0) {
        evm = rhou;
        c = R(0.5) * (evm + rhoevm);
      } else if (m == 4) {
        R hs = h, ps = pp;
        if constexpr (sizeof(R) == sizeof(double)) {  // scaled for weno_rec
          hs = g.wsc_c * h;
          ps = g.wsc_c * pp;
        }
        evm = hs * rhou;
        c = R(0.5) * (evm + evmax * (rho * hs - ps));
      } else {
        const R vd = m == 1 ? vel[0] : (m == 2 ? vel[1] : vel[2]);
        evm = vd * rhou;
        if (m == 1 + DIR) evm = evm + pp;
        c = R(0.5) * (evm + rhoevm * vd);
      }
      gp[l] = c;
      gm[l] = evm - c;
    }
    R v;
    if constexpr (sizeof(R) == sizeof(double)) {
      R p[2 * WS - 1], q[2 * WS - 1];
#pragma unroll
      for (int l = 0; l < 2 * WS - 1; ++l) {
        p[l] = gp[l];
        q[l] = gm[2 * WS - 1 - l];
      }
      v = weno_rec<WS, WZ, FULL>(p, q, ord, m == 0 ? g.weps_a : (m == 4 ? g.weps_c : g.weps_b),
                                 m == 0 || m == 4 ? 1.0 : g.wzs_b);
      if (m == 4) v = v * g.wsr_c;
    } else {
      v = wenorec<WS>(gp, gm, ord, WZ ? 1 : 0, m == 0 ? R(g.wbs_a) : (m == 4 ? R(g.wbs_c) : R(g.wbs_b)));
    }
#pragma unroll
    for (int mm = 0; mm < 5; ++mm)
      if (mm == m) f[mm] = double(v);
  }
}

}  // namespace sb200
