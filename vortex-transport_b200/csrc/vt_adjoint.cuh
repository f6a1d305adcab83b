// Derivatives of the pointwise pieces of the right-hand side, for the
// discrete adjoint and the tangent-linear model:
//
//   roe_flux2_vjp        reverse sweep of roe_flux2 (vt_device.cuh): given the
//                        adjoint of the doubled flux, the adjoints of both
//                        states, through the Roe averages, the c2^2 "sound
//                        speed" and the entropy fix (Numericalflux.cpp:99-156);
//   contravariant_vjp    reverse sweep of contravariant_flux (the nodal Euler
//                        flux of Timestepping.cpp:141-158 contracted with J^-1);
//   roe_flux2_jvp,
//   contravariant_jvp    their derivatives along a direction, for the
//                        tangent-linear model;
//   Dual<N>, roe_flux_t  the flux on dual numbers, the independent check of
//                        both (on the host).
//
// All functions are __host__ __device__ so the reverse sweeps can be checked
// against the dual-number Jacobians on the CPU.
#pragma once

#include <cmath>

#include "vt_device.cuh"

namespace vt {

// 1/x: recip_nr (vt_device.cuh) in device code, IEEE division on the host, where
// the reverse sweeps are checked against the dual-number Jacobians.
__host__ __device__ inline double rcp(double x) {
#ifdef __CUDA_ARCH__
  return recip_nr(x);
#else
  return 1.0 / x;
#endif
}

// 1/sqrt(x), likewise: rsqrt_nr on the device, IEEE operations on the host.
__host__ __device__ inline double rsq(double x) {
#ifdef __CUDA_ARCH__
  return rsqrt_nr(x);
#else
  return 1.0 / sqrt(x);
#endif
}

// ---- dual numbers -------------------------------------------------------------
template <int N>
struct Dual {
  double v;
  double d[N];
  __host__ __device__ Dual() : v(0.0) {
    for (int i = 0; i < N; ++i) d[i] = 0.0;
  }
  __host__ __device__ Dual(double x) : v(x) {  // NOLINT: constants promote
    for (int i = 0; i < N; ++i) d[i] = 0.0;
  }
};

template <int N>
__host__ __device__ inline Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v + b.v;
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] + b.d[i];
  return r;
}
template <int N>
__host__ __device__ inline Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v - b.v;
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] - b.d[i];
  return r;
}
template <int N>
__host__ __device__ inline Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  r.v = a.v * b.v;
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
  return r;
}
template <int N>
__host__ __device__ inline Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r;
  const double ib = 1.0 / b.v;
  r.v = a.v * ib;
  for (int i = 0; i < N; ++i) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
  return r;
}
template <int N>
__host__ __device__ inline Dual<N> operator+(const Dual<N>& a, double b) { return a + Dual<N>(b); }
template <int N>
__host__ __device__ inline Dual<N> operator+(double a, const Dual<N>& b) { return Dual<N>(a) + b; }
template <int N>
__host__ __device__ inline Dual<N> operator-(const Dual<N>& a, double b) { return a - Dual<N>(b); }
template <int N>
__host__ __device__ inline Dual<N> operator-(double a, const Dual<N>& b) { return Dual<N>(a) - b; }
template <int N>
__host__ __device__ inline Dual<N> operator-(const Dual<N>& a) { return Dual<N>(0.0) - a; }
template <int N>
__host__ __device__ inline Dual<N> operator*(const Dual<N>& a, double b) {
  Dual<N> r;
  r.v = a.v * b;
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b;
  return r;
}
template <int N>
__host__ __device__ inline Dual<N> operator*(double a, const Dual<N>& b) { return b * a; }
template <int N>
__host__ __device__ inline Dual<N> operator/(double a, const Dual<N>& b) { return Dual<N>(a) / b; }
template <int N>
__host__ __device__ inline Dual<N> dsqrt(const Dual<N>& a) {
  Dual<N> r;
  r.v = sqrt(a.v);
  const double h = 0.5 / r.v;
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * h;
  return r;
}
template <int N>
__host__ __device__ inline Dual<N> dabs(const Dual<N>& a) { return a.v < 0 ? -a : a; }
template <int N>
__host__ __device__ inline double val(const Dual<N>& a) { return a.v; }
__host__ __device__ inline double val(double a) { return a; }
__host__ __device__ inline double dsqrt(double a) { return sqrt(a); }
__host__ __device__ inline double dabs(double a) { return fabs(a); }

// ---- forward formulas on any scalar type ------------------------------------------
template <typename T>
__host__ __device__ inline int roe_flux_t(const T* uL, const T* uR, double nx, double ny, T* f) {
  const T rL = uL[0], rR = uR[0];
  const T irLR = 1.0 / (rL * rR);
  const T irL = rR * irLR, irR = rL * irLR;
  const T vxL = uL[1] * irL, vyL = uL[2] * irL;
  const T unL = vxL * nx + vyL * ny;
  const T pL = kGm1 * (uL[3] - 0.5 * (uL[1] * vxL + uL[2] * vyL));
  int code = 0;
  if ((val(pL) <= 0) || (val(rL) <= 0)) code = 1;
  const T rHL = uL[3] + pL;
  const T HL = rHL * irL;
  const T vxR = uR[1] * irR, vyR = uR[2] * irR;
  const T unR = vxR * nx + vyR * ny;
  const T pR = kGm1 * (uR[3] - 0.5 * (uR[1] * vxR + uR[2] * vyR));
  if (code == 0 && ((val(pR) <= 0) || (val(rR) <= 0))) code = 2;
  const T rHR = uR[3] + pR;
  const T HR = rHR * irR;
  const T du0 = uR[0] - uL[0], du1 = uR[1] - uL[1], du2 = uR[2] - uL[2], du3 = uR[3] - uL[3];
  const T di = dsqrt(rR * irL);
  const T d1 = 1.0 / (1.0 + di);
  const T ui = (di * vxR + vxL) * d1;
  const T vi = (di * vyR + vyL) * d1;
  const T Hi = (di * HR + HL) * d1;
  const T af = 0.5 * (ui * ui + vi * vi);
  const T ucp = ui * nx + vi * ny;
  const T c2 = kGm1 * (Hi - af);
  if (code == 0 && val(c2) <= 0) code = 3;
  const T ci = c2 * c2;
  const T ci1 = 1.0 / ci;
  const T eps = 0.1 * ci;
  const T ieps = 10.0 * ci1;
  T l0 = ucp + ci, l1 = ucp - ci, l3 = ucp;
  l0 = val(dabs(l0)) < val(eps) ? 0.5 * (eps + l0 * l0 * ieps) : dabs(l0);
  l1 = val(dabs(l1)) < val(eps) ? 0.5 * (eps + l1 * l1 * ieps) : dabs(l1);
  l3 = val(dabs(l3)) < val(eps) ? 0.5 * (eps + l3 * l3 * ieps) : dabs(l3);
  const T s1 = 0.5 * (l0 + l1);
  const T s2 = 0.5 * (l0 - l1);
  const T G1 = kGm1 * (af * du0 - ui * du1 - vi * du2 + du3);
  const T G2 = -ucp * du0 + du1 * nx + du2 * ny;
  const T C1 = (G1 * (s1 - l3) * ci1 + G2 * s2) * ci1;
  const T C2 = G1 * s2 * ci1 + G2 * (s1 - l3);
  f[0] = 0.5 * ((uL[1] * nx + uL[2] * ny) + (uR[1] * nx + uR[2] * ny)) - 0.5 * (l3 * du0 + C1);
  f[1] = 0.5 * ((uL[1] * unL + pL * nx) + (uR[1] * unR + pR * nx)) - 0.5 * (l3 * du1 + C1 * ui + C2 * nx);
  f[2] = 0.5 * ((uL[2] * unL + pL * ny) + (uR[2] * unR + pR * ny)) - 0.5 * (l3 * du2 + C1 * vi + C2 * ny);
  f[3] = 0.5 * (rHL * unL + rHR * unR) - 0.5 * (l3 * du3 + C1 * Hi + C2 * ucp);
  return code;
}

// ---- reverse sweeps ------------------------------------------------------------------
// b: adjoint of roe_flux2's doubled flux (4); writes the adjoints of uL and uR
// to buL, buR. The reverse sweep of roe_flux2's own arrangement: about 190 FP64
// instructions, where the sweep of the flux written through both sides'
// velocities and enthalpies took about 360 (the reverse stage is bound by
// them: FP64 pipe 44% busy at two blocks per SM). What makes it short:
//   C1 = A / ci, G1 = (gamma-1) X / ci: the adjoint of 1/ci is needed only as
//     -(bA A + bG1 G1) / ci added to that of ci;
//   the averages x = (g xR + xL) / s with s = rhoL + w: the adjoint of s is
//     -sum (bx / s) x, and g = sqrt(rhoL/rhoR), w = sqrt(rhoL rhoR) have the
//     logarithmic derivatives -+ 1/2 and 1/2;
//   for |u_n| < 7/8 ci the acoustic part is (|l0| + |l1|)/2 = ci and
//     (|l0| - |l1|)/2 = u_n.
__host__ __device__ inline void roe_flux2_vjp(const double* uL, const double* uR, double nx, double ny,
                                              const double* b, double* buL, double* buR) {
  // forward
  const double rL = uL[0], rR = uR[0];
  const double rLR = rL * rR;
  const double y = rsq(rLR);
  const double irLR = y * y, w = rLR * y;
  const double irL = rR * irLR, irR = rL * irLR;
  const double unL = (uL[1] * nx + uL[2] * ny) * irL, unR = (uR[1] * nx + uR[2] * ny) * irR;
  const double kinL = (uL[1] * uL[1] + uL[2] * uL[2]) * irL, kinR = (uR[1] * uR[1] + uR[2] * uR[2]) * irR;
  const double rHL = uL[3] + kGm1 * (uL[3] - 0.5 * kinL), rHR = uR[3] + kGm1 * (uR[3] - 0.5 * kinR);
  const double du0 = rR - rL, du1 = uR[1] - uL[1], du2 = uR[2] - uL[2], du3 = uR[3] - uL[3];
  const double g = w * irR;
  const double d1 = rcp(rL + w);
  const double ui = (g * uR[1] + uL[1]) * d1, vi = (g * uR[2] + uL[2]) * d1, Hi = (g * rHR + rHL) * d1;
  const double h = 0.5 * (ui * ui + vi * vi);
  const double ucp = ui * nx + vi * ny;
  const double c2 = kGm1 * (Hi - h);
  const double ci = c2 * c2;
  const double ci1 = rcp(ci);
  const double t = ucp * ci1;
  // l3 with its derivatives by u_n and ci
  const bool fix = fabs(t) < 0.1;
  const double l3 = fix ? 5.0 * ucp * t + 0.05 * ci : fabs(ucp);
  const double l3u = fix ? 10.0 * t : (ucp < 0 ? -1.0 : 1.0);
  const double l3c = fix ? 0.05 - 5.0 * t * t : 0.0;
  const bool usual = fabs(t) < 0.875;
  double s1 = ci, s2 = ucp;  // (|l0| + |l1|)/2 and (|l0| - |l1|)/2
  double l0u = 1.0, l0c = 0.0, l1u = -1.0, l1c = 0.0;
  if (!usual) {
    const double l0r = ucp + ci, l1r = ucp - ci, eps = 0.1 * ci;
    double l0 = fabs(l0r), l1 = fabs(l1r);
    l0u = l0r < 0 ? -1.0 : 1.0;
    l1u = l1r < 0 ? -1.0 : 1.0;
    if (l0 < eps) {
      const double z = l0r * ci1;
      l0 = 5.0 * l0r * z + 0.05 * ci, l0u = 10.0 * z, l0c = 0.05 - 5.0 * z * z;
    }
    if (l1 < eps) {
      const double z = l1r * ci1;
      l1 = 5.0 * l1r * z + 0.05 * ci, l1u = 10.0 * z, l1c = 0.05 - 5.0 * z * z;
    }
    s1 = 0.5 * (l0 + l1);
    s2 = 0.5 * (l0 - l1);
  }
  const double s1l3 = s1 - l3;
  const double k1 = kGm1 * ci1;
  const double G1 = k1 * (h * du0 - ui * du1 - vi * du2 + du3);
  const double G2 = du1 * nx + du2 * ny - ucp * du0;
  const double A = G1 * s1l3 + G2 * s2;
  const double C1 = A * ci1;
  const double C2 = G1 * s2 + G2 * s1l3;

  // the flux's terms
  const double bn = b[1] * nx + b[2] * ny;  // adjoint of both pressures
  const double b_C2 = -(bn + b[3] * ucp);
  const double b_C1 = -(b[0] + b[1] * ui + b[2] * vi + b[3] * Hi);
  double b_l3 = -(b[0] * du0 + b[1] * du1 + b[2] * du2 + b[3] * du3);
  double b_ucp = -C2 * b[3], b_ui = -C1 * b[1], b_vi = -C1 * b[2], b_Hi = -C1 * b[3];
  const double b_A = b_C1 * ci1;
  const double b_G1 = b_A * s1l3 + b_C2 * s2, b_G2 = b_A * s2 + b_C2 * s1l3;
  const double b_s1 = b_A * G1 + b_C2 * G2, b_s2 = b_A * G2 + b_C2 * G1;
  double b_ci = -ci1 * (b_A * A + b_G1 * G1);
  b_l3 -= b_s1;
  if (usual) {
    b_ci += b_s1;
    b_ucp += b_s2;
  } else {
    const double b_l0 = 0.5 * (b_s1 + b_s2), b_l1 = 0.5 * (b_s1 - b_s2);
    b_ucp += b_l0 * l0u + b_l1 * l1u;
    b_ci += b_l0 * (l0u + l0c) + b_l1 * (l1c - l1u);
  }
  b_ucp += b_l3 * l3u;
  b_ci += b_l3 * l3c;
  const double b_X = k1 * b_G1;
  const double b_du0 = b_X * h - l3 * b[0] - b_G2 * ucp;
  const double b_du1 = b_G2 * nx - l3 * b[1] - b_X * ui;
  const double b_du2 = b_G2 * ny - l3 * b[2] - b_X * vi;
  const double b_du3 = b_X - l3 * b[3];
  b_ucp -= b_G2 * du0;
  // ci = c2^2, c2 = (gamma-1) (Hi - h), h = (ui^2 + vi^2)/2, u_n = ui nx + vi ny
  const double z = 2.0 * kGm1 * c2 * b_ci;
  b_Hi += z;
  const double b_h = b_X * du0 - z;
  b_ui += b_h * ui + b_ucp * nx - b_X * du1;
  b_vi += b_h * vi + b_ucp * ny - b_X * du2;
  // the averages
  const double ai = b_ui * d1, av = b_vi * d1, aH = b_Hi * d1;
  const double b_s = -(ai * ui + av * vi + aH * Hi);
  const double gg = 0.5 * g * (ai * uR[1] + av * uR[2] + aH * rHR), ws = 0.5 * w * b_s;
  // each side: rho H = rho E + p, p = (gamma-1) (rho E - kin/2), kin = |m|^2/rho, u_n = m.n/rho
  const double rhL = b[3] * unL + aH, rhR = b[3] * unR + g * aH;
  const double tL = kGm1 * (bn + rhL), tR = kGm1 * (bn + rhR);
  const double eL = (b[1] * uL[1] + b[2] * uL[2] + b[3] * rHL) * irL;
  const double eR = (b[1] * uR[1] + b[2] * uR[2] + b[3] * rHR) * irR;
  const double cL = b[0] + eL, cR = b[0] + eR, mL = tL * irL, mR = tR * irR;
  buL[0] = irL * (ws + gg + 0.5 * tL * kinL) - eL * unL + b_s - b_du0;
  buL[1] = cL * nx + b[1] * unL + ai - mL * uL[1] - b_du1;
  buL[2] = cL * ny + b[2] * unL + av - mL * uL[2] - b_du2;
  buL[3] = rhL + tL - b_du3;
  buR[0] = irR * (ws - gg + 0.5 * tR * kinR) - eR * unR + b_du0;
  buR[1] = cR * nx + b[1] * unR + g * ai - mR * uR[1] + b_du1;
  buR[2] = cR * ny + b[2] * unR + g * av - mR * uR[2] + b_du2;
  buR[3] = rhR + tR + b_du3;
}

// Derivative of roe_flux2's doubled flux along (dL, dR), in the same
// arrangement (names as in roe_flux2_vjp; d... are derivatives).
__host__ __device__ inline void roe_flux2_jvp(const double* uL, const double* uR, double nx, double ny, const double* dL,
                                              const double* dR, double* df) {
  const double rL = uL[0], rR = uR[0];
  const double rLR = rL * rR;
  const double y = rsq(rLR);
  const double irLR = y * y, w = rLR * y;
  const double irL = rR * irLR, irR = rL * irLR;
  const double unL = (uL[1] * nx + uL[2] * ny) * irL, unR = (uR[1] * nx + uR[2] * ny) * irR;
  const double kinL = (uL[1] * uL[1] + uL[2] * uL[2]) * irL, kinR = (uR[1] * uR[1] + uR[2] * uR[2]) * irR;
  const double rHL = uL[3] + kGm1 * (uL[3] - 0.5 * kinL), rHR = uR[3] + kGm1 * (uR[3] - 0.5 * kinR);
  const double dmL = dL[1] * nx + dL[2] * ny, dmR = dR[1] * nx + dR[2] * ny;
  const double dunL = (dmL - unL * dL[0]) * irL, dunR = (dmR - unR * dR[0]) * irR;
  const double dpL = kGm1 * (dL[3] - (uL[1] * dL[1] + uL[2] * dL[2] - 0.5 * kinL * dL[0]) * irL);
  const double dpR = kGm1 * (dR[3] - (uR[1] * dR[1] + uR[2] * dR[2] - 0.5 * kinR * dR[0]) * irR);
  const double drHL = dL[3] + dpL, drHR = dR[3] + dpR;
  const double du0 = rR - rL, du1 = uR[1] - uL[1], du2 = uR[2] - uL[2], du3 = uR[3] - uL[3];
  const double e0 = dR[0] - dL[0], e1 = dR[1] - dL[1], e2 = dR[2] - dL[2], e3 = dR[3] - dL[3];
  // averages
  const double g = w * irR, d1 = rcp(rL + w);
  const double lL = 0.5 * dL[0] * irL, lR = 0.5 * dR[0] * irR;  // halved logarithmic derivatives of the densities
  const double dg = g * (lL - lR), ds = dL[0] + w * (lL + lR);
  const double ui = (g * uR[1] + uL[1]) * d1, vi = (g * uR[2] + uL[2]) * d1, Hi = (g * rHR + rHL) * d1;
  const double dui = (dg * uR[1] + g * dR[1] + dL[1] - ui * ds) * d1;
  const double dvi = (dg * uR[2] + g * dR[2] + dL[2] - vi * ds) * d1;
  const double dHi = (dg * rHR + g * drHR + drHL - Hi * ds) * d1;
  const double h = 0.5 * (ui * ui + vi * vi), dh = ui * dui + vi * dvi;
  const double ucp = ui * nx + vi * ny, ducp = dui * nx + dvi * ny;
  const double c2 = kGm1 * (Hi - h), ci = c2 * c2, dci = 2.0 * c2 * kGm1 * (dHi - dh);
  const double ci1 = rcp(ci);
  const double t = ucp * ci1;
  const bool fix = fabs(t) < 0.1;
  const double l3 = fix ? 5.0 * ucp * t + 0.05 * ci : fabs(ucp);
  const double dl3 = fix ? 10.0 * t * ducp + (0.05 - 5.0 * t * t) * dci : (ucp < 0 ? -ducp : ducp);
  double s1 = ci, s2 = ucp, ds1 = dci, ds2 = ducp;
  if (!(fabs(t) < 0.875)) {
    const double l0r = ucp + ci, l1r = ucp - ci, eps = 0.1 * ci;
    double l0 = fabs(l0r), l1 = fabs(l1r);
    double dl0 = l0r < 0 ? -(ducp + dci) : ducp + dci, dl1 = l1r < 0 ? dci - ducp : ducp - dci;
    if (l0 < eps) {
      const double z = l0r * ci1;
      l0 = 5.0 * l0r * z + 0.05 * ci, dl0 = 10.0 * z * (ducp + dci) + (0.05 - 5.0 * z * z) * dci;
    }
    if (l1 < eps) {
      const double z = l1r * ci1;
      l1 = 5.0 * l1r * z + 0.05 * ci, dl1 = 10.0 * z * (ducp - dci) + (0.05 - 5.0 * z * z) * dci;
    }
    s1 = 0.5 * (l0 + l1), s2 = 0.5 * (l0 - l1);
    ds1 = 0.5 * (dl0 + dl1), ds2 = 0.5 * (dl0 - dl1);
  }
  const double S = s1 - l3, dS = ds1 - dl3, k1 = kGm1 * ci1;
  const double G1 = k1 * (h * du0 - ui * du1 - vi * du2 + du3);
  const double dG1 = k1 * (dh * du0 + h * e0 - dui * du1 - ui * e1 - dvi * du2 - vi * e2 + e3) - G1 * ci1 * dci;
  const double G2 = du1 * nx + du2 * ny - ucp * du0, dG2 = e1 * nx + e2 * ny - ducp * du0 - ucp * e0;
  const double C1 = (G1 * S + G2 * s2) * ci1;
  const double dC1 = (dG1 * S + G1 * dS + dG2 * s2 + G2 * ds2 - C1 * dci) * ci1;
  const double C2 = G1 * s2 + G2 * S, dC2 = dG1 * s2 + G1 * ds2 + dG2 * S + G2 * dS;
  const double dp = dpL + dpR - dC2;
  df[0] = dmL + dmR - dl3 * du0 - l3 * e0 - dC1;
  df[1] = dL[1] * unL + uL[1] * dunL + dR[1] * unR + uR[1] * dunR + dp * nx - dl3 * du1 - l3 * e1 - dC1 * ui - C1 * dui;
  df[2] = dL[2] * unL + uL[2] * dunL + dR[2] * unR + uR[2] * dunR + dp * ny - dl3 * du2 - l3 * e2 - dC1 * vi - C1 * dvi;
  df[3] = drHL * unL + rHL * dunL + drHR * unR + rHR * dunR - dl3 * du3 - l3 * e3 - dC1 * Hi - C1 * dHi - dC2 * ucp -
          C2 * ducp;
}

// Derivative of the contravariant flux of a node's state s along d.
__host__ __device__ inline void contravariant_jvp(const double* s, const double* d, double j00, double j01, double j10,
                                                  double j11, double* dgxi, double* dgeta) {
  const double ir = rcp(s[0]);
  const double vx = s[1] * ir, vy = s[2] * ir;
  const double dvx = (d[1] - vx * d[0]) * ir, dvy = (d[2] - vy * d[0]) * ir;
  const double rH = s[3] + kGm1 * (s[3] - 0.5 * (s[1] * vx + s[2] * vy));
  const double dp = kGm1 * (d[3] - 0.5 * (d[1] * vx + d[2] * vy + s[1] * dvx + s[2] * dvy));
  const double drH = d[3] + dp;
  const double vxi = j00 * vx + j01 * vy, veta = j10 * vx + j11 * vy;
  const double dvxi = j00 * dvx + j01 * dvy, dveta = j10 * dvx + j11 * dvy;
  dgxi[0] = j00 * d[1] + j01 * d[2];
  dgxi[1] = d[1] * vxi + s[1] * dvxi + j00 * dp;
  dgxi[2] = d[2] * vxi + s[2] * dvxi + j01 * dp;
  dgxi[3] = drH * vxi + rH * dvxi;
  dgeta[0] = j10 * d[1] + j11 * d[2];
  dgeta[1] = d[1] * veta + s[1] * dveta + j10 * dp;
  dgeta[2] = d[2] * veta + s[2] * dveta + j11 * dp;
  dgeta[3] = drH * veta + rH * dveta;
}

// bf: adjoint of the flux itself (4). Adds the adjoints of uL and uR to buL, buR.
__host__ __device__ inline void roe_flux_vjp(const double* uL, const double* uR, double nx, double ny,
                                             const double* bf, double* buL, double* buR) {
  const double b[4] = {0.5 * bf[0], 0.5 * bf[1], 0.5 * bf[2], 0.5 * bf[3]};
  double bl[4], br[4];
  roe_flux2_vjp(uL, uR, nx, ny, b, bl, br);
  for (int c = 0; c < 4; ++c) {
    buL[c] += bl[c];
    buR[c] += br[c];
  }
}

// bgxi, bgeta: adjoints of the contravariant flux (4 each); writes the state's adjoint to bs.
__host__ __device__ inline void contravariant_vjp(const double* s, double j00, double j01, double j10, double j11,
                                                  const double* bgxi, const double* bgeta, double* bs) {
  const double ir = rcp(s[0]);
  const double vx = s[1] * ir, vy = s[2] * ir;
  const double kin = s[1] * vx + s[2] * vy;
  const double rH = s[3] + kGm1 * (s[3] - 0.5 * kin);
  const double vxi = j00 * vx + j01 * vy, veta = j10 * vx + j11 * vy;
  // g[0] = rho v, g[1] = m1 v + j0 p, g[2] = m2 v + j1 p, g[3] = rho H v for v = vxi, veta
  const double b_vxi = bgxi[1] * s[1] + bgxi[2] * s[2] + bgxi[3] * rH;
  const double b_veta = bgeta[1] * s[1] + bgeta[2] * s[2] + bgeta[3] * rH;
  const double b_rH = bgxi[3] * vxi + bgeta[3] * veta;
  const double t = kGm1 * (bgxi[1] * j00 + bgxi[2] * j01 + bgeta[1] * j10 + bgeta[2] * j11 + b_rH);
  const double wxi = bgxi[0] + b_vxi * ir, weta = bgeta[0] + b_veta * ir;  // m.j = rho v
  bs[0] = ir * (0.5 * t * kin - b_vxi * vxi - b_veta * veta);
  bs[1] = wxi * j00 + weta * j10 + bgxi[1] * vxi + bgeta[1] * veta - t * vx;
  bs[2] = wxi * j01 + weta * j11 + bgxi[2] * vxi + bgeta[2] * veta - t * vy;
  bs[3] = b_rH + t;
}

}  // namespace vt
