// Device-side building blocks of the stepper: state layout, folded operators,
// Roe flux, nodal flux and the first-error record.
//
// HBM layout of a state vector (U, a stage, the RK accumulator): structure of
// arrays of double2, row r = 2*i + h for node i and component pair h
// (h = 0: rho, rho u; h = 1: rho v, rho E), element e in the column:
//   state[r * Kpad + e]
// A warp touching 32 consecutive elements of one row reads 512 contiguous
// bytes; one element's state is 2*Np 16-byte loads.
#pragma once

#include <cuda.h>

#include <cstdint>

namespace vt {

constexpr double kGamma = 1.4;
// (gamma - 1) exactly as the reference forms it (1.4 - 1.0 = 0.3999999999999999).
constexpr double kGm1 = 1.4 - 1.0;

__host__ __device__ constexpr int np_of_p(int p) { return (p + 1) * (p + 2) / 2; }

// Node numbering of Meshgeneration.cpp:208-216: j (eta) outer, i (xi) inner.
__host__ __device__ constexpr int node_id(int p, int i, int j) { return j * (p + 1) - j * (j - 1) / 2 + i; }

// k-th node (0..p) on side s of the reference triangle: s = 0 is the side
// eta = 0 (reference side 1), s = 1 is xi + eta = 1 (side 2), s = 2 is
// xi = 0 (side 3). Only these p + 1 basis functions are non-zero on the side.
__host__ __device__ constexpr int edge_node(int p, int s, int k) {
  return s == 0 ? node_id(p, k, 0) : (s == 1 ? node_id(p, p - k, k) : node_id(p, 0, k));
}

// Operators shared by all elements, folded on the host (vt_solver.cu):
//   D[0] = M_ref^-1 S_xi, D[1] = M_ref^-1 S_eta          (volume term)
//   lift[s][i][q] = sum_j M_ref^-1[i][j] phi+_s(q)_j w_q  (surface term)
//   tp[s][q][k], tm[s][q][k]: own / neighbour basis at face point q restricted
//   to the p + 1 nodes of side s.
// Passed by value as a kernel parameter, so every coefficient is an immediate
// constant-bank operand of the FMA that uses it.
template <int P, int NFQ>
struct StageOps {
  static constexpr int NP = np_of_p(P);
  static constexpr int NE = P + 1;
  double D[2][NP][NP];
  double lift[3][NP][NFQ];
  double tp[3][NFQ][NE];
  double tm[3][NFQ][NE];
};

// ---- the reflection xi <-> eta of the reference triangle ---------------------
// It maps node (i, j) to (j, i), side 0 onto side 2 and side 1 onto itself, the
// last two with the face points in reverse order, and swaps the two reference
// derivatives. The nodes fall into pairs and the fixed ones on the diagonal.
// fold_node(p, a) lists one node of each pair (a < fold_pairs), then the fixed
// ones (a < fold_nodes).
__host__ __device__ constexpr int fold_fixed(int p) { return p / 2 + 1; }
__host__ __device__ constexpr int fold_pairs(int p) { return (np_of_p(p) - fold_fixed(p)) / 2; }
__host__ __device__ constexpr int fold_nodes(int p) { return fold_pairs(p) + fold_fixed(p); }
__host__ __device__ constexpr int fold_node(int p, int a) {
  int n = 0;
  for (int fixed = 0; fixed < 2; ++fixed)
    for (int j = 0; j <= p; ++j)
      for (int i = fixed ? j : j + 1; i + j <= p && (!fixed || i == j); ++i)
        if (n++ == a) return node_id(p, i, j);
  return 0;
}
__host__ __device__ constexpr int mirror_node(int p, int node) {
  for (int j = 0; j <= p; ++j)
    for (int i = 0; i + j <= p; ++i)
      if (node_id(p, i, j) == node) return node_id(p, j, i);
  return node;
}

// StageOps split into the parts that are even and odd under the reflection
// (fold_operators, vt_stage_inst.cuh). With Pj the mirror image of node j and
// r_i the residual of node i, the even part e_a = (r_a + r_Pa) / 2 and the odd
// part o_a = (r_a - r_Pa) / 2 of a node pair are
//   e_a = sum_j Dxi_e[a][j] (Gxi_j + Geta_Pj) + sum_q lift_e ...
//   o_a = sum_j Dxi_o[a][j] (Gxi_j - Geta_Pj) + sum_q lift_o ...
// and in the lift side 0's point q goes with side 2's point nfq-1-q, side 1's
// point q with its own nfq-1-q (a middle point only enters the even part).
// That is Np (NS + NO) = Np^2 multiply-adds for the volume instead of 2 Np^2,
// and Np nfq 3/2 for the lift instead of 3 Np nfq. The lift carries the sign of
// the surface term and the 1/2 of roe_flux2.
template <int P, int NFQ>
struct FoldedOps {
  static constexpr int NP = np_of_p(P);
  static constexpr int NE = P + 1;
  static constexpr int NS = fold_nodes(P);                    // even parts
  static constexpr int NO = fold_pairs(P);                    // odd parts
  static constexpr int NOA = NO > 0 ? NO : 1;
  static constexpr int HQ = (NFQ + 1) / 2;
  double De[NS][NP], Do[NOA][NP];
  double Le[NS][NFQ], Lo[NOA][NFQ];                            // sides 0 and 2
  double L1e[NS][HQ], L1o[NOA][HQ];                            // side 1
  double tp[3][NFQ][NE];
  double tm[3][NFQ][NE];
};

// What one stage launch reads and writes. Geometry rows (double2, Kpad each):
//   0: (Jinv00, Jinv01)  1: (Jinv10, Jinv11)  2..4: normal of side 0..2
//   5: (len0/detJ, len1/detJ)  6: (len2/detJ, 0)
// nbr[e] = (neighbour across side 0, 1, 2, unused).
//
// Tiles: tiles[t] = (start0, len0, start1, len1), two runs of consecutive
// elements (local columns 0..31 and 32..63). tile_items[t * kMaxItems + i],
// i < tile_count[t], lists the (element, side) faces tile t evaluates:
//   bits 0-7 local element, 8-9 side, 10 mirror (the neighbour is in the tile
//   and receives -F), 11-18 the neighbour's local column when mirrored.
struct StageArgs {
  const double2* in;    // state the right-hand side is evaluated on
  const double2* base;  // U_n (RK4 stages 1, 2)
  double2* acc;         // RK4 accumulator X (written by stage 1, read by stage 3; vt_tile.cuh)
  double2* out;         // next stage state / new U / the right-hand side itself
  const double2* geo;
  const int4* nbr;
  const int4* tiles;
  const int* tile_items;
  const int* tile_count;
  const double* tile_dt;  // per-tile time step (batched problems), or null: c_* hold dt
  unsigned long long* err;  // [0] first-error key, [1] steps done, [2] blocks done
  long long Kpad;
  int K;
  int ntiles;
  int stage;     // 0..3 RK4 stages, 4 forward Euler, 5 right-hand side only
  double c_acc;  // accumulator coefficient (stage 1)
  double c_out;  // output coefficient
  // Test hook of the bounded waits (vt_test_bulk_wait): polls of the tile's
  // mbarrier before a wait gives up (0: the default bound), and bit 0 of
  // test_flags issues no state copies at all, so every wait gives up.
  unsigned wait_tries = 0;
  int test_flags = 0;
  // RK4 stages 0-2 that only produce the next stage state (a step rerun to
  // keep its stage states): stage 1 does not form the accumulator
  int no_acc = 0;
  // 2-D tensor maps of in / acc / base, [2 Np rows] x [2 Kpad doubles], box of
  // 2 Np rows x 64 doubles (one 32-element run); encoded on the host by the
  // launcher, read by the tensor copies through this grid-constant parameter
  CUtensorMap map_in, map_acc, map_base;
};

enum : int { kTestNoCopies = 1 };

constexpr int kTileRun = 32;            // elements per run
constexpr int kTileElems = 2 * kTileRun;  // elements per tile
constexpr int kMaxItems = 3 * kTileElems;

enum : int { kStageEuler = 4, kStageRhs = 5 };

// Warp mappings of the stage kernel (vt_tile.cuh): one thread per (element,
// component), or per (element, component pair, node half). kMapFolded is the
// form that kMapPair takes where the operators have the reference triangle's
// reflection symmetry (select_kernel, vt_launch.cu).
enum : int { kMapComponent = 0, kMapPair = 1, kMapFolded = 2 };

// First-error key: (stage epoch << 40) | (((e * nfq + q) * 3 + s) * 4 + code).
// The minimum over all failures is the failure the reference's serial loop
// meets first: earliest stage, then element, face point, side, check.
__device__ __forceinline__ void record_error(const StageArgs& a, int nfq, int e, int q, int s,
                                             int code) {
  const unsigned long long steps = *(volatile unsigned long long*)&a.err[1];
  const int slot = a.stage < 4 ? a.stage : 0;
  const unsigned long long epoch = steps * 4ull + static_cast<unsigned long long>(slot);
  const unsigned long long local =
      ((static_cast<unsigned long long>(e) * nfq + q) * 3ull + s) * 4ull + code;
  atomicMin(&a.err[0], (epoch << 40) | local);
}

// 1/x for the positive, normal x of the flux formulas (densities, Roe-average
// terms): the hardware reciprocal estimate r (rcp.approx.ftz.f64, relative
// error at most 1e-6 measured on B200) refined once by the first terms of the
// geometric series 1/x = r / (1 - e) = r (1 + e + e^2 + ...) with the residual
// e = 1 - x r formed by one fused multiply-add: the cubic member of the family
// of iterations for the reciprocal in A. S. Householder, "The Numerical
// Treatment of a Single Nonlinear Equation" (1970), sec. 4.4. The truncated
// terms are below e^3 = 1e-18, so the result is within rounding of 1/x, with
// three multiply-adds instead of the four of two Newton-Raphson steps
// (tests/test_gpu_reciprocal.py bounds the difference from 1.0 / x at one
// ulp). Zero, subnormal and non-finite x are not handled (those states are
// non-physical and reported by the flux's checks).
__device__ __forceinline__ double recip_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// 1/sqrt(x) for positive, normal x, the same way: the hardware estimate y
// (rsqrt.approx.ftz.f64) refined once by the binomial series
// x^-1/2 = y (1 - e)^-1/2 = y (1 + e/2 + 3 e^2/8 + ...) with e = 1 - x y^2
// (at most 1.9e-6 measured on B200, so the truncated terms are below 3e-18).
// At most two ulps from the exact value (tests/test_gpu_flux.py).
__device__ __forceinline__ double rsqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y, fma(0.375, e, 0.5) * e, y);
}

// The reference's checks of a face's two states in its order
// (Numericalflux.cpp:42-115): 1 left state, 2 right state, 3 c2 <= 0, else 0;
// the sign of a pressure is taken from rho times it, which needs no division.
// A NaN fails no check. Reached only when a sign test says that one may fail.
__device__ __forceinline__ int flux_error_code(const double* uL, const double* uR, double c2) {
  const double sL = fma(uL[0], uL[3], -0.5 * fma(uL[1], uL[1], uL[2] * uL[2]));
  const double sR = fma(uR[0], uR[3], -0.5 * fma(uR[1], uR[1], uR[2] * uR[2]));
  if (uL[0] <= 0 || sL <= 0) return 1;
  if (uR[0] <= 0 || sR <= 0) return 2;
  return c2 <= 0 ? 3 : 0;
}

// Twice the Roe flux with the reference's entropy fix and its squared "sound
// speed" ci = c2^2 (Numericalflux.cpp:13-157); the callers take the factor 1/2
// into the lift's coefficients, which is exact. The FP64 pipe is what bounds
// the face phase (two cycles per warp instruction and scheduler), so the
// formula is arranged for the fewest FP64 instructions, 94 where the previous
// arrangement took 134 (rk4 at 768 x 768, p = 3: see the stage kernel):
//   y = (rhoL rhoR)^-1/2 gives both densities' reciprocals (y^2) and the Roe
//     weights: with w = sqrt(rhoL rhoR), multiplying the averages through by
//     sqrt(rhoL) makes them (rhoL qL + w qR) / (rhoL + w), where rhoL qL is
//     the conserved variable itself, so neither side's velocities nor its
//     enthalpy are formed;
//   p = (gamma-1) (rhoE - |m|^2 / (2 rho));
//   t = u_n / ci decides the entropy fix of l3 (|t| < 1/10: l3 =
//     ci/20 + 5 u_n t, else |u_n|);
//   for |t| < 7/8 the acoustic eigenvalues keep their signs and lie above the
//     fix's threshold (|u_n| + ci/10 < ci), so (|l0| + |l1|)/2 = ci and
//     (|l0| - |l1|)/2 = u_n exactly; other states take the general form;
//   the pressure sum and C2 share the normal's coefficients.
// The checks look at the sign words of both densities, both pressures and c2
// with integer instructions; only when one is not positive does
// flux_error_code decide as the reference does.
// Equal to the reference's expression up to rounding. Returns the reference's
// error code (1 left state, 2 right state, 3 c2 <= 0) or 0.
__device__ __forceinline__ int roe_flux2(const double* uL, const double* uR, double nx, double ny, double* f) {
  const double rL = uL[0], rR = uR[0];
  const double rLR = rL * rR;
  const double y = rsqrt_nr(rLR);
  const double irLR = y * y, w = rLR * y;
  const double irL = rR * irLR, irR = rL * irLR;

  const double mnL = fma(uL[1], nx, uL[2] * ny);
  const double unL = mnL * irL;
  const double pL = kGm1 * fma(-0.5, fma(uL[1], uL[1], uL[2] * uL[2]) * irL, uL[3]);
  const double rHL = uL[3] + pL;
  const double mnR = fma(uR[1], nx, uR[2] * ny);
  const double unR = mnR * irR;
  const double pR = kGm1 * fma(-0.5, fma(uR[1], uR[1], uR[2] * uR[2]) * irR, uR[3]);
  const double rHR = uR[3] + pR;
  const double du0 = rR - rL, du1 = uR[1] - uL[1], du2 = uR[2] - uL[2], du3 = uR[3] - uL[3];

  const double g = w * irR;  // sqrt(rhoL / rhoR)
  const double d1 = recip_nr(rL + w);
  const double ui = fma(g, uR[1], uL[1]) * d1;
  const double vi = fma(g, uR[2], uL[2]) * d1;
  const double Hi = fma(g, rHR, rHL) * d1;
  const double q2 = fma(ui, ui, vi * vi);
  const double ucp = fma(ui, nx, vi * ny);
  const double c2 = kGm1 * fma(-0.5, q2, Hi);
  const double ci = c2 * c2;
  const double ci1 = recip_nr(ci);

  const int sign = min(min(min(__double2hiint(rL), __double2hiint(rR)), min(__double2hiint(pL), __double2hiint(pR))),
                       __double2hiint(c2));
  int code = 0;
  if (__builtin_expect(sign <= 0, 0)) code = flux_error_code(uL, uR, c2);

  const double t = ucp * ci1;
  const double l3 = fabs(t) < 0.1 ? fma(5.0 * ucp, t, 0.05 * ci) : fabs(ucp);
  double s1l3, s2;  // (|l0| + |l1|)/2 - l3 and (|l0| - |l1|)/2
  if (__builtin_expect((__double2hiint(t) & 0x7fffffff) < 0x3fec0000, 1)) {  // |t| < 7/8
    s1l3 = ci - l3;
    s2 = ucp;
  } else {
    const double l0r = ucp + ci, l1r = ucp - ci, eps = 0.1 * ci;
    const double l0 = fabs(l0r) < eps ? fma(l0r * l0r, 5.0 * ci1, 0.05 * ci) : fabs(l0r);
    const double l1 = fabs(l1r) < eps ? fma(l1r * l1r, 5.0 * ci1, 0.05 * ci) : fabs(l1r);
    s1l3 = fma(0.5, l0 + l1, -l3);
    s2 = 0.5 * (l0 - l1);
  }
  const double G1 = (kGm1 * ci1) * fma(0.5 * q2, du0, fma(-ui, du1, fma(-vi, du2, du3)));  // over ci
  const double G2 = fma(-ucp, du0, fma(du1, nx, du2 * ny));
  const double C1 = fma(G1, s1l3, G2 * s2) * ci1;
  const double C2 = fma(G1, s2, G2 * s1l3);
  const double pC = (pL + pR) - C2;
  f[0] = (mnL + mnR) - fma(l3, du0, C1);
  f[1] = fma(uL[1], unL, fma(uR[1], unR, fma(pC, nx, -fma(l3, du1, C1 * ui))));
  f[2] = fma(uL[2], unL, fma(uR[2], unR, fma(pC, ny, -fma(l3, du2, C1 * vi))));
  f[3] = fma(rHL, unL, fma(rHR, unR, -fma(l3, du3, fma(C1, Hi, C2 * ucp))));
  return code;
}

// Nodal Euler flux of one node's state (the formula of Timestepping.cpp:141-158)
// contracted with the inverse Jacobian rows: gxi = Jinv00 Fx + Jinv01 Fy,
// geta = Jinv10 Fx + Jinv11 Fy, formed through the contravariant velocities
// (25 FP64 instructions and a reciprocal estimate against 34 when Fx and Fy
// are formed first).
__device__ __forceinline__ void contravariant_flux(const double* s, double j00, double j01,
                                                   double j10, double j11, double* gxi,
                                                   double* geta) {
  const double ir = recip_nr(s[0]);
  const double p = kGm1 * fma(-0.5, fma(s[1], s[1], s[2] * s[2]) * ir, s[3]);
  const double rH = s[3] + p;
  gxi[0] = fma(j00, s[1], j01 * s[2]);
  geta[0] = fma(j10, s[1], j11 * s[2]);
  const double vxi = gxi[0] * ir, veta = geta[0] * ir;
  gxi[1] = fma(s[1], vxi, j00 * p);
  gxi[2] = fma(s[2], vxi, j01 * p);
  gxi[3] = rH * vxi;
  geta[1] = fma(s[1], veta, j10 * p);
  geta[2] = fma(s[2], veta, j11 * p);
  geta[3] = rH * veta;
}

}  // namespace vt
