// Device-side building blocks of the stepper: state layout, folded operators,
// Roe flux, nodal flux and the first-error record.
//
// Layout in HBM. The elements are renumbered into columns: a tile is 64
// columns (some may be empty), and half a tile, 32 columns, is a block. A state
// vector (U, a stage, the RK accumulator) holds each block's 2 Np rows of 32
// double2, row 2*i + h for node i and component pair h (h = 0: rho, rho u;
// h = 1: rho v, rho E): a block is contiguous (10 KB at p = 3), so a tile
// arrives by two bulk copies, a thread's rows lie at constant distances (the
// loads and stores of a phase share one address computation), and a warp
// touching the 32 columns of one row reads 512 contiguous bytes. The geometry
// has the same form with 7 rows. Columns follow the mesh: the triangles of
// type 0 of a tile are its first block, those of type 1 its second, so that
// the faces of one kind join consecutive columns (Numbering).
#pragma once

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
// (fold_operators). With Pj the mirror image of node j and
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

// Even and odd parts of the operators under the reflection (FoldedOps). Each
// coefficient takes both of the entries that the symmetry makes equal, so the
// rounding of the two is averaged.
template <int P, int NFQ>
inline void fold_operators(const StageOps<P, NFQ>& o, FoldedOps<P, NFQ>* f) {
  constexpr int NP = np_of_p(P), NS = fold_nodes(P), NO = fold_pairs(P);
  *f = FoldedOps<P, NFQ>{};
  for (int a = 0; a < NS; ++a) {
    const int i = fold_node(P, a), m = mirror_node(P, i);
    for (int j = 0; j < NP; ++j) {
      const int mj = mirror_node(P, j);
      const double x = 0.5 * (o.D[0][i][j] + o.D[1][m][mj]), y = 0.5 * (o.D[0][m][j] + o.D[1][i][mj]);
      f->De[a][j] = 0.5 * (x + y);
      if (a < NO) f->Do[a][j] = 0.5 * (x - y);
    }
    for (int q = 0; q < NFQ; ++q) {
      const int r = NFQ - 1 - q;
      const double x = 0.5 * (o.lift[0][i][q] + o.lift[2][m][r]), y = 0.5 * (o.lift[0][m][q] + o.lift[2][i][r]);
      f->Le[a][q] = -0.25 * (x + y);
      if (a < NO) f->Lo[a][q] = -0.25 * (x - y);
      if (q <= r) {
        const double v = 0.5 * (o.lift[1][i][q] + o.lift[1][m][r]), z = 0.5 * (o.lift[1][m][q] + o.lift[1][i][r]);
        f->L1e[a][q] = -0.25 * (v + z);
        if (a < NO) f->L1o[a][q] = -0.25 * (v - z);
      }
    }
  }
  for (int s = 0; s < 3; ++s)
    for (int q = 0; q < NFQ; ++q)
      for (int k = 0; k < FoldedOps<P, NFQ>::NE; ++k) {
        f->tp[s][q][k] = o.tp[s][q][k];
        f->tm[s][q][k] = o.tm[s][q][k];
      }
}

constexpr int kTileRun = 32;              // columns per block (half a tile)
constexpr int kTileElems = 2 * kTileRun;  // columns per tile
constexpr int kGeoRows = 7;

// Index (in double2) of row `row` of column x of a state vector / the geometry.
__host__ __device__ __forceinline__ long long state_index(int np, long long x, int row) {
  return ((x >> 5) * 2 * np + row) * kTileRun + (x & 31);
}
__host__ __device__ __forceinline__ long long geo_index(long long x, int row) {
  return ((x >> 5) * kGeoRows + row) * kTileRun + (x & 31);
}

// Which column holds which element. On the reference's structured mesh of nx x
// ny cells (Meshgeneration.cpp:57-117: cell (j, row) holds elements
// 2(row*nx + j) and +1, of types 0 and 1) a tile is a block of W x H cells, W H
// <= 32, narrower at the mesh's right and upper edge; cell k of the tile has
// its type-0 triangle in column k and its type-1 triangle in column 32 + k. On
// any other mesh (nx = 0) a tile is 64 consecutive elements, the even ones in
// its first block and the odd ones in its second. The elements' own order
// (error reports, the callers' arrays) is never the columns' order.
struct Numbering {
  int K = 0, nx = 0, ny = 0, W = 0, H = 0, ntx = 0, ntiles = 0;
  __host__ __device__ int column(int e) const {
    if (nx == 0) return (e & ~63) | ((e & 1) << 5) | ((e & 63) >> 1);
    const int cell = e >> 1, r = cell / nx, j = cell - r * nx;
    const int ti = j / W, tj = r / H, w = W < nx - ti * W ? W : nx - ti * W;
    return (tj * ntx + ti) * kTileElems + (e & 1) * kTileRun + (r - tj * H) * w + (j - ti * W);
  }
  // -1 for an empty column
  __host__ __device__ int element(int x) const {
    const int tile = x / kTileElems, half = (x >> 5) & 1, k = x & 31;
    if (nx == 0) {
      const int e = tile * kTileElems + 2 * k + half;
      return e < K ? e : -1;
    }
    const int tj = tile / ntx, ti = tile - tj * ntx;
    const int w = W < nx - ti * W ? W : nx - ti * W, r = k / w, j = k - r * w;
    return r < H && tj * H + r < ny ? 2 * ((tj * H + r) * nx + ti * W + j) + half : -1;
  }
};

// What one stage launch reads and writes. Geometry rows (double2 per column):
//   0: (Jinv00, Jinv01)  1: (Jinv10, Jinv11)  2: (len0/detJ, len1/detJ)
//   3: (len2/detJ, detJ)  4..6: normal of side 0..2
// nbr[x] = (column across side 0, 1, 2, unused).
//
// lists holds kTileListBytes per tile, built once per mesh (vt_schedule.cuh):
//   uint16 [kMaxItems]  the (column, side) faces the tile evaluates, by class:
//     both columns in the tile, the neighbour staged in a slot, the neighbour
//     read from global memory (no slot left: FarFace, vt_tile.cuh). Bits 0-5 the
//     column in the tile, 6-7 the side, 8 both in the tile, 9-15 the neighbour's
//     column in the tile or its slot;
//   uint32 [4]  the work items (FaceCounts);
//   uint32 [2][kSlots]  per block, the neighbours to stage: 4 * column + side,
//     kNoNeighbour where a slot is empty (the used slots come first).
struct StageArgs {
  const double2* in;    // state the right-hand side is evaluated on
  const double2* base;  // U_n (RK4 stages 1, 2)
  double2* acc;         // RK4 accumulator X (written by stage 1, read by stage 3; vt_tile.cuh)
  double2* out;         // next stage state / new U / the right-hand side itself
  const double2* geo;
  const int4* nbr;
  const int* elem;      // element of each column (-1: empty), or null: Numbering with nx = 0
  const unsigned char* lists;
  const double* tile_dt;  // per-tile time step (batched problems), or null: c_* hold dt
  unsigned long long* err;  // kErrWords words, below
  int K;
  int ntiles;
  int stage;     // 0..3 RK4 stages, 4 forward Euler, 5 right-hand side only
  double c_acc;  // accumulator coefficient (stage 1)
  double c_out;  // output coefficient
  // Test hook of the bounded waits (vt_test_bulk_wait): polls of the tile's
  // mbarrier before a wait gives up (0: the default bound), and bit 0 of
  // test_flags issues no copies at all, so every wait gives up.
  unsigned wait_tries = 0;
  int test_flags = 0;
  // RK4 stages 0-2 that only produce the next stage state (a step rerun to
  // keep its stage states): stage 1 does not form the accumulator
  int no_acc = 0;
};

enum : int { kTestNoCopies = 1 };

// The words behind `err`, cleared before every call (word 0 to all ones):
// [0] first-error key, [1] steps done, [2] blocks of the running stage kernel
// that are done, [3] flags (1 bad neighbour, 2 a wait gave up), [4] tiles its
// blocks have taken beyond their first, [5], [6] likewise of the reverse stage,
// [7] the flags of vt_rhs_jvp, which leaves the other words as they are.
constexpr int kErrWords = 8;

constexpr int kMaxItems = 3 * kTileElems;
// A block of a W x H tile has W + H faces that leave the tile (12 of 8 x 4
// cells). 24 slots are what the stage kernel's three blocks per SM and the
// reverse stage's two have room for at p = 3; of 64 consecutive elements in a
// row of the reference's mesh, each half has 33.
constexpr int kSlots = 24;
constexpr int kOuterWords = (2 * kSlots + 3) / 4 * 4;
constexpr int kListCount = 2 * kMaxItems;      // byte offset of the counts
constexpr int kListOuter = kListCount + 16;    // byte offset of the slots
constexpr int kTileListBytes = kListOuter + kOuterWords * 4;
static_assert(kListCount % 16 == 0 && kTileListBytes % 16 == 0, "16-byte copies");
constexpr unsigned kNoNeighbour = 0xffffffffu;

__host__ __device__ constexpr unsigned face_item(int col, int side, bool inside, int x) {
  return static_cast<unsigned>(col | (side << 6) | (inside ? 1 << 8 : 0) | (x << 9));
}

// The work items of a face list: first the n0 faces inside the tile times the
// parts of their nfq points (p0 points each), then the n1 with a slot (p1 points
// each), part-major: item w < first is part w / n0 of face w % n0. The factor
// 2^20 / n + 1 makes w / n one multiplication, exact while w n < 2^20 (w < 10 n,
// n <= 192). The n2 faces without a slot are the end of the list (FarFace,
// vt_tile.cuh).
struct FaceCounts {
  unsigned n;        // n0 | n1 << 8 | n2 << 16
  unsigned points;   // p0 | p1 << 8 | first << 16 (the items of the faces inside the tile)
  unsigned factor0, factor1;
};
__host__ __device__ constexpr unsigned face_factor(int n) { return n > 0 ? (1u << 20) / n + 1 : 0; }

__host__ __device__ constexpr FaceCounts face_counts(int n0, int n1, int n2, int nfq, int p0, int p1) {
  return {static_cast<unsigned>(n0 | n1 << 8 | n2 << 16), static_cast<unsigned>(p0 | p1 << 8 | (n0 * ((nfq + p0 - 1) / p0)) << 16),
          face_factor(n0), face_factor(n1)};
}
// What the face phase costs a thread with i and j points per item, in tenths of
// a point inside the tile (the other ones take the neighbour's trace as well).
__device__ __forceinline__ int face_cost(int n0, int n1, int nfq, int i, int j, int threads) {
  const int items = n0 * ((nfq + i - 1) / i) + n1 * ((nfq + j - 1) / j);
  return (items + threads - 1) / threads * max(n0 ? 10 * i : 0, n1 ? 14 * j : 0);
}

// Work item w: its entry in the list and its points [q0, q1); false past the last one.
template <int NFQ>
__device__ __forceinline__ bool face_work(const FaceCounts& f, int w, int* entry, int* q0, int* q1) {
  const int first = f.points >> 16, n0 = f.n & 0xff;
  const bool in = w < first;
  const int v = in ? w : w - first, n = in ? n0 : (f.n >> 8) & 0xff, pts = in ? f.points & 0xff : (f.points >> 8) & 0xff;
  if (n == 0) return false;
  const int part = static_cast<int>((v * (in ? f.factor0 : f.factor1)) >> 20);
  *q0 = part * pts;
  *q1 = min(*q0 + pts, NFQ);
  *entry = (in ? 0 : n0) + v - part * n;
  return *q0 < NFQ;
}

enum : int { kStageEuler = 4, kStageRhs = 5 };

// Mappings of the stage kernel (vt_tile.cuh), one thread per (element,
// component) in each: kMapComponent applies the operators as they are;
// kMapDefault takes the form kMapFolded where the operators have the reference
// triangle's reflection symmetry, else kMapComponent's (select_kernel,
// vt_launch.cu).
enum : int { kMapComponent = 0, kMapDefault = 1, kMapFolded = 2 };

// First-error key: (stage epoch << 40) | (((e * nfq + q) * 3 + s) * 4 + code).
// The minimum over all failures is the failure the reference's serial loop
// meets first: earliest stage, then element, face point, side, check.
__device__ __forceinline__ void record_error_at(unsigned long long* err, unsigned long long epoch, int nfq, int e, int q,
                                                int s, int code) {
  const unsigned long long local =
      ((static_cast<unsigned long long>(e) * nfq + q) * 3ull + s) * 4ull + code;
  atomicMin(&err[0], (epoch << 40) | local);
}
__device__ __forceinline__ void record_error(const StageArgs& a, int nfq, int e, int q, int s,
                                             int code) {
  const unsigned long long steps = *(volatile unsigned long long*)&a.err[1];
  const int slot = a.stage < 4 ? a.stage : 0;
  record_error_at(a.err, steps * 4ull + static_cast<unsigned long long>(slot), nfq, e, q, s, code);
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
// flux_error_code decide as the reference does; one branch serves this and the
// eigenvalue test. Equal to the reference's expression up to rounding.
// on_error is called with the reference's error code (1 left state, 2 right
// state, 3 c2 <= 0).
// In three parts, so that several points can be evaluated side by side
// (face_points, vt_resident.cuh): the first two need no branch.
struct RoeAverages {
  double mn, unL, unR, pLR, rHL, rHR, du0, du1, du2, du3;  // mn: both sides' normal momentum
  double ui, vi, Hi, q2, ucp, c2, ci, ci1, l3, s1l3, s2;
  int usual;  // positive where |t| < 7/8 and the checked values are positive
};
__device__ __forceinline__ void roe_averages(const double* uL, const double* uR, double nx, double ny, RoeAverages& r) {
  const double rL = uL[0], rR = uR[0];
  const double rLR = rL * rR;
  const double y = rsqrt_nr(rLR);
  const double irLR = y * y, w = rLR * y;
  const double irL = rR * irLR, irR = rL * irLR;

  const double mnL = fma(uL[1], nx, uL[2] * ny);
  r.unL = mnL * irL;
  const double pL = kGm1 * fma(-0.5, fma(uL[1], uL[1], uL[2] * uL[2]) * irL, uL[3]);
  r.rHL = uL[3] + pL;
  const double mnR = fma(uR[1], nx, uR[2] * ny);
  r.unR = mnR * irR;
  const double pR = kGm1 * fma(-0.5, fma(uR[1], uR[1], uR[2] * uR[2]) * irR, uR[3]);
  r.rHR = uR[3] + pR;
  r.mn = mnL + mnR;
  r.pLR = pL + pR;
  r.du0 = rR - rL, r.du1 = uR[1] - uL[1], r.du2 = uR[2] - uL[2], r.du3 = uR[3] - uL[3];

  const double g = w * irR;  // sqrt(rhoL / rhoR)
  const double d1 = recip_nr(rL + w);
  r.ui = fma(g, uR[1], uL[1]) * d1;
  r.vi = fma(g, uR[2], uL[2]) * d1;
  r.Hi = fma(g, r.rHR, r.rHL) * d1;
  r.q2 = fma(r.ui, r.ui, r.vi * r.vi);
  r.ucp = fma(r.ui, nx, r.vi * ny);
  r.c2 = kGm1 * fma(-0.5, r.q2, r.Hi);
  r.ci = r.c2 * r.c2;
  r.ci1 = recip_nr(r.ci);

  const double t = r.ucp * r.ci1;
  r.l3 = fabs(t) < 0.1 ? fma(5.0 * r.ucp, t, 0.05 * r.ci) : fabs(r.ucp);
  r.s1l3 = r.ci - r.l3;  // (|l0| + |l1|)/2 - l3
  r.s2 = r.ucp;          // (|l0| - |l1|)/2
  r.usual = min(min(min(__double2hiint(rL), __double2hiint(rR)), min(__double2hiint(pL), __double2hiint(pR))),
                min(__double2hiint(r.c2), 0x3fec0000 - (__double2hiint(t) & 0x7fffffff)));
}
template <typename OnError>
__device__ __forceinline__ void roe_unusual(const double* uL, const double* uR, RoeAverages& r, OnError&& on_error) {
  const int code = flux_error_code(uL, uR, r.c2);
  if (code) on_error(code);
  const double l0r = r.ucp + r.ci, l1r = r.ucp - r.ci, eps = 0.1 * r.ci;
  const double l0 = fabs(l0r) < eps ? fma(l0r * l0r, 5.0 * r.ci1, 0.05 * r.ci) : fabs(l0r);
  const double l1 = fabs(l1r) < eps ? fma(l1r * l1r, 5.0 * r.ci1, 0.05 * r.ci) : fabs(l1r);
  r.s1l3 = fma(0.5, l0 + l1, -r.l3);
  r.s2 = 0.5 * (l0 - l1);
}
__device__ __forceinline__ void roe_sum(const double* uL, const double* uR, double nx, double ny, const RoeAverages& r,
                                        double* f) {
  const double G1 = (kGm1 * r.ci1) * fma(0.5 * r.q2, r.du0, fma(-r.ui, r.du1, fma(-r.vi, r.du2, r.du3)));  // over ci
  const double G2 = fma(-r.ucp, r.du0, fma(r.du1, nx, r.du2 * ny));
  const double C1 = fma(G1, r.s1l3, G2 * r.s2) * r.ci1;
  const double C2 = fma(G1, r.s2, G2 * r.s1l3);
  const double pC = r.pLR - C2;
  f[0] = r.mn - fma(r.l3, r.du0, C1);
  f[1] = fma(uL[1], r.unL, fma(uR[1], r.unR, fma(pC, nx, -fma(r.l3, r.du1, C1 * r.ui))));
  f[2] = fma(uL[2], r.unL, fma(uR[2], r.unR, fma(pC, ny, -fma(r.l3, r.du2, C1 * r.vi))));
  f[3] = fma(r.rHL, r.unL, fma(r.rHR, r.unR, -fma(r.l3, r.du3, fma(C1, r.Hi, C2 * r.ucp))));
}
template <typename OnError>
__device__ __forceinline__ void roe_flux2(const double* uL, const double* uR, double nx, double ny, double* f,
                                          OnError&& on_error) {
  RoeAverages r;
  roe_averages(uL, uR, nx, ny, r);
  if (__builtin_expect(r.usual <= 0, 0)) roe_unusual(uL, uR, r, on_error);
  roe_sum(uL, uR, nx, ny, r, f);
}

// Nodal Euler flux of one node's state (the formula of Timestepping.cpp:141-158)
// contracted with the inverse Jacobian rows: gxi = Jinv00 Fx + Jinv01 Fy,
// geta = Jinv10 Fx + Jinv11 Fy, formed through the contravariant velocities
// (25 FP64 instructions and a reciprocal estimate against 34 when Fx and Fy
// are formed first). With FACTORED the energy flux stays a product: gxi[3] and
// geta[3] are the contravariant velocities and gxi[4] = geta[4] = rH.
template <bool FACTORED = false>
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
  geta[1] = fma(s[1], veta, j10 * p);
  geta[2] = fma(s[2], veta, j11 * p);
  if constexpr (FACTORED) {
    gxi[3] = vxi, geta[3] = veta;
    gxi[4] = geta[4] = rH;
  } else {
    gxi[3] = rH * vxi;
    geta[3] = rH * veta;
  }
}

}  // namespace vt
