// Kernels of the discrete adjoint on meshes without the fused form.
//
// One reverse RK4 stage (the transpose of one stage's right-hand side at the
// stage state U, applied to the stage adjoint a) is two launches:
//
//   adjoint_face_kernel     thread (element e, side s, face point q): a block
//                           is 32 consecutive elements of one side s, a warp
//                           one face point q:
//                           bF = -(len_s / detJ) sa * sum_i lift[s][i][q] a_i
//                           (transposed lift and mass inverse), then the
//                           transposed Roe Jacobian at (U+, U-) gives the face
//                           adjoints of the own trace (bp) and of the
//                           neighbour's trace (bm);
//   adjoint_element_kernel  thread (element e, node j): the transposed volume
//                           operator sum_i D[d][i][j] a_i, the transposed nodal
//                           flux Jacobian at U_j, and the transposed traces of
//                           the own faces (tp, bp of e) and of the neighbours'
//                           faces (tm, bm of the neighbour across side s, whose
//                           side s faces e), then the reverse RK4 combine.
//
// On meshes whose faces take the edge-once form the whole reverse stage is
// one launch instead, adjoint_tile_kernel (vt_adjoint_tile.cuh).
//
// Both read the state through the column layout of the stage kernel
// (vt_device.cuh), so a warp's 32 columns are contiguous 512-byte rows; e below
// is a column. The face adjoints bp/bm hold 2 double2 rows per (s, q) face
// point:
//   bp[((s * NFQ + q) * 2 + h) * ncols + e]
#pragma once

#include "vt_adjoint.cuh"
#include "vt_device.cuh"

namespace vt {

struct AdjArgs {
  const double2* U;       // stage state the right-hand side was evaluated on
  const double2* a;       // stage adjoint (multiplied by sa)
  const double2* lam;     // adjoint of U_{n+1}, or null when lam_coef = 0 and a_out is null
  const double2* acc_in;  // running adjoint of U_n, or null
  double2* acc_out;       // acc_in + lam_coef * lam + g
  double2* a_out;         // cl * lam + cg * g, or null
  double2* bp;            // face adjoints, own trace
  double2* bm;            // face adjoints, neighbour trace
  const double2* geo;
  const int4* nbr;
  const int* elem;  // element of each column (-1: empty)
  // Per-tile time steps (a batch group with uneven steps), or null: then sa
  // (when sa_dt is set), cl and cg are fractions of the tile's step.
  const double* tile_dt;
  int sa_dt;
  // The stage kernel's tile schedule (adjoint_tile_kernel) and error words.
  const unsigned char* lists;
  int ntiles;
  unsigned long long* err;
  long long ncols;
  double sa, lam_coef, cl, cg;
};

constexpr int kAdjRun = 32;  // elements per block (one per lane)

template <int P, int NFQ>
__global__ void __launch_bounds__(kAdjRun * NFQ)
    adjoint_face_kernel(const AdjArgs a, const StageOps<P, NFQ> o) {
  constexpr int NP = np_of_p(P), NE = P + 1;
  const int e = blockIdx.x * kAdjRun + threadIdx.x;
  if (__ldg(a.elem + e) < 0) return;
  const int s = blockIdx.y, q = threadIdx.y;  // uniform per block / warp
  const int w = s * NFQ + q;
  const long long KP = a.ncols;
  const int4 nb4 = __ldg(a.nbr + e);
  const int nb = s == 0 ? nb4.x : (s == 1 ? nb4.y : nb4.z);
  double up[4] = {0.0, 0.0, 0.0, 0.0}, um[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    const int node = edge_node(P, s, k);
    const double cp = o.tp[s][q][k], cm = o.tm[s][q][k];
    const double2 *pe = a.U + state_index(NP, e, 2 * node), *pn = a.U + state_index(NP, nb, 2 * node);
    const double2 x0 = __ldg(pe), x1 = __ldg(pe + kTileRun);
    const double2 y0 = __ldg(pn), y1 = __ldg(pn + kTileRun);
    up[0] = fma(cp, x0.x, up[0]);
    up[1] = fma(cp, x0.y, up[1]);
    up[2] = fma(cp, x1.x, up[2]);
    up[3] = fma(cp, x1.y, up[3]);
    um[0] = fma(cm, y0.x, um[0]);
    um[1] = fma(cm, y0.y, um[1]);
    um[2] = fma(cm, y1.x, um[2]);
    um[3] = fma(cm, y1.y, um[3]);
  }
  double bf[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const double l = o.lift[s][i][q];
    const double2* pa = a.a + state_index(NP, e, 2 * i);
    const double2 a0 = __ldg(pa), a1 = __ldg(pa + kTileRun);
    bf[0] = fma(l, a0.x, bf[0]);
    bf[1] = fma(l, a0.y, bf[1]);
    bf[2] = fma(l, a1.x, bf[2]);
    bf[3] = fma(l, a1.y, bf[3]);
  }
  const double2 lsa = __ldg(a.geo + geo_index(e, 2)), lsb = __ldg(a.geo + geo_index(e, 3));
  const double sa = (a.tile_dt && a.sa_dt) ? a.sa * __ldg(a.tile_dt + e / kTileElems) : a.sa;
  const double sc = -(s == 0 ? lsa.x : (s == 1 ? lsa.y : lsb.x)) * sa;
#pragma unroll
  for (int c = 0; c < 4; ++c) bf[c] *= sc;
  const double2 n = __ldg(a.geo + geo_index(e, 4 + s));
  double bu[4] = {0.0, 0.0, 0.0, 0.0}, bv[4] = {0.0, 0.0, 0.0, 0.0};
  roe_flux_vjp(up, um, n.x, n.y, bf, bu, bv);
  const long long r0 = static_cast<long long>(2 * w) * KP + e;
  a.bp[r0] = make_double2(bu[0], bu[1]);
  a.bp[r0 + KP] = make_double2(bu[2], bu[3]);
  a.bm[r0] = make_double2(bv[0], bv[1]);
  a.bm[r0 + KP] = make_double2(bv[2], bv[3]);
}

template <int P, int NFQ>
__global__ void __launch_bounds__(kAdjRun * np_of_p(P), 3)
    adjoint_element_kernel(const AdjArgs a, const StageOps<P, NFQ> o) {
  constexpr int NP = np_of_p(P), NE = P + 1;
  __shared__ double2 sA[2 * NP][kAdjRun];  // the block's stage adjoints, row pair j loaded by warp j
  const int e = blockIdx.x * kAdjRun + threadIdx.x;
  const int j = threadIdx.y;  // node, uniform per warp
  const long long KP = a.ncols;
  const bool valid = __ldg(a.elem + e) >= 0;
  // every global operand of this thread is requested before the barrier
  const long long r0 = state_index(NP, e, 2 * j), r1 = r0 + kTileRun;
  double2 u0 = make_double2(1.0, 0.0), u1 = make_double2(0.0, 0.0), j0 = u1, j1 = u1, l0 = u1, l1 = u1, c0 = u1,
          c1 = u1;
  int4 nb4 = make_int4(0, 0, 0, 0);
  if (valid) {
    sA[2 * j][threadIdx.x] = __ldg(a.a + r0);
    sA[2 * j + 1][threadIdx.x] = __ldg(a.a + r1);
    u0 = __ldg(a.U + r0);
    u1 = __ldg(a.U + r1);
    j0 = __ldg(a.geo + geo_index(e, 0));
    j1 = __ldg(a.geo + geo_index(e, 1));
    nb4 = __ldg(a.nbr + e);
    if (a.lam_coef != 0.0 || a.a_out) {
      l0 = a.lam[r0];
      l1 = a.lam[r1];
    }
    if (a.acc_in) {
      c0 = a.acc_in[r0];
      c1 = a.acc_in[r1];
    }
  }
  __syncthreads();
  if (!valid) return;
  double g[4] = {0.0, 0.0, 0.0, 0.0};
  if (P > 0) {
    double bx[4] = {0.0, 0.0, 0.0, 0.0}, by[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const double d0 = o.D[0][i][j], d1 = o.D[1][i][j];
      const double2 a0 = sA[2 * i][threadIdx.x], a1 = sA[2 * i + 1][threadIdx.x];
      bx[0] = fma(d0, a0.x, bx[0]);
      bx[1] = fma(d0, a0.y, bx[1]);
      bx[2] = fma(d0, a1.x, bx[2]);
      bx[3] = fma(d0, a1.y, bx[3]);
      by[0] = fma(d1, a0.x, by[0]);
      by[1] = fma(d1, a0.y, by[1]);
      by[2] = fma(d1, a1.x, by[2]);
      by[3] = fma(d1, a1.y, by[3]);
    }
    const double sa = (a.tile_dt && a.sa_dt) ? a.sa * __ldg(a.tile_dt + e / kTileElems) : a.sa;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      bx[c] *= sa;
      by[c] *= sa;
    }
    const double sv[4] = {u0.x, u0.y, u1.x, u1.y};
    contravariant_vjp(sv, j0.x, j0.y, j1.x, j1.y, bx, by, g);
  }
  // two-sided faces: own bp (tp) and the neighbour's bm (tm)
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int nb = s == 0 ? nb4.x : (s == 1 ? nb4.y : nb4.z);
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      if (edge_node(P, s, k) != j) continue;  // uniform per warp
#pragma unroll
      for (int q = 0; q < NFQ; ++q) {
        const long long r0 = static_cast<long long>(2 * (s * NFQ + q)) * KP;
        const double cp = o.tp[s][q][k], cm = o.tm[s][q][k];
        const double2 p0 = __ldg(a.bp + r0 + e), p1 = __ldg(a.bp + r0 + KP + e);
        g[0] = fma(cp, p0.x, g[0]);
        g[1] = fma(cp, p0.y, g[1]);
        g[2] = fma(cp, p1.x, g[2]);
        g[3] = fma(cp, p1.y, g[3]);
        const double2 m0 = __ldg(a.bm + r0 + nb), m1 = __ldg(a.bm + r0 + KP + nb);
        g[0] = fma(cm, m0.x, g[0]);
        g[1] = fma(cm, m0.y, g[1]);
        g[2] = fma(cm, m1.x, g[2]);
        g[3] = fma(cm, m1.y, g[3]);
      }
    }
  }
  const double lam[4] = {l0.x, l0.y, l1.x, l1.y};
  double acc[4] = {c0.x, c0.y, c1.x, c1.y};
#pragma unroll
  for (int c = 0; c < 4; ++c) acc[c] = fma(a.lam_coef, lam[c], acc[c]) + g[c];
  if (a.a_out) {
    const double h = a.tile_dt ? __ldg(a.tile_dt + e / kTileElems) : 1.0;
    const double cl = a.tile_dt ? a.cl * h : a.cl, cg = a.tile_dt ? a.cg * h : a.cg;
    double an[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) an[c] = fma(cl, lam[c], cg * g[c]);
    a.a_out[r0] = make_double2(an[0], an[1]);
    a.a_out[r1] = make_double2(an[2], an[3]);
  }
  a.acc_out[r0] = make_double2(acc[0], acc[1]);
  a.acc_out[r1] = make_double2(acc[2], acc[3]);
}

}  // namespace vt
