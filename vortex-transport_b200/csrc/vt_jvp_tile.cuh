// The derivative of one stage's right-hand side along a direction, dk = R'(U) V,
// with the tangent-linear RK4 combine, on the stage kernel's tiles: the same
// phases as the stage (vt_tile.cuh), each quantity beside its derivative.
//
// State and direction each have a tile, the neighbours' side nodes and a face
// buffer: 130 KB at p = 3, nfq = 6, so one block per SM, with the registers of
// one. The derivative of a face's flux overwrites the direction's traces; the
// nodal flux's derivative goes over the state's.
//
// At 64 x 64 cells, p = 3 a tangent-linear step (four stages, four of these)
// took 187 us with one thread per element on dual numbers (31 us a launch,
// spilling) and two separate linear combinations per stage, and takes 72 us.
#pragma once

#include "vt_adjoint.cuh"
#include "vt_tile.cuh"

namespace vt {

struct JvpArgs {
  const double2 *U, *V;
  const double2 *x1, *x2;  // out1 = x1 + c1 dk, out2 = x2 + c2 dk; x1 null: out1 = dk; out2 may be null
  double2 *out1, *out2;
  double c1, c2;
  unsigned long long* flags;  // the error word whose bit 1 says that a wait gave up
};

template <int P, int NFQ>
struct JvpLayout {
  using B = TileLayout<P, NFQ>;
  static constexpr int kV = (B::kBytes + 127) / 128 * 128;                 // double2 [2][2NP][32] the direction
  static constexpr int kHV = kV + 2 * B::NP * kTileElems * 16;              // its neighbours' side nodes
  static constexpr int kFV = kHV + 2 * B::NE * 2 * kSlots * 16;             // its traces, then the flux's derivative
  static constexpr int kBytes = kFV + 6 * NFQ * kTileElems * 16;
};

template <int P, int NFQ, int MAP, bool FAR>
__global__ void __launch_bounds__(4 * kTileElems, 1)
    jvp_tile_kernel(const __grid_constant__ StageArgs a, const __grid_constant__ JvpArgs ja,
                    const OpsOf<P, NFQ, MAP> ops) {
  using B = TileLayout<P, NFQ>;
  using L = JvpLayout<P, NFQ>;
  constexpr int E = B::E;
  constexpr int NP = B::NP;
  constexpr int NE = B::NE;
  constexpr int T = 4 * E;
  constexpr bool FOLD = MAP == kMapFolded;
  constexpr unsigned kState = 2 * NP * kTileRun * 16;
  extern __shared__ __align__(128) unsigned char smem[];
  double2* S = reinterpret_cast<double2*>(smem + B::kS);
  double2* V = reinterpret_cast<double2*>(smem + L::kV);
  double2* H = reinterpret_cast<double2*>(smem + B::kH);
  double2* HV = reinterpret_cast<double2*>(smem + L::kHV);
  double* FU = reinterpret_cast<double*>(smem + B::kFB);
  double2* FU2 = reinterpret_cast<double2*>(smem + B::kFB);
  double* FV = reinterpret_cast<double*>(smem + L::kFV);
  double2* FV2 = reinterpret_cast<double2*>(smem + L::kFV);
  double2* GE = reinterpret_cast<double2*>(smem + B::kGE);
  double* TM = reinterpret_cast<double*>(smem + B::kTM);
  const int* EL = reinterpret_cast<const int*>(smem + B::kEL);
  const unsigned short* items = reinterpret_cast<const unsigned short*>(smem + B::kItems);
  const FaceCounts* counts = reinterpret_cast<const FaceCounts*>(smem + B::kItems + kListCount);
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + B::kBar);
  int* abort_flag = reinterpret_cast<int*>(smem + B::kBar + 8);

  const int t = threadIdx.x;
  const int lane = t & 31;
  const int which = (t >> 5) & 1;
  const int grp = t >> 6;
  const int col = t % E;
  const int el = work_column(t), c = work_component(t);

  {
    const double* tm = &ops.tm[0][0][0];
    for (int l = t; l < 3 * NFQ * NE; l += T) TM[l] = tm[l];
  }
  if (t == 0) {
    mbar_init(bar, 4);  // per half: the mesh and state copies, and the direction's
    *abort_flag = 0;
  }
  __syncthreads();
  unsigned parity = 0;
  bool waited = false;

  for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
    const long long blk = 2ll * tile + which;
    // ---- 1. load ------------------------------------------------------------------
    const unsigned code = neighbour_code(a.lists, tile, which, lane);
    if (grp == 0 && lane == 0) issue_mesh_copies<P, NFQ>(a, tile, which, smem);
    if (!waited) {
      wait_for_previous();
      let_next_start();
      waited = true;
    }
    if (grp == 0 && lane == 0) {
      issue_state_copy<P, NFQ>(ja.U, tile, which, smem, 0);
      mbar_arrive_expect_tx(bar, kState);
      bulk_g2s(smem + L::kV + which * kState, ja.V + blk * (2 * NP * kTileRun), kState, bar);
    }
    copy_neighbours<P>(H, ja.U, code, which, grp, lane);
    copy_neighbours<P>(HV, ja.V, code, which, grp, lane);
    cp_async_commit();
    {
      bool ok = false;
      for (unsigned n = 0; n < kMaxWaitTries && !ok; ++n) ok = mbar_try_wait(bar, parity);
      if (!ok) {
        atomicOr(ja.flags, 2ull);
        *abort_flag = 1;
      }
    }
    parity ^= 1u;

    // ---- 2. own traces ---------------------------------------------------------------
    own_traces<P, NFQ>(ops, S, FU, el, c);
    own_traces<P, NFQ>(ops, V, FV, el, c);
    cp_async_wait_all();
    __syncthreads();
    if (*abort_flag) break;

    // ---- 3. faces: the (doubled) flux's derivative overwrites the direction's traces ----
    const FaceCounts faces = *counts;
    int entry, q, q1;
    for (int w = t; face_work<NFQ>(faces, w, &entry, &q, &q1); w += T) {
      const int it = items[entry];
      const int fl = it & 63, s = (it >> 6) & 3, x = it >> 9;
      const bool mirror = (it >> 8) & 1;
      const double2 n = GE[((fl >> 5) * kGeoRows + 4 + s) * kTileRun + (fl & 31)];
      int own = (s * NFQ + q) * 2 * E + fl, oth = (s * NFQ + NFQ - 1 - q) * 2 * E + (mirror ? x : 0);
#pragma unroll 1
      for (; q < q1; ++q, own += 2 * E, oth -= 2 * E) {
        const double2 u0 = FU2[own], u1 = FU2[own + E], v0 = FV2[own], v1 = FV2[own + E];
        const double up[4] = {u0.x, u0.y, u1.x, u1.y}, dp[4] = {v0.x, v0.y, v1.x, v1.y};
        double um[4] = {0.0, 0.0, 0.0, 0.0}, dm[4] = {0.0, 0.0, 0.0, 0.0};
        if (mirror) {
          const double2 y0 = FU2[oth], y1 = FU2[oth + E], z0 = FV2[oth], z1 = FV2[oth + E];
          um[0] = y0.x, um[1] = y0.y, um[2] = y1.x, um[3] = y1.y;
          dm[0] = z0.x, dm[1] = z0.y, dm[2] = z1.x, dm[3] = z1.y;
        } else {
          const double* cm = TM + (s * NFQ + q) * NE;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const double2 n0 = H[2 * k * 2 * kSlots + x], n1 = H[(2 * k + 1) * 2 * kSlots + x];
            const double2 m0 = HV[2 * k * 2 * kSlots + x], m1 = HV[(2 * k + 1) * 2 * kSlots + x];
            um[0] = fma(cm[k], n0.x, um[0]), um[1] = fma(cm[k], n0.y, um[1]);
            um[2] = fma(cm[k], n1.x, um[2]), um[3] = fma(cm[k], n1.y, um[3]);
            dm[0] = fma(cm[k], m0.x, dm[0]), dm[1] = fma(cm[k], m0.y, dm[1]);
            dm[2] = fma(cm[k], m1.x, dm[2]), dm[3] = fma(cm[k], m1.y, dm[3]);
          }
        }
        double f[4];
        roe_flux2_jvp(up, um, n.x, n.y, dp, dm, f);
        FV2[own] = make_double2(f[0], f[1]);
        FV2[own + E] = make_double2(f[2], f[3]);
        if (mirror) {
          FV2[oth] = make_double2(-f[0], -f[1]);
          FV2[oth + E] = make_double2(-f[2], -f[3]);
        }
      }
    }
    if constexpr (FAR) {
      FarFace x;
      for (int w = t; far_face<NFQ>(faces, items, a.nbr, tile, w, &x); w += T) {
        const double2 n = GE[((x.col >> 5) * kGeoRows + 4 + x.s) * kTileRun + (x.col & 31)];
        const int own = (x.s * NFQ + x.q) * 2 * E + x.col;
        const double2 u0 = FU2[own], u1 = FU2[own + E], v0 = FV2[own], v1 = FV2[own + E];
        const double up[4] = {u0.x, u0.y, u1.x, u1.y}, dp[4] = {v0.x, v0.y, v1.x, v1.y};
        double um[4], dm[4], f[4];
        const double* cm = TM + (x.s * NFQ + x.q) * NE;
        far_trace<P>(ja.U, x, cm, um, [](const double2* p) { return *p; });
        far_trace<P>(ja.V, x, cm, dm, [](const double2* p) { return *p; });
        roe_flux2_jvp(up, um, n.x, n.y, dp, dm, f);
        FV2[own] = make_double2(f[0], f[1]);
        FV2[own + E] = make_double2(f[2], f[3]);
      }
    }
    __syncthreads();

    // ---- 4. lift ---------------------------------------------------------------------
    const bool valid = EL[el] >= 0;
    const int at = ((c >> 1) * E + el) * 2 + (c & 1);
    double r[NP];
    {
      const double2* ge = GE + which * kGeoRows * kTileRun + (el & 31);
      lift_term<P, NFQ>(ops, FV + at, ge[2 * kTileRun], ge[3 * kTileRun], r);
    }

    // ---- 5. derivative of the nodal flux, over the state's traces -----------------------
    if (P > 0) {
      const double2* ge = GE + which * kGeoRows * kTileRun + lane;
      const double2 j0 = ge[0], j1 = ge[kTileRun];
      auto flux = [&](int j, double* gxi, double* geta) {
        const double2 s0 = S[sidx<NP>(2 * j, col)], s1 = S[sidx<NP>(2 * j + 1, col)];
        const double2 d0 = V[sidx<NP>(2 * j, col)], d1 = V[sidx<NP>(2 * j + 1, col)];
        const double sv[4] = {s0.x, s0.y, s1.x, s1.y}, dv[4] = {d0.x, d0.y, d1.x, d1.y};
        contravariant_jvp(sv, dv, j0.x, j0.y, j1.x, j1.y, gxi, geta);
      };
      if constexpr (FOLD) {
        folded_flux_rows<P>(FU2, col, grp, flux);
      } else {
        for (int j = grp; j < NP; j += 4) {
          double gxi[4], geta[4];
          flux(j, gxi, geta);
          double2* g = FU2 + j * 4 * E + col;
          g[0] = make_double2(gxi[0], gxi[1]);
          g[E] = make_double2(gxi[2], gxi[3]);
          g[2 * E] = make_double2(geta[0], geta[1]);
          g[3 * E] = make_double2(geta[2], geta[3]);
        }
      }
    }
    run_sync(t);

    // ---- 6. volume, combine -------------------------------------------------------------
    if (P > 0) volume_term<P, NFQ>(ops, FU + at, r);
    if constexpr (FOLD) unfold<P>(r);
    if (valid) {
      constexpr int kStep = 4 * kTileRun;
      const long long off0 = blk * (4 * NP * kTileRun) + (c >> 1) * (2 * kTileRun) + (el & 31) * 2 + (c & 1);
      const double* x1 = reinterpret_cast<const double*>(ja.x1) + off0;
      const double* x2 = reinterpret_cast<const double*>(ja.x2) + off0;
      double* out1 = reinterpret_cast<double*>(ja.out1) + off0;
      double* out2 = reinterpret_cast<double*>(ja.out2) + off0;
      double y1[NP], y2[NP];  // every load before the first store: out1 may be x1
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        y1[i] = ja.x1 ? x1[i * kStep] : 0.0;
        y2[i] = ja.out2 ? x2[i * kStep] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        out1[i * kStep] = ja.x1 ? fma(ja.c1, r[i], y1[i]) : r[i];
        if (ja.out2) out2[i * kStep] = fma(ja.c2, r[i], y2[i]);
      }
    }
    __syncthreads();  // the next tile's copies overwrite what this one's threads read
  }
  cp_async_wait_all();
  if (*abort_flag) {
    for (unsigned n = 0; n < kMaxWaitTries; ++n)
      if (mbar_try_wait(bar, parity ^ 1u)) break;
  }
}

}  // namespace vt
