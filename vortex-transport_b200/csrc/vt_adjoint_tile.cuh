// One reverse RK stage fused into one kernel on the stage kernel's tiles.
//
// The transpose of the stage right-hand side R at the stage state U applied to
// the stage adjoint a (times sa), g = R'(U)^T (sa a), followed by the reverse
// RK4 combine of adjoint_element_kernel, for meshes on which the face phase
// may take the edge-once form (a face's flux is evaluated once for both
// sides: F(u-, u+, -n) = -F(u+, u-, n)). The operators come folded (FoldedOps)
// where they reflect, else as they are (kMapComponent; 10 steps' gradient at
// 128 x 128, p = 2: 1.73 ms, with the two-launch form 2.59). A persistent block
// walks the forward stage kernel's tiles (64 columns, Numbering in
// vt_device.cuh) and keeps every intermediate in shared memory, so nothing but
// the state, the adjoints and the geometry crosses HBM:
//
//   1. load   the tile's stage state, stage adjoint, geometry and face list by
//             bulk copies (issued during the previous tile); the side nodes of
//             the neighbours outside the tile by cp.async;
//   2. lift^T thread (element, component): the lifted face adjoint
//             bF(s, q) = -(len_s/detJ) sa sum_i LIFT_s[i][q] a_i at every face
//             point (the transpose of the lift and of the folded mass
//             inverse), halved: the adjoint of roe_flux2's doubled flux;
//   3. faces  one work item per face and part of its points from the tile's
//             face list. A face between two tile elements is taken once: the
//             transposed Roe Jacobian at (U+, U-) applied to
//             bF_e(q) - bF_nb(nfq-1-q) gives the adjoints of both traces, each
//             written over its element's bF slot. A face leaving the tile is
//             taken by each side, with the neighbour's bF recomputed from its
//             stage adjoint in phase 2, and gives the own trace's adjoint only
//             (the neighbour's tile takes the other);
//   4. traces^T  thread (element, component): the trace adjoints onto the
//             side nodes (transposed trace weights) into Np accumulators; then
//             the transposed volume operator sa sum_i D[d][i][j] a_i per node;
//   5. flux^T the transposed nodal flux Jacobian of every node (its state in
//             shared memory), once; the state tile is then free and the next
//             tile's copies are issued;
//   6. combine acc_out = acc_in + lam_coef lam + g, a_out = cl lam + cg g,
//             thread (element, component).
//
// Threads, columns, buffers and barriers are the stage kernel's (vt_tile.cuh):
// from phase 4 on every shared-memory access stays within an element's threads,
// which lie in one half's four warps, so the barriers after phases 4a, 4b and 5
// are per-half named barriers and each half issues its own next copies; the
// load phase has no block barrier (phase 2 reads only the thread's own column,
// phase 3 comes after a barrier), and a tile ends with a per-half barrier (the
// next tile's phase 2 reuses rows that this tile's phase 6 reads).
//
// Every wait on the mbarrier is bounded; a wait that gives up sets bit 1 of
// err[3] and the block stops taking tiles.
#pragma once

#include "vt_adjoint.cuh"
#include "vt_adjoint_kernels.cuh"
#include "vt_tile.cuh"

namespace vt {

// The operators: as they are, or folded, with the lift as it is for the
// neighbours' adjoints.
template <int P, int NFQ, int MAP>
struct AdjOps {
  StageOps<P, NFQ> o;
  __host__ __device__ static const double* lift(const AdjOps& a) { return &a.o.lift[0][0][0]; }
};
template <int P, int NFQ>
struct AdjOps<P, NFQ, kMapFolded> {
  FoldedOps<P, NFQ> o;
  double full_lift[3][np_of_p(P)][NFQ];
  __host__ __device__ static const double* lift(const AdjOps& a) { return &a.full_lift[0][0][0]; }
};

// The stage kernel's buffers, the stage adjoint tile, and the operator tables
// that the face phase indexes at run time (the face point and the side of a
// work item are not known at compile time).
template <int P, int NFQ>
struct AdjTileLayout {
  using B = TileLayout<P, NFQ>;
  static constexpr int NP = B::NP;
  static constexpr int NE = B::NE;
  static constexpr int kTP = B::kBytes;                        // double [3][NFQ][NE] own trace weights
  static constexpr int kLF = kTP + 3 * NFQ * NE * 8 + 8 * (3 * NFQ * NE % 2);  // double [3][NFQ][NP] LIFT by point
  static constexpr int kA = (kLF + 3 * NP * NFQ * 8 + 127) / 128 * 128;  // double2 [2][2NP][32] stage adjoint
  // double2 [kHARows][2 kSlots]: the slots' stage adjoints, then their lifted face adjoints
  static constexpr int kHARows = 2 * NP > 2 * NFQ ? 2 * NP : 2 * NFQ;
  static constexpr int kHA = kA + 2 * NP * kTileElems * 16;
  static constexpr int kBytes = kHA + kHARows * 2 * kSlots * 16;
};

// The stage adjoint of the neighbour in slot `lane` of half `which`, component
// pair g, by the one thread that lifts it (lift_neighbour).
template <int P>
__device__ __forceinline__ void copy_neighbour_adjoint(double2* HA, const double2* a, unsigned code, int which, int g,
                                                       int lane) {
  constexpr int NP = np_of_p(P);
  if (g > 1 || code == kNoNeighbour) return;
  const double2* src = a + state_index(NP, code >> 2, g);
  double2* dst = HA + g * 2 * kSlots + which * kSlots + lane;
#pragma unroll
  for (int i = 0; i < NP; ++i) cp_async16(dst + i * 4 * kSlots, src + i * 2 * kTileRun);
}

// Its lifted face adjoint at this side's face points (the neighbour's point
// nfq-1-q for point q), in place: row 2 q + h for component pair h = g. Taken
// once per face, from shared memory; formed per face point from the
// neighbour's rows in global memory it was most of the reverse stage's waiting
// (3.4 of 11 cycles per instruction on L2, 2.2 at the barrier behind the face
// phase; 128 x 128 cells, p = 3).
template <int P, int NFQ>
__device__ __forceinline__ void lift_neighbour(double2* HA, const double* LF, unsigned code, double scale, int which,
                                               int g, int lane) {
  constexpr int NP = np_of_p(P);
  if (g > 1 || code == kNoNeighbour) return;
  double2* own = HA + g * 2 * kSlots + which * kSlots + lane;
  double2 v[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) v[i] = own[i * 4 * kSlots];
  const double* lf = LF + (code & 3) * NFQ * NP;
#pragma unroll
  for (int q = 0; q < NFQ; ++q) {
    double x = 0.0, y = 0.0;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const double l = lf[(NFQ - 1 - q) * NP + i];
      x = fma(l, v[i].x, x);
      y = fma(l, v[i].y, y);
    }
    own[q * 4 * kSlots] = make_double2(scale * x, scale * y);
  }
}

// The neighbour's side length over det J.
__device__ __forceinline__ double neighbour_scale(const double2* geo, unsigned code, int g) {
  if (g > 1 || code == kNoNeighbour) return 0.0;
  const unsigned s = code & 3;
  return __ldg(reinterpret_cast<const double*>(geo + geo_index(code >> 2, s < 2 ? 2 : 3)) + (s == 1 ? 1 : 0));
}

// One thread per half announces the bulk copies of block `which` of a tile and
// issues those of the mesh's arrays (geometry and, for block 0, the face list),
// then those of the stage state and stage adjoint.
template <int P, int NFQ>
__device__ __forceinline__ void issue_adj_mesh_copies(const AdjArgs& a, int tile, int which, unsigned char* smem) {
  using B = TileLayout<P, NFQ>;
  constexpr unsigned kState = 2 * B::NP * kTileRun * 16, kGeo = kGeoRows * kTileRun * 16;
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + B::kBar);
  fence_proxy_async_smem();
  mbar_arrive_expect_tx(bar, 2 * kState + kGeo + (which == 0 ? kListOuter : 0u));
  bulk_g2s(smem + B::kGE + which * kGeo, a.geo + (2ll * tile + which) * (kGeoRows * kTileRun), kGeo, bar);
  if (which == 0) bulk_g2s(smem + B::kItems, a.lists + static_cast<long long>(tile) * kTileListBytes, kListOuter, bar);
}
template <int P, int NFQ>
__device__ __forceinline__ void issue_adj_state_copies(const AdjArgs& a, int tile, int which, unsigned char* smem) {
  using L = AdjTileLayout<P, NFQ>;
  using B = TileLayout<P, NFQ>;
  constexpr unsigned kState = 2 * B::NP * kTileRun * 16;
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + B::kBar);
  const long long at = (2ll * tile + which) * (2 * B::NP * kTileRun);
  bulk_g2s(smem + B::kS + which * kState, a.U + at, kState, bar);
  bulk_g2s(smem + L::kA + which * kState, a.a + at, kState, bar);
}

// Even and odd parts of one component of a column's stage adjoint (node pairs
// as sums and differences, the fixed nodes in the even part). Of an empty
// column they are whatever lies there; nothing that is read comes from them.
template <int P>
__device__ __forceinline__ void folded_adjoint(const double* Ad, double* e, double* o) {
  constexpr int NS = fold_nodes(P), NO = fold_pairs(P);
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    const int i = fold_node(P, k);
    const double u = Ad[i * 4 * kTileRun];
    if (k < NO) {
      const double v = Ad[mirror_node(P, i) * 4 * kTileRun];
      e[k] = u + v;
      o[k] = u - v;
    } else {
      e[k] = u;
    }
  }
}

// Two 256-thread blocks per SM: the transposed Roe Jacobian needs more than the
// 80 registers of three blocks, and two leave shared memory for the stage
// adjoint tile.
template <int P, int NFQ, int MAP, bool FAR>
__global__ void __launch_bounds__(4 * kTileElems, 2)
    adjoint_tile_kernel(const __grid_constant__ AdjArgs a, const AdjOps<P, NFQ, MAP> ops) {
  constexpr bool FOLD = MAP == kMapFolded;
  const auto& o = ops.o;
  using B = TileLayout<P, NFQ>;
  using L = AdjTileLayout<P, NFQ>;
  constexpr int E = B::E;
  constexpr int NP = B::NP;
  constexpr int NE = B::NE;
  constexpr int NS = fold_nodes(P), NO = fold_pairs(P), NOA = NO > 0 ? NO : 1;
  constexpr int T = 4 * E;
  extern __shared__ __align__(128) unsigned char smem[];
  double2* S = reinterpret_cast<double2*>(smem + B::kS);  // stage state tile
  double2* H = reinterpret_cast<double2*>(smem + B::kH);
  double* FB = reinterpret_cast<double*>(smem + B::kFB);
  double2* FB2 = reinterpret_cast<double2*>(smem + B::kFB);
  double2* GE = reinterpret_cast<double2*>(smem + B::kGE);
  double* TM = reinterpret_cast<double*>(smem + B::kTM);
  const unsigned short* items = reinterpret_cast<const unsigned short*>(smem + B::kItems);
  const FaceCounts* counts = reinterpret_cast<const FaceCounts*>(smem + B::kItems + kListCount);
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + B::kBar);
  int* abort_flag = reinterpret_cast<int*>(smem + B::kBar + 8);
  int* NEXT = reinterpret_cast<int*>(smem + B::kBar + 12);
  double* TP = reinterpret_cast<double*>(smem + L::kTP);
  double* LF = reinterpret_cast<double*>(smem + L::kLF);
  double2* HA = reinterpret_cast<double2*>(smem + L::kHA);
  const double* Ad = reinterpret_cast<const double*>(smem + L::kA);  // stage adjoint tile

  const int t = threadIdx.x;
  const int lane = t & 31;
  const int which = (t >> 5) & 1;  // this warp's half of the tile
  const int grp = t >> 6;          // and its number among the half's four
  const int col = t % E;           // load and transposed flux phases
  const int el = work_column(t), c = work_component(t);
  const int G = gridDim.x;
  const bool hand_out = a.ntiles > kHandOut * G;

  {
    const double* tm = &o.tm[0][0][0];
    const double* tp = &o.tp[0][0][0];
    const double* lf = AdjOps<P, NFQ, MAP>::lift(ops);
    for (int l = t; l < 3 * NFQ * NE; l += T) {
      TM[l] = tm[l];
      TP[l] = tp[l];
    }
    for (int l = t; l < 3 * NP * NFQ; l += T) {
      const int s = l / (NP * NFQ), i = l / NFQ % NP, q = l % NFQ;
      LF[(s * NFQ + q) * NP + i] = lf[l];
    }
  }
  if (t == 0) {
    mbar_init(bar, 2);
    *abort_flag = 0;
  }

  int tile = blockIdx.x;  // the grid has at most ntiles blocks
  unsigned code = neighbour_code(a.lists, tile, which, lane);
  __syncthreads();
  if (grp == 0 && lane == 0) issue_adj_mesh_copies<P, NFQ>(a, tile, which, smem);
  wait_for_previous();
  let_next_start();
  if (grp == 0 && lane == 0) issue_adj_state_copies<P, NFQ>(a, tile, which, smem);
  copy_neighbours<P>(H, a.U, code, which, grp, lane);
  copy_neighbour_adjoint<P>(HA, a.a, code, which, grp, lane);
  cp_async_commit();
  double scale = neighbour_scale(a.geo, code, grp);
  unsigned parity = 0;
  Ad += sidx<NP>(c >> 1, el) * 2 + (c & 1);              // this thread's component and column
  double* FBt = FB + ((c >> 1) * E + el) * 2 + (c & 1);  // likewise in the face buffer

  while (true) {
    const long long blk = 2ll * tile + which;
    unsigned taken = 0;
    if (t == 224 && hand_out) taken = take_tile(a.err + 6);

    // ---- 1. load ------------------------------------------------------------------
    const bool valid = __ldg(a.elem + blk * kTileRun + (el & 31)) >= 0;
    const double dtt = a.tile_dt ? __ldg(a.tile_dt + tile) : 1.0;
    const double sa = a.sa_dt ? a.sa * dtt : a.sa;
    {
      bool ok = false;
      for (unsigned n = 0; n < kMaxWaitTries && !ok; ++n) ok = mbar_try_wait(bar, parity);
      if (!ok) {
        atomicOr(&a.err[3], 2ull);
        *abort_flag = 1;
      }
    }
    parity ^= 1u;

    // ---- 2. lifted face adjoints (half of them), component c of column el --------------
    const double2* ge = GE + which * kGeoRows * kTileRun + (el & 31);
    const double l0 = sa * ge[2 * kTileRun].x, l1 = sa * ge[2 * kTileRun].y, l2 = sa * ge[3 * kTileRun].x;
    if constexpr (FOLD) {
      double ev[NS], od[NOA];
      folded_adjoint<P>(Ad, ev, od);
#pragma unroll
      for (int q = 0; q < NFQ; ++q) {
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int k = 0; k < NS; ++k) x = fma(o.Le[k][q], ev[k], x);
#pragma unroll
        for (int k = 0; k < NO; ++k) y = fma(o.Lo[k][q], od[k], y);
        FBt[q * 4 * E] = l0 * (x + y);
        FBt[(2 * NFQ + NFQ - 1 - q) * 4 * E] = l2 * (x - y);
      }
#pragma unroll
      for (int q = 0; q < (NFQ + 1) / 2; ++q) {
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int k = 0; k < NS; ++k) x = fma(o.L1e[k][q], ev[k], x);
        if (q < NFQ / 2) {
#pragma unroll
          for (int k = 0; k < NO; ++k) y = fma(o.L1o[k][q], od[k], y);
          FBt[(NFQ + NFQ - 1 - q) * 4 * E] = l1 * (x - y);
        }
        FBt[(NFQ + q) * 4 * E] = l1 * (x + y);
      }
    } else {
      double u[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) u[i] = Ad[i * 4 * kTileRun];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const double ls = -0.5 * (s == 0 ? l0 : (s == 1 ? l1 : l2));
#pragma unroll
        for (int q = 0; q < NFQ; ++q) {
          double x = 0.0;
#pragma unroll
          for (int i = 0; i < NP; ++i) x = fma(o.lift[s][i][q], u[i], x);
          FBt[(s * NFQ + q) * 4 * E] = ls * x;
        }
      }
    }
    cp_async_wait_all();  // this thread's copies of neighbour rows
    lift_neighbour<P, NFQ>(HA, LF, code, -0.5 * sa * scale, which, grp, lane);
    __syncthreads();
    if (*abort_flag) break;

    // ---- 3. faces: transposed Roe Jacobian; the trace adjoints overwrite bF ----------
    const FaceCounts faces = *counts;
    int entry, q, q1;
    for (int w = t; face_work<NFQ>(faces, w, &entry, &q, &q1); w += T) {
      const int it = items[entry];
      const int fl = it & 63, s = (it >> 6) & 3, x = it >> 9;
      const bool mirror = (it >> 8) & 1;
      const double2 n = GE[((fl >> 5) * kGeoRows + 4 + s) * kTileRun + (fl & 31)];
#pragma unroll 1
      for (; q < q1; ++q) {
        const int qm = NFQ - 1 - q;
        double up[4] = {0.0, 0.0, 0.0, 0.0}, um[4] = {0.0, 0.0, 0.0, 0.0}, bf[4];
        double2* own = FB2 + (s * NFQ + q) * 2 * E + fl;
        double2* oth = FB2 + (s * NFQ + qm) * 2 * E + (mirror ? x : 0);
        const double* cp = TP + (s * NFQ + q) * NE;
        const double* cm = (mirror ? TP + (s * NFQ + qm) * NE : TM + (s * NFQ + q) * NE);
        const double2 b0 = own[0], b1 = own[E];
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          const int node = s == 0 ? edge_node(P, 0, k) : (s == 1 ? edge_node(P, 1, k) : edge_node(P, 2, k));
          const double2 x0 = S[sidx<NP>(2 * node, fl)], x1 = S[sidx<NP>(2 * node + 1, fl)];
          up[0] = fma(cp[k], x0.x, up[0]);
          up[1] = fma(cp[k], x0.y, up[1]);
          up[2] = fma(cp[k], x1.x, up[2]);
          up[3] = fma(cp[k], x1.y, up[3]);
          double2 y0, y1;
          if (mirror) {  // the partner's own trace at its point nfq-1-q, as the stage kernel reads it
            y0 = S[sidx<NP>(2 * node, x)];
            y1 = S[sidx<NP>(2 * node + 1, x)];
          } else {
            y0 = H[2 * k * 2 * kSlots + x];
            y1 = H[(2 * k + 1) * 2 * kSlots + x];
          }
          um[0] = fma(cm[k], y0.x, um[0]);
          um[1] = fma(cm[k], y0.y, um[1]);
          um[2] = fma(cm[k], y1.x, um[2]);
          um[3] = fma(cm[k], y1.y, um[3]);
        }
        // the partner's or the neighbour's lifted adjoint at its point nfq-1-q
        const double2* m = mirror ? oth : HA + 4 * q * kSlots + x;
        const double2 m0 = m[0], m1 = m[mirror ? E : 2 * kSlots];
        bf[0] = b0.x - m0.x, bf[1] = b0.y - m0.y, bf[2] = b1.x - m1.x, bf[3] = b1.y - m1.y;
        double bu[4], bv[4];
        roe_flux2_vjp(up, um, n.x, n.y, bf, bu, bv);
        own[0] = make_double2(bu[0], bu[1]);
        own[E] = make_double2(bu[2], bu[3]);
        if (mirror) {
          oth[0] = make_double2(bv[0], bv[1]);
          oth[E] = make_double2(bv[2], bv[3]);
        }
      }
    }
    if constexpr (FAR) {
      FarFace x;
      for (int w = t; far_face<NFQ>(faces, items, a.nbr, tile, w, &x); w += T) {
        const double2 n = GE[((x.col >> 5) * kGeoRows + 4 + x.s) * kTileRun + (x.col & 31)];
        double2* own = FB2 + (x.s * NFQ + x.q) * 2 * E + x.col;
        const double2 b0 = own[0], b1 = own[E];
        double up[4] = {0.0, 0.0, 0.0, 0.0}, um[4];
        const double* cp = TP + (x.s * NFQ + x.q) * NE;
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          const int node = x.s == 0 ? edge_node(P, 0, k) : (x.s == 1 ? edge_node(P, 1, k) : edge_node(P, 2, k));
          const double2 x0 = S[sidx<NP>(2 * node, x.col)], x1 = S[sidx<NP>(2 * node + 1, x.col)];
          up[0] = fma(cp[k], x0.x, up[0]);
          up[1] = fma(cp[k], x0.y, up[1]);
          up[2] = fma(cp[k], x1.x, up[2]);
          up[3] = fma(cp[k], x1.y, up[3]);
        }
        far_trace<P>(a.U, x, TM + (x.s * NFQ + x.q) * NE, um, [](const double2* p) { return *p; });
        // the neighbour's lifted adjoint at its point nfq-1-q
        const double* gn = reinterpret_cast<const double*>(a.geo + geo_index(x.nb, x.s < 2 ? 2 : 3));
        const double sc = -0.5 * sa * __ldg(gn + (x.s == 1 ? 1 : 0));
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        const double* lf = LF + (x.s * NFQ + NFQ - 1 - x.q) * NP;
        const double2* src = a.a + state_index(NP, x.nb, 0);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          const double2 a0 = src[2 * i * kTileRun], a1 = src[(2 * i + 1) * kTileRun];
          v[0] = fma(lf[i], a0.x, v[0]);
          v[1] = fma(lf[i], a0.y, v[1]);
          v[2] = fma(lf[i], a1.x, v[2]);
          v[3] = fma(lf[i], a1.y, v[3]);
        }
        const double bf[4] = {fma(-sc, v[0], b0.x), fma(-sc, v[1], b0.y), fma(-sc, v[2], b1.x), fma(-sc, v[3], b1.y)};
        double bu[4], bv[4];
        roe_flux2_vjp(up, um, n.x, n.y, bf, bu, bv);
        own[0] = make_double2(bu[0], bu[1]);
        own[E] = make_double2(bu[2], bu[3]);
      }
    }
    if (t == 224) *NEXT = hand_out ? static_cast<int>(taken) + G : tile + G;
    __syncthreads();
    const int next = *NEXT;
    const bool has_next = next < a.ntiles;

    // the next tile's neighbours: their codes now, their rows after the transposed flux
    code = has_next ? neighbour_code(a.lists, next, which, lane) : kNoNeighbour;

    // ---- 4a. trace adjoints onto the side nodes, component c --------------------------
    double g[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) g[i] = 0.0;
#pragma unroll
    for (int s = 0; s < 3; ++s)
#pragma unroll
      for (int q = 0; q < NFQ; ++q) {
        const double b = FBt[(s * NFQ + q) * 4 * E];
#pragma unroll
        for (int k = 0; k < NE; ++k) g[edge_node(P, s, k)] = fma(o.tp[s][q][k], b, g[edge_node(P, s, k)]);
      }
    run_sync(t);

    // ---- 4b. transposed volume operator: rows j*4 + h (xi), j*4 + 2 + h (eta) ----------
    if constexpr (P > 0 && FOLD) {
      double ev[NS], od[NOA];
      folded_adjoint<P>(Ad, ev, od);
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int k = 0; k < NS; ++k) x = fma(o.De[k][j], ev[k], x);
#pragma unroll
        for (int k = 0; k < NO; ++k) y = fma(o.Do[k][j], od[k], y);
        FBt[j * 8 * E] = sa * (x + y);
        FBt[(mirror_node(P, j) * 8 + 4) * E] = sa * (x - y);
      }
    } else if constexpr (P > 0) {
      double u[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) u[i] = Ad[i * 4 * kTileRun];
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          x = fma(o.D[0][i][j], u[i], x);
          y = fma(o.D[1][i][j], u[i], y);
        }
        FBt[j * 8 * E] = sa * x;
        FBt[(j * 8 + 4) * E] = sa * y;
      }
    }
    // the combine's operands, requested now so that they are in flight during
    // the transposed flux (every load before the first store: acc_in and
    // acc_out are the same array in three of the four reverse stages)
    constexpr int kStep = 4 * kTileRun;  // doubles between node rows of the same pair
    const long long off0 = blk * (4 * NP * kTileRun) + (c >> 1) * (2 * kTileRun) + (el & 31) * 2 + (c & 1);
    double lv[NP], av[NP];
    {
      const bool need_lam = valid && (a.lam_coef != 0.0 || a.a_out);
      const bool need_acc = valid && a.acc_in;
      const double* lam = reinterpret_cast<const double*>(a.lam) + off0;
      const double* acc_in = reinterpret_cast<const double*>(a.acc_in) + off0;
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        lv[i] = need_lam ? ld_early_rw(lam + i * kStep) : 0.0;
        av[i] = need_acc ? ld_early_rw(acc_in + i * kStep) : 0.0;
      }
    }
    run_sync(t);

    // ---- 5. transposed nodal flux Jacobian of every node, in place over the xi rows ----
    if (P > 0) {
      const double2* ge = GE + which * kGeoRows * kTileRun + lane;
      const double2 j0 = ge[0], j1 = ge[kTileRun];
      for (int j = grp; j < NP; j += 4) {
        const double2 s0 = S[sidx<NP>(2 * j, col)], s1 = S[sidx<NP>(2 * j + 1, col)];
        const double sv[4] = {s0.x, s0.y, s1.x, s1.y};
        double2* gp = FB2 + j * 4 * E + col;
        const double2 x0 = gp[0], x1 = gp[E], y0 = gp[2 * E], y1 = gp[3 * E];
        const double bx[4] = {x0.x, x0.y, x1.x, x1.y}, by[4] = {y0.x, y0.y, y1.x, y1.y};
        double gv[4];
        contravariant_vjp(sv, j0.x, j0.y, j1.x, j1.y, bx, by, gv);
        gp[0] = make_double2(gv[0], gv[1]);
        gp[E] = make_double2(gv[2], gv[3]);
      }
    }
    run_sync(t);

    // this half's columns of the state and adjoint tiles are free: start its
    // next copies and the next tile's neighbour rows
    if (has_next) {
      if (grp == 0 && lane == 0) {
        issue_adj_mesh_copies<P, NFQ>(a, next, which, smem);
        issue_adj_state_copies<P, NFQ>(a, next, which, smem);
      }
      copy_neighbours<P>(H, a.U, code, which, grp, lane);
      copy_neighbour_adjoint<P>(HA, a.a, code, which, grp, lane);
      scale = neighbour_scale(a.geo, code, grp);
    }
    cp_async_commit();

    // ---- 6. reverse RK combine -------------------------------------------------------------
    if (valid) {
      const double cl = a.tile_dt ? a.cl * dtt : a.cl, cg = a.tile_dt ? a.cg * dtt : a.cg;
      double* acc_out = reinterpret_cast<double*>(a.acc_out) + off0;
      double* a_out = reinterpret_cast<double*>(a.a_out) + off0;
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        const double gi = P > 0 ? g[i] + FBt[i * 8 * E] : g[i];
        acc_out[i * kStep] = fma(a.lam_coef, lv[i], av[i]) + gi;
        if (a.a_out) a_out[i * kStep] = fma(cl, lv[i], cg * gi);
      }
    }
    // the four warps of a half hold different components of the same columns:
    // none may start the next tile's phase 2 (which reuses rows of the face /
    // flux buffer) before the others are done with this tile's
    run_sync(t);
    if (!has_next) break;
    tile = next;
  }

  cp_async_wait_all();  // none may land after the block has left
  if (*abort_flag) {
    // the bulk copies of a tile whose wait gave up may still land: wait for
    // them once more, with the same bound, before the block leaves
    for (unsigned n = 0; n < kMaxWaitTries; ++n)
      if (mbar_try_wait(bar, parity ^ 1u)) break;
  }
  if (t == 0 && hand_out) {
    __threadfence();
    if (atomicAdd(&a.err[5], 1ull) == gridDim.x - 1) {
      a.err[5] = 0ull;
      a.err[6] = 0ull;
    }
  }
}

}  // namespace vt
