// The fused RK stage kernel, tiled through shared memory.
//
// A persistent block walks tiles of 64 columns (two blocks of 32 elements,
// Numbering in vt_device.cuh) and advances each through one stage of the nodal
// DG scheme (Evolve.cpp:135-308, numerical_flux Numericalflux.cpp:13-157,
// stage update Timestepping.cpp:85-306 / :39-82). The state crosses HBM once
// per stage:
//
//   1. load   the tile's state, geometry and face list arrive in shared memory
//             by bulk copies (cp.async.bulk, contiguous in HBM, completion on
//             an mbarrier), issued when that half finished the previous tile's
//             flux phase; the side nodes of the neighbours outside the tile
//             (one slot per face that leaves it) come by cp.async at the same
//             time;
//   2. traces a thread evaluates its element's own trace of its component at
//             every face point from the p+1 side nodes (coefficients are
//             immediates);
//   3. faces  one work item per face and part of its points from the list
//             built once at set-up (vt_schedule.cuh), sorted so warps stay on
//             one path. A face between two tile elements is evaluated once, by
//             the earlier element: its outer state is the partner's own trace
//             at the mirrored point nfq-1-q, and the flux is written over both
//             traces (the partner gets -F, its outward normal being -n). A
//             face leaving the tile is evaluated by each side, as in the
//             reference, with the outer trace from the neighbour's nodes;
//   4. lift   surface term -(len_s/detJ) LIFT_s F_s into Np accumulators;
//   5. flux   the nodal Euler flux of every node, contracted with the inverse
//             Jacobian, once, into shared memory; the state tile is then free
//             and the next tile's copies are issued;
//   6. volume D_xi G_xi + D_eta G_eta, then the RK stage update written back.
//
// From phase 4 on, every shared-memory access stays within an element's
// threads, which lie in the four warps of equal parity (warps 0, 2, 4, 6 hold
// the first block's columns, 1, 3, 5, 7 the second's). So the barriers after
// phases 4 and 5 are per-half 128-thread named barriers, and each half issues
// its own next copies (the tile's mbarrier expects one arrival per half). The
// load phase has no block barrier either: the traces read only columns of the
// thread's own half of the state tile, which its own wait on the mbarrier
// covers, and the other half's geometry and element numbers and the neighbour
// rows are first read in phase 3, after the barrier that follows the traces. A
// tile ends with a per-half barrier: the four warps of a half share its columns, and the
// next tile's traces reuse rows of the buffer that this tile's volume phase
// reads. So the two halves of a block run apart from phase 4 of one tile to the
// end of the next tile's trace phase.
//
// What bounds it (768 x 768 cells, p = 3, nfq = 6; phase clocks and counters):
// neither HBM nor one pipe, but the instructions and latencies of 24 warps per
// SM (80 registers and 75 KB of shared memory allow three blocks), a warp
// issuing one instruction in about nine cycles. So the layout and the
// formulas are chosen for few instructions:
//   - the bulk copies and the constant row distances of the block layout leave
//     one address computation per phase, and no registers hold anything of the
//     next tile but its neighbours' codes;
//   - every shared-memory access takes its minimum of wavefronts: the face and
//     flux buffers are rows of 64 columns of component pairs (double2); phases
//     2, 4 and 6 put 16 consecutive columns x the two components of a pair into
//     a warp (8-byte accesses to 256 contiguous bytes, in shared and in global
//     memory), and a warp's faces are consecutive in the list, which on the
//     reference's mesh means consecutive columns, all at the same point;
//   - roe_flux2, contravariant_flux and the folded operators (vt_device.cuh).
// The reference's mass-inverse apply is folded into D and LIFT on the host.
//
// Every wait on the mbarrier is bounded; a wait that gives up sets bit 1 of
// err[3], and the block stops taking tiles. StageArgs::wait_tries and
// test_flags (vt_test_bulk_wait) let a test shorten the bound and issue no
// copies, so that the give-up path runs without any copy in flight.
#pragma once

#include "vt_device.cuh"

namespace vt {

template <int P, int NFQ>
struct TileLayout {
  static constexpr int E = kTileElems;
  static constexpr int NP = np_of_p(P);
  static constexpr int NE = P + 1;
  static constexpr int kFBRows = 6 * NFQ > NP * 4 ? 6 * NFQ : NP * 4;
  // byte offsets into dynamic shared memory, each 16-byte aligned
  static constexpr int kS = 0;                               // double2 [2][2NP][32]
  static constexpr int kH = kS + 2 * NP * E * 16;            // double2 [2NE][2 kSlots] neighbours' side nodes
  static constexpr int kFB = kH + 2 * NE * 2 * kSlots * 16;  // double2 [3][NFQ][2][E] | [NP][4][E]
  static constexpr int kGE = kFB + kFBRows * E * 16;         // double2 [2][kGeoRows][32] geometry
  static constexpr int kTM = kGE + kGeoRows * E * 16;        // double [3][NFQ][NE]
  static constexpr int kEL = kTM + 3 * NFQ * NE * 8 + 8 * (3 * NFQ * NE % 2);  // int [E] element of each column
  static constexpr int kItems = kEL + E * 4;                 // uint16 [kMaxItems], uint32 [4] (face list)
  static constexpr int kBar = kItems + kListOuter;           // mbarrier (8 B), abort flag, next tile
  static constexpr int kBytes = kBar + 16;
};

// ---- asynchronous copies ---------------------------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}

// true once the phase with parity `parity` has completed.
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Global-to-shared copies that bypass the registers (cp.async, completed per
// thread by cp.async.wait_all): 16 bytes (both addresses 16-byte aligned),
// cached in L2 only.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(__cvta_generic_to_global(src))
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Contiguous bulk copies: both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(src)), "r"(bytes)
               : "memory");
}

// Programmatic dependent launch (launch_dependent, vt_launch.h): after
// let_next_start the next kernel of the stream may be scheduled where this grid
// leaves room, and does its set-up there until wait_for_previous, which returns
// when the kernel before it has ended and its writes are visible. Every kernel
// launched that way waits before it reads or writes anything that another
// kernel writes or reads; only the mesh's own arrays, which no kernel of the
// stream writes, are read before. Only those are read by non-coherent loads
// (__ldg), too: a vector that the kernel before writes changes while this grid
// exists, which such loads do not allow for. let_next_start comes after the own wait, so
// that at most one later kernel is resident: when it came first, several were,
// and blocks of one kernel shared an SM while other SMs had none. 50 RK4 steps
// at 64 x 64 cells, p = 2 (128 tiles) take 1.23 ms without it, 1.79 with
// let_next_start first and 1.12 as it is; 250 at 8 x 8, p = 3 6.35, 6.42 and
// 6.18; 20 at 150 x 90, p = 3 0.91, 0.88 and 0.87; large meshes the same.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Which tile a block takes next. A block's first tile is blockIdx.x, the others
// are handed out in order by an atomic counter, so that the blocks of SMs that
// run ahead (their distance to the L2 slices differs) take more of them: with
// tiles blockIdx.x + k gridDim.x the blocks ended up to 30 us apart at 768 x
// 768, p = 3. The counter is read while the previous tile's faces are
// evaluated; the last block to finish clears it. No result depends on the
// assignment. A pass of 5 RK4 steps at 768 x 768, p = 3 (41 tiles a block)
// takes 7.28 ms handed out, 7.54 ms otherwise; with few tiles a block there is
// little to even out and the counter costs more: 384 x 384, p = 1 (10 tiles a
// block) 4.22 against 4.18 ms, a gradient at 128 x 128, p = 3 (1 or 2 tiles)
// 16.1 against 14.1 ms. So it is used from kHandOut tiles a block on.
constexpr int kHandOut = 16;
__device__ __forceinline__ unsigned take_tile(unsigned long long* taken) {
  return atomicAdd(reinterpret_cast<unsigned*>(taken), 1u);
}

constexpr unsigned kMaxWaitTries = 1u << 22;

// Shared-memory index of (row, column) of the state tile: the two blocks as they lie in HBM.
template <int NP>
__device__ __forceinline__ int sidx(int row, int col) {
  return ((col >> 5) * 2 * NP + row) * kTileRun + (col & (kTileRun - 1));
}

// One thread per half announces the bulk copies of block `which` of a tile and
// issues those of the mesh's arrays (geometry, element numbers and, for block
// 0, the face list), then the state's.
template <int P, int NFQ>
__device__ __forceinline__ void issue_mesh_copies(const StageArgs& a, int tile, int which, unsigned char* smem) {
  using L = TileLayout<P, NFQ>;
  constexpr unsigned kState = 2 * L::NP * kTileRun * 16, kGeo = kGeoRows * kTileRun * 16, kElem = kTileRun * 4;
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + L::kBar);
  if (a.test_flags & kTestNoCopies) return;  // test hook: nothing arrives, every wait gives up
  fence_proxy_async_smem();
  mbar_arrive_expect_tx(bar, kState + kGeo + (a.elem ? kElem : 0u) + (which == 0 ? kListOuter : 0u));
  const long long blk = 2ll * tile + which;
  bulk_g2s(smem + L::kGE + which * kGeo, a.geo + blk * (kGeoRows * kTileRun), kGeo, bar);
  if (a.elem) bulk_g2s(smem + L::kEL + which * kElem, a.elem + blk * kTileRun, kElem, bar);
  if (which == 0) bulk_g2s(smem + L::kItems, a.lists + static_cast<long long>(tile) * kTileListBytes, kListOuter, bar);
}
template <int P, int NFQ>
__device__ __forceinline__ void issue_state_copy(const double2* in, int tile, int which, unsigned char* smem,
                                                 int test_flags) {
  using L = TileLayout<P, NFQ>;
  constexpr unsigned kState = 2 * L::NP * kTileRun * 16;
  if (test_flags & kTestNoCopies) return;
  bulk_g2s(smem + L::kS + which * kState, in + (2ll * tile + which) * (2 * L::NP * kTileRun), kState,
           reinterpret_cast<unsigned long long*>(smem + L::kBar));
}

// Barrier of the four warps that hold one half's columns (warps of equal parity).
__device__ __forceinline__ void run_sync(int t) {
  if ((t >> 5) & 1) asm volatile("bar.sync 2, 128;" ::: "memory");
  else asm volatile("bar.sync 1, 128;" ::: "memory");
}

// ---- threads and work -------------------------------------------------------------
// Phases 2, 4 and 6: a thread holds one component of one element and all its
// nodes. Warp w works on half w & 1, component pair (w >> 1) & 1 and columns
// 16 (w >> 2) ... + 15 of the half; its lanes are the columns x the pair's two
// components. (Phase 5, one element and all components per thread, uses column
// t % 64 and the group t / 64.)
//
// Two forms of the lift and the volume operator (select_kernel, vt_launch.cu):
// kMapComponent applies the operators as they are; kMapFolded, where they
// reflect under xi <-> eta, holds the even and odd parts of the node pairs
// (FoldedOps): 117 + 128 FP64 instructions per element and component at p = 3,
// nfq = 6, against 198 + 200. The FP64 pipe was the stage kernel's most used
// unit (54% busy) and these two 44% of its instructions.
__device__ __forceinline__ int work_column(int t) {
  return ((t >> 5) & 1) * kTileRun + (t >> 7) * 16 + ((t & 31) >> 1);
}
__device__ __forceinline__ int work_component(int t) { return ((t >> 6) & 1) * 2 + (t & 1); }

// Traces of component c of column el at every face point (or at the points
// FIRST ... END - 1 of the three sides').
template <int P, int NFQ, int FIRST = 0, int END = 3 * NFQ, typename Ops>
__device__ __forceinline__ void own_traces(const Ops& ops, const double2* S, double* FB, int el, int c) {
  constexpr int NP = np_of_p(P), NE = P + 1, ES = kTileElems;
  const double* Sd = reinterpret_cast<const double*>(S) + sidx<NP>(c >> 1, el) * 2 + (c & 1);
  double* out = FB + ((c >> 1) * ES + el) * 2 + (c & 1);
  double u[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) u[i] = Sd[i * 4 * kTileRun];
#pragma unroll
  for (int s = 0; s < 3; ++s)
#pragma unroll
    for (int q = 0; q < NFQ; ++q) {
      if (s * NFQ + q < FIRST || s * NFQ + q >= END) continue;
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < NE; ++k) v = fma(ops.tp[s][q][k], u[edge_node(P, s, k)], v);
      out[(s * NFQ + q) * 4 * ES] = v;
    }
}

// F points at the thread's component and column of the face buffer's row 0 (a
// face point's rows are 4 ES doubles apart), G likewise at the flux buffer's.
template <int P, int NFQ>
__device__ __forceinline__ void lift_term(const StageOps<P, NFQ>& ops, const double* F, double2 lsa, double2 lsb,
                                          double* r) {
  constexpr int NP = np_of_p(P), ES = kTileElems;
#pragma unroll
  for (int i = 0; i < NP; ++i) r[i] = 0.0;
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const double ls = 0.5 * (s == 0 ? lsa.x : (s == 1 ? lsa.y : lsb.x));  // the half of roe_flux2
#pragma unroll
    for (int q = 0; q < NFQ; ++q) {
      const double fs = ls * F[(s * NFQ + q) * 4 * ES];
#pragma unroll
      for (int i = 0; i < NP; ++i) r[i] = fma(-ops.lift[s][i][q], fs, r[i]);
    }
  }
}

template <int P, int NFQ>
__device__ __forceinline__ void volume_term(const StageOps<P, NFQ>& ops, const double* G, double* r) {
  constexpr int NP = np_of_p(P), ES = kTileElems;
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const double gx = G[j * 8 * ES], gy = G[(j * 8 + 4) * ES];
#pragma unroll
    for (int i = 0; i < NP; ++i) r[i] = fma(ops.D[0][i][j], gx, fma(ops.D[1][i][j], gy, r[i]));
  }
}

// The folded terms give the even parts, the odd parts, or both in this order.
template <int P, int NFQ, bool EVEN = true, bool ODD = true>
__device__ __forceinline__ void lift_term(const FoldedOps<P, NFQ>& ops, const double* F, double2 lsa, double2 lsb,
                                          double* r) {
  constexpr int ES = kTileElems, NS = EVEN ? FoldedOps<P, NFQ>::NS : 0, NO = ODD ? FoldedOps<P, NFQ>::NO : 0;
#pragma unroll
  for (int a = 0; a < NS + NO; ++a) r[a] = 0.0;
#pragma unroll
  for (int q = 0; q < NFQ; ++q) {
    const double f0 = lsa.x * F[q * 4 * ES], f2 = F[(2 * NFQ + NFQ - 1 - q) * 4 * ES];
    const double fe = fma(lsb.x, f2, f0), fo = fma(-lsb.x, f2, f0);
#pragma unroll
    for (int a = 0; a < NS; ++a) r[a] = fma(ops.Le[a][q], fe, r[a]);
#pragma unroll
    for (int a = 0; a < NO; ++a) r[NS + a] = fma(ops.Lo[a][q], fo, r[NS + a]);
  }
#pragma unroll
  for (int q = 0; q < (NFQ + 1) / 2; ++q) {
    const double f1 = lsa.y * F[(NFQ + q) * 4 * ES];
    double fe = f1, fo = 0.0;
    if (q < NFQ / 2) {
      const double fm = F[(NFQ + NFQ - 1 - q) * 4 * ES];
      fe = fma(lsa.y, fm, f1);
      fo = fma(-lsa.y, fm, f1);
    }
#pragma unroll
    for (int a = 0; a < NS; ++a) r[a] = fma(ops.L1e[a][q], fe, r[a]);
    if (q < NFQ / 2) {
#pragma unroll
      for (int a = 0; a < NO; ++a) r[NS + a] = fma(ops.L1o[a][q], fo, r[NS + a]);
    }
  }
}

// Stage 3's U3 / (3 c_out) (f = 1 / (3 c_out)) added to the even and odd parts.
template <int P, bool EVEN = true, bool ODD = true>
__device__ __forceinline__ void folded_state(const double2* S, int el, int c, double f, double* r) {
  constexpr int NP = np_of_p(P), NS = fold_nodes(P), NO = fold_pairs(P);
  const double* Sd = reinterpret_cast<const double*>(S) + sidx<NP>(c >> 1, el) * 2 + (c & 1);
#pragma unroll
  for (int a = 0; a < (EVEN ? NS : NO); ++a) {
    const double u = Sd[fold_node(P, a) * 4 * kTileRun];
    if (a < NO) {
      const double v = Sd[mirror_node(P, fold_node(P, a)) * 4 * kTileRun];
      if (EVEN) r[a] = fma(0.5 * f, u + v, r[a]);
      if (ODD) r[(EVEN ? NS : 0) + a] = fma(0.5 * f, u - v, r[(EVEN ? NS : 0) + a]);
    } else {
      r[a] = fma(f, u, r[a]);
    }
  }
}

// Nodal fluxes in the form that the folded volume operator reads: for node j
// with mirror image Pj, rows j*4 + h hold Gxi_j + Geta_Pj and rows j*4 + 2 + h
// Gxi_j - Geta_Pj (component pair h). A thread takes both nodes of a pair, or
// one fixed node, of column el (group grp of G); flux(j, gxi, geta) is node j's.
// With FACTORED it gives the energy flux as contravariant_flux<true> does: the
// roundings of the sums are then spelled out (the first node's products are
// rounded, the second's go into multiply-adds), since the kernels that share
// this function must agree bit for bit and the compiler's choice varies. Both
// nodes' products in multiply-adds, which need more registers, took 0.888 ms
// at 150 x 90, p = 3, 20 steps, against 0.869.
template <int P, int G = 4, bool FACTORED = false, typename Flux>
__device__ __forceinline__ void folded_flux_rows(double2* G2, int el, int grp, Flux&& flux) {
  constexpr int ES = kTileElems, NS = fold_nodes(P), NO = fold_pairs(P);
  auto store = [&](int j, const double* gxi, const double* geta, double even, double odd) {
    double2* g = G2 + j * 4 * ES + el;
    g[0] = make_double2(gxi[0] + geta[0], gxi[1] + geta[1]);
    g[ES] = make_double2(gxi[2] + geta[2], even);
    g[2 * ES] = make_double2(gxi[0] - geta[0], gxi[1] - geta[1]);
    g[3 * ES] = make_double2(gxi[2] - geta[2], odd);
  };
#pragma unroll
  for (int u0 = 0; u0 < NS; u0 += G) {
    const int u = u0 + grp;  // uniform per warp
    if (u >= NS) break;
    int j = 0;
#pragma unroll
    for (int k = u0; k < u0 + G && k < NS; ++k)
      if (u == k) j = fold_node(P, k);
    double gxi[5], geta[5];
    flux(j, gxi, geta);
    if constexpr (FACTORED) gxi[3] = __dmul_rn(gxi[4], gxi[3]), geta[3] = __dmul_rn(geta[4], geta[3]);
    if (u < NO) {
      int m = 0;
#pragma unroll
      for (int k = u0; k < u0 + G && k < NO; ++k)
        if (u == k) m = mirror_node(P, fold_node(P, k));
      double hxi[5], heta[5];
      flux(m, hxi, heta);
      if constexpr (FACTORED) {
        store(j, gxi, heta, fma(heta[4], heta[3], gxi[3]), fma(-heta[4], heta[3], gxi[3]));
        store(m, hxi, geta, fma(hxi[4], hxi[3], geta[3]), fma(hxi[4], hxi[3], -geta[3]));
      } else {
        store(j, gxi, heta, gxi[3] + heta[3], gxi[3] - heta[3]);
        store(m, hxi, geta, hxi[3] + geta[3], hxi[3] - geta[3]);
      }
    } else {
      store(j, gxi, geta, gxi[3] + geta[3], gxi[3] - geta[3]);
    }
  }
}

template <int P, int G = 4>
__device__ __forceinline__ void folded_nodal_flux(const double2* S, double2* G2, int el, int grp, double2 j0,
                                                  double2 j1) {
  constexpr int NP = np_of_p(P);
  folded_flux_rows<P, G, true>(G2, el, grp, [&](int j, double* gxi, double* geta) {
    const double2 s0 = S[sidx<NP>(2 * j, el)], s1 = S[sidx<NP>(2 * j + 1, el)];
    const double sv[4] = {s0.x, s0.y, s1.x, s1.y};
    contravariant_flux<true>(sv, j0.x, j0.y, j1.x, j1.y, gxi, geta);
  });
}

template <int P, int NFQ, bool EVEN = true, bool ODD = true>
__device__ __forceinline__ void volume_term(const FoldedOps<P, NFQ>& ops, const double* G, double* r) {
  constexpr int NP = np_of_p(P), ES = kTileElems;
  constexpr int NS = EVEN ? FoldedOps<P, NFQ>::NS : 0, NO = ODD ? FoldedOps<P, NFQ>::NO : 0;
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const double ge = G[j * 8 * ES], go = G[(j * 8 + 4) * ES];
#pragma unroll
    for (int a = 0; a < NS; ++a) r[a] = fma(ops.De[a][j], ge, r[a]);
#pragma unroll
    for (int a = 0; a < NO; ++a) r[NS + a] = fma(ops.Do[a][j], go, r[NS + a]);
  }
}

// Even and odd parts -> the nodes' own values, in place.
template <int P>
__device__ __forceinline__ void unfold(double* r) {
  constexpr int NP = np_of_p(P), NS = fold_nodes(P), NO = fold_pairs(P);
  double v[NP];
#pragma unroll
  for (int a = 0; a < NS; ++a) {
    const int j = fold_node(P, a);
    if (a < NO) {
      v[j] = r[a] + r[NS + a];
      v[mirror_node(P, j)] = r[a] - r[NS + a];
    } else {
      v[j] = r[a];
    }
  }
#pragma unroll
  for (int i = 0; i < NP; ++i) r[i] = v[i];
}

// The nodal flux as the unfolded volume operator reads it: rows j*4 + h xi,
// j*4 + 2 + h eta (component pair h). A thread takes every fourth node.
template <int P>
__device__ __forceinline__ void plain_nodal_flux(const double2* S, double2* G2, int el, int grp, double2 j0,
                                                 double2 j1) {
  constexpr int NP = np_of_p(P), ES = kTileElems;
  for (int j = grp; j < NP; j += 4) {
    const double2 s0 = S[sidx<NP>(2 * j, el)], s1 = S[sidx<NP>(2 * j + 1, el)];
    const double sv[4] = {s0.x, s0.y, s1.x, s1.y};
    double gxi[4], geta[4];
    contravariant_flux(sv, j0.x, j0.y, j1.x, j1.y, gxi, geta);
    double2* g = G2 + j * 4 * ES + el;
    g[0] = make_double2(gxi[0], gxi[1]);
    g[ES] = make_double2(gxi[2], gxi[3]);
    g[2 * ES] = make_double2(geta[0], geta[1]);
    g[3 * ES] = make_double2(geta[2], geta[3]);
  }
}

// Loads issued where they are written, so that the stage update's first operand
// is in flight during the volume phase (the compiler would otherwise sink them
// to their use), and so that stage 1's re-read of its input stays in the update
// (plain loads were hoisted and spilled). They do not allocate in L1: three
// 73 KB blocks leave about 30 KB of it, which the tile's geometry rows use, and
// each operand row is read once (0.2% faster at 768 x 768, p = 3).
__device__ __forceinline__ double ld_early(const double* p) {
  double v;
  asm volatile("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// The same for an array that this kernel writes elsewhere (no other thread
// writes the loaded element).
__device__ __forceinline__ double ld_early_rw(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}

// The RK4 step in 12 state-vector passes. Classical RK4 (Timestepping.cpp:85-306)
// with k_i the right-hand side at stage i's input has the stage states
// U1 = U + dt/2 k1, U2 = U + dt/2 k2, U3 = U + dt k3, and since
// dt/6 k1 = (U1 - U)/3 and dt/3 k3 = (U3 - U)/3 its new state is
// X + U3/3 + dt/6 k4 with X = (U + U1)/3 + dt/3 k2:
//   stage 0: reads U,              writes U1
//   stage 1: reads U1, U (and U1 again from L2), writes U2 and X
//   stage 2: reads U2, U,          writes U3
//   stage 3: reads U3, X,          writes U_{n+1}
// against 16 passes when the accumulator is carried through every stage. The
// stage states are formed as before, bit for bit; only the last stage's sum is
// grouped differently (rounding level). Stage 3 adds U3/3 by starting its
// accumulators at U3/(3 c_out) while the state tile is still in shared memory.
// The coefficient ratios are classical RK4's: (dt/6)/(dt/2) = (dt/3)/dt = 1/3.
constexpr double kThird = 1.0 / 3.0;

// The stage's read-only operand that the update needs besides the
// accumulator: U_n (stage 0, forward Euler), X (stage 3) or the base U_n
// (stages 1, 2); none for the bare right-hand side.
__device__ __forceinline__ const double2* first_operand(const StageArgs& a) {
  return (a.stage == 0 || a.stage == kStageEuler) ? a.in : (a.stage == 3 ? a.acc : a.base);
}

// Neighbours' side nodes of a tile into the slots of half `which`: warp g of
// the half's four copies the two rows of side node g (16 bytes each) of the
// neighbour whose code (StageArgs::lists) each lane holds.
template <int P>
__device__ __forceinline__ void copy_neighbours(double2* H, const double2* in, unsigned code, int which, int g, int lane) {
  static_assert(P + 1 <= 4, "a warp per side node");
  if (g > P || code == kNoNeighbour) return;  // lanes past the slots hold no code
  const int base = g * (P + 1) - g * (g - 1) / 2;  // node_id(P, 0, g)
  const unsigned s = code & 3;
  const int node = s == 0 ? g : (s == 1 ? base + P - g : base);  // edge_node(P, s, g)
  const double2* src = in + state_index(np_of_p(P), code >> 2, 2 * node);
  double2* dst = H + 2 * g * 2 * kSlots + which * kSlots + lane;
  cp_async16(dst, src);
  cp_async16(dst + 2 * kSlots, src + kTileRun);
}

// The code of slot `lane` of half `which` of a tile.
__device__ __forceinline__ unsigned neighbour_code(const unsigned char* lists, int tile, int which, int lane) {
  if (lane >= kSlots) return kNoNeighbour;
  return __ldg(reinterpret_cast<const unsigned*>(lists + static_cast<long long>(tile) * kTileListBytes + kListOuter) +
               which * kSlots + lane);
}

// Face points of faces whose neighbour has no slot: a tile has up to 192 leaving
// faces where the elements' order does not follow the mesh (33 per half where it
// follows its rows, from 23 cells a row on). Only the kernels with FAR take them,
// and a mesh without such faces takes the others: the loop costs registers. Point
// w is point w % nfq of far face w / nfq, so that the lanes of a warp read the
// same few neighbours' nodes; when each lane had a face of its own, as in the
// list's other classes, and read it again for each of its points, 4 RK4 steps at
// 200 x 200 cells in random order, p = 3 took 1.55 ms (now 0.80) and a gradient
// of 10 steps 20.8 (now 8.8).
struct FarFace {
  int col, s, q;  // column in the tile, side, point
  int nb;         // the neighbour's column
};
template <int NFQ>
__device__ __forceinline__ bool far_face(const FaceCounts& f, const unsigned short* items, const int4* nbr, int tile, int w,
                                         FarFace* x) {
  const int k = w / NFQ;
  if (k >= static_cast<int>(f.n >> 16)) return false;
  const int it = items[(f.n & 0xff) + ((f.n >> 8) & 0xff) + k];
  x->col = it & 63, x->s = (it >> 6) & 3, x->q = w - k * NFQ;
  x->nb = __ldg(reinterpret_cast<const int*>(nbr + (static_cast<long long>(tile) * kTileElems + x->col)) + x->s);
  return true;
}
// The neighbour's trace there: weights cm of its side nodes, loaded by ld.
template <int P, typename Load>
__device__ __forceinline__ void far_trace(const double2* v, const FarFace& x, const double* cm, double* um, Load&& ld) {
  um[0] = um[1] = um[2] = um[3] = 0.0;
#pragma unroll
  for (int k = 0; k <= P; ++k) {
    const int node = x.s == 0 ? edge_node(P, 0, k) : (x.s == 1 ? edge_node(P, 1, k) : edge_node(P, 2, k));
    const double2* src = v + state_index(np_of_p(P), x.nb, 2 * node);
    const double2 n0 = ld(src), n1 = ld(src + kTileRun);
    um[0] = fma(cm[k], n0.x, um[0]);
    um[1] = fma(cm[k], n0.y, um[1]);
    um[2] = fma(cm[k], n1.x, um[2]);
    um[3] = fma(cm[k], n1.y, um[3]);
  }
}

template <int P, int NFQ, int MAP>
struct OpsOfMap {
  using type = StageOps<P, NFQ>;
};
template <int P, int NFQ>
struct OpsOfMap<P, NFQ, kMapFolded> {
  using type = FoldedOps<P, NFQ>;
};
template <int P, int NFQ, int MAP>
using OpsOf = typename OpsOfMap<P, NFQ, MAP>::type;

template <int P, int NFQ, int MAP, bool FAR>
// Three 256-thread blocks per SM (<= 80 registers per thread) keep 24 warps
// resident alongside 3 x ~75 KB of shared memory.
__global__ void __launch_bounds__(4 * kTileElems, 3) tile_stage_kernel(const __grid_constant__ StageArgs a,
                                                                        const OpsOf<P, NFQ, MAP> ops) {
  using L = TileLayout<P, NFQ>;
  constexpr int E = L::E;
  constexpr int NP = L::NP;
  constexpr int NE = L::NE;
  constexpr int T = 4 * E;
  constexpr bool FOLD = MAP == kMapFolded;
  extern __shared__ __align__(128) unsigned char smem[];
  double2* S = reinterpret_cast<double2*>(smem + L::kS);
  double2* H = reinterpret_cast<double2*>(smem + L::kH);
  double* FB = reinterpret_cast<double*>(smem + L::kFB);
  double2* FB2 = reinterpret_cast<double2*>(smem + L::kFB);
  double2* GE = reinterpret_cast<double2*>(smem + L::kGE);
  double* TM = reinterpret_cast<double*>(smem + L::kTM);
  int* EL = reinterpret_cast<int*>(smem + L::kEL);
  const unsigned short* items = reinterpret_cast<const unsigned short*>(smem + L::kItems);
  const FaceCounts* counts = reinterpret_cast<const FaceCounts*>(smem + L::kItems + kListCount);
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + L::kBar);
  int* abort_flag = reinterpret_cast<int*>(smem + L::kBar + 8);
  int* NEXT = reinterpret_cast<int*>(smem + L::kBar + 12);

  const int t = threadIdx.x;
  const int lane = t & 31;
  const int which = (t >> 5) & 1;                 // this warp's half of the tile
  const int grp = t >> 6;                         // and its number among the half's four
  const int col = t % E;                          // load and nodal flux phases
  const int el = work_column(t), c = work_component(t);
  const int G = gridDim.x;
  const bool hand_out = a.ntiles > kHandOut * G;
  const unsigned max_tries = a.wait_tries ? a.wait_tries : kMaxWaitTries;

  {
    const double* tm = &ops.tm[0][0][0];
    for (int l = t; l < 3 * NFQ * NE; l += T) TM[l] = tm[l];
  }
  if (t == 0) {
    mbar_init(bar, 2);
    *abort_flag = 0;
  }

  int tile = blockIdx.x;  // the grid has at most ntiles blocks
  unsigned code = neighbour_code(a.lists, tile, which, lane);
  __syncthreads();
  if (grp == 0 && lane == 0) issue_mesh_copies<P, NFQ>(a, tile, which, smem);
  wait_for_previous();
  let_next_start();
  if (grp == 0 && lane == 0) issue_state_copy<P, NFQ>(a.in, tile, which, smem, a.test_flags);
  copy_neighbours<P>(H, a.in, code, which, grp, lane);
  cp_async_commit();
  unsigned parity = 0;

  while (true) {
    const long long blk = 2ll * tile + which;  // this half's block
    unsigned taken = 0;
    if (t == 224 && hand_out) taken = take_tile(a.err + 4);

    // ---- 1. load ------------------------------------------------------------------
    // this half's RK operand block (read in phase 6) into L2. The next tile's
    // state is not prefetched: its bulk copies, issued in phase 5, read it from
    // HBM themselves (prefetching it as well was 1.6% slower)
    if (!a.elem && grp == 3) {
      Numbering n;
      n.K = a.K;
      EL[col] = n.element(tile * E + col);
    }
    if (grp == 2 && lane == 0 && a.stage >= 1 && a.stage <= 3)
      bulk_prefetch_l2((a.stage == 3 ? a.acc : a.base) + blk * (2 * NP * kTileRun), 2 * NP * kTileRun * 16);
    {
      bool ok = false;
      for (unsigned n = 0; n < max_tries && !ok; ++n) ok = mbar_try_wait(bar, parity);
      if (!ok) {
        atomicOr(&a.err[3], 2ull);
        *abort_flag = 1;
      }
    }
    parity ^= 1u;

    // ---- 2. own traces at every face point -------------------------------------------
    own_traces<P, NFQ>(ops, S, FB, el, c);
    cp_async_wait_all();  // this thread's copies of neighbour rows
    __syncthreads();
    if (*abort_flag) break;

    // ---- 3. faces: the (doubled) flux overwrites the traces it consumed ------------------
    const FaceCounts faces = *counts;
    int entry, q, q1;
    for (int w = t; face_work<NFQ>(faces, w, &entry, &q, &q1); w += T) {
      const int it = items[entry];
      const int fl = it & 63, s = (it >> 6) & 3, x = it >> 9;
      const bool mirror = (it >> 8) & 1;
      const double2 n = GE[((fl >> 5) * kGeoRows + 4 + s) * kTileRun + (fl & 31)];
      double2* own = FB2 + (s * NFQ + q) * 2 * E + fl;
      double2* oth = FB2 + (s * NFQ + NFQ - 1 - q) * 2 * E + (mirror ? x : 0);
#pragma unroll 1
      for (; q < q1; ++q, own += 2 * E, oth -= 2 * E) {
        const double2 x0 = own[0], x1 = own[E];
        const double up[4] = {x0.x, x0.y, x1.x, x1.y};
        double um[4];
        if (mirror) {
          const double2 y0 = oth[0], y1 = oth[E];
          um[0] = y0.x, um[1] = y0.y, um[2] = y1.x, um[3] = y1.y;
        } else {
          um[0] = um[1] = um[2] = um[3] = 0.0;
          const double* cm = TM + (s * NFQ + q) * NE;
          // one node at a time: with all 2 NE loads in flight, which take the
          // flux's registers, 5 RK4 steps at 768 x 768, p = 3 took 6.78 ms (6.68),
          // 20 at 384 x 384, p = 1 4.12 (4.04)
#pragma unroll 1
          for (int k = 0; k < NE; ++k) {
            const double2 n0 = H[2 * k * 2 * kSlots + x], n1 = H[(2 * k + 1) * 2 * kSlots + x];
            um[0] = fma(cm[k], n0.x, um[0]);
            um[1] = fma(cm[k], n0.y, um[1]);
            um[2] = fma(cm[k], n1.x, um[2]);
            um[3] = fma(cm[k], n1.y, um[3]);
          }
        }
        double f[4];
        roe_flux2(up, um, n.x, n.y, f, [&](int err) { record_error(a, NFQ, EL[fl], q, s, err); });
        own[0] = make_double2(f[0], f[1]);
        own[E] = make_double2(f[2], f[3]);
        if (mirror) {
          oth[0] = make_double2(-f[0], -f[1]);
          oth[E] = make_double2(-f[2], -f[3]);
        }
      }
    }
    if constexpr (FAR) {
      FarFace x;
      for (int w = t; far_face<NFQ>(faces, items, a.nbr, tile, w, &x); w += T) {
        const double2 n = GE[((x.col >> 5) * kGeoRows + 4 + x.s) * kTileRun + (x.col & 31)];
        double2* own = FB2 + (x.s * NFQ + x.q) * 2 * E + x.col;
        const double2 x0 = own[0], x1 = own[E];
        const double up[4] = {x0.x, x0.y, x1.x, x1.y};
        double um[4], f[4];
        far_trace<P>(a.in, x, TM + (x.s * NFQ + x.q) * NE, um, [](const double2* p) { return *p; });
        roe_flux2(up, um, n.x, n.y, f, [&](int err) { record_error(a, NFQ, EL[x.col], x.q, x.s, err); });
        own[0] = make_double2(f[0], f[1]);
        own[E] = make_double2(f[2], f[3]);
      }
    }
    if (t == 224) *NEXT = hand_out ? static_cast<int>(taken) + G : tile + G;
    __syncthreads();
    const int next = *NEXT;
    const bool has_next = next < a.ntiles;

    // the next tile's neighbours: their codes now, their rows after the nodal flux
    code = has_next ? neighbour_code(a.lists, next, which, lane) : kNoNeighbour;

    // ---- 4. lift ---------------------------------------------------------------------------
    const bool valid = EL[el] >= 0;
    double* FBt = FB + ((c >> 1) * E + el) * 2 + (c & 1);  // this thread's component and column
    double r[NP];  // per node, or FOLD: the even parts, then the odd parts, of the node pairs
    {
      const double2* ge = GE + which * kGeoRows * kTileRun + (el & 31);
      lift_term<P, NFQ>(ops, FBt, ge[2 * kTileRun], ge[3 * kTileRun], r);
    }
    // stage 3: U3 / (3 c_out) into the accumulators while the state tile still
    // holds U3 (the update then writes X + c_out (k4 + U3 / (3 c_out)))
    if (a.stage == 3 && valid) {
      const double dtt = a.tile_dt ? __ldg(a.tile_dt + tile) : 1.0;
      const double f = kThird / (a.c_out * dtt);
      if constexpr (FOLD) {
        folded_state<P>(S, el, c, f, r);
      } else {
        const double* Sd = reinterpret_cast<const double*>(S) + sidx<NP>(c >> 1, el) * 2 + (c & 1);
#pragma unroll
        for (int i = 0; i < NP; ++i) r[i] = fma(f, Sd[i * 4 * kTileRun], r[i]);
      }
    }
    run_sync(t);

    // ---- 5. nodal flux of every node, once, contracted with the inverse Jacobian --------
    if (P > 0) {
      const double2* ge = GE + which * kGeoRows * kTileRun + lane;
      const double2 j0 = ge[0], j1 = ge[kTileRun];
      if constexpr (FOLD) folded_nodal_flux<P>(S, FB2, col, grp, j0, j1);
      else plain_nodal_flux<P>(S, FB2, col, grp, j0, j1);
    }
    run_sync(t);

    // this half's state and geometry are free: start its next copies and neighbour rows
    if (has_next) {
      if (grp == 0 && lane == 0) {
        issue_mesh_copies<P, NFQ>(a, next, which, smem);
        issue_state_copy<P, NFQ>(a.in, next, which, smem, a.test_flags);
      }
      copy_neighbours<P>(H, a.in, code, which, grp, lane);
    }
    cp_async_commit();

    // the stage update's first operand, requested now so that it is in flight
    // during the volume phase
    constexpr int kStep = 4 * kTileRun;  // doubles between node rows of the same pair
    const long long off0 = blk * (4 * NP * kTileRun) + (c >> 1) * (2 * kTileRun) + (el & 31) * 2 + (c & 1);
    double pre[NP];
    {
      const bool upd = valid && a.stage != kStageRhs;
      const double* src = reinterpret_cast<const double*>(first_operand(a)) + off0;
#pragma unroll
      for (int i = 0; i < NP; ++i) pre[i] = upd ? ld_early(src + i * kStep) : 0.0;
    }

    // ---- 6a. volume D_xi G_xi + D_eta G_eta --------------------------------------------
    if (P > 0) volume_term<P, NFQ>(ops, FBt, r);
    if constexpr (FOLD) unfold<P>(r);

    // ---- 6b. stage update ------------------------------------------------------------------
    // The outputs are written with streaming stores (st.global.cs, evict
    // first): where the stage is memory-bound its vectors exceed L2, and
    // evicting them first keeps the rows that tiles in flight still read there
    // (neighbour rows, prefetched operand rows); 0.3% faster at 768 x 768, p = 3.
    if (valid) {
      const double dtt = a.tile_dt ? __ldg(a.tile_dt + tile) : 1.0;
      const double c_acc = a.c_acc * dtt, c_out = a.c_out * dtt;
      double* out = reinterpret_cast<double*>(a.out) + off0;
      if (a.stage == 1 && !a.no_acc) {
        // X = (U_n + U1) / 3 + c_acc k2, U1 being this stage's input, re-read
        // here (its tile was copied one tile ago and is still in L2) by loads
        // that stay where they are written (plain loads were hoisted and
        // spilled). Half of the rows at a time: a load that follows a store to
        // another array cannot be moved above it, and all of them before the
        // first store took 0.3% longer at 150 x 90, p = 3
        const double* in = reinterpret_cast<const double*>(a.in) + off0;
        double* acc = reinterpret_cast<double*>(a.acc) + off0;
        constexpr int kHalf = (NP + 1) / 2;
#pragma unroll
        for (int h = 0; h < NP; h += kHalf) {
          double iv[kHalf];
#pragma unroll
          for (int i = h; i < h + kHalf && i < NP; ++i) iv[i - h] = ld_early(in + i * kStep);
#pragma unroll
          for (int i = h; i < h + kHalf && i < NP; ++i)
            __stcs(acc + i * kStep, fma(c_acc, r[i], (pre[i] + iv[i - h]) * kThird));
        }
      }
      if (a.stage != kStageRhs) {
#pragma unroll
        for (int i = 0; i < NP; ++i) __stcs(out + i * kStep, fma(c_out, r[i], pre[i]));
      } else {
#pragma unroll
        for (int i = 0; i < NP; ++i) __stcs(out + i * kStep, r[i]);
      }
    }
    // the four warps of a half work on the same columns: none may start the
    // next tile's traces (which reuse rows of the face / flux buffer) before
    // the others are done with this tile's volume phase
    run_sync(t);
    if (!has_next) break;
    tile = next;
  }

  cp_async_wait_all();  // none may land after the block has left
  if (*abort_flag) {
    // the bulk copies of a tile whose wait gave up may still land: wait for
    // them once more, with the same bound, before the block leaves
    for (unsigned n = 0; n < max_tries; ++n)
      if (mbar_try_wait(bar, parity ^ 1u)) break;
  }
  const bool step_ends = a.stage == 3 || a.stage == kStageEuler;
  if (t == 0 && (step_ends || hand_out)) {
    __threadfence();
    const unsigned long long done = atomicAdd(&a.err[2], 1ull);
    if (done == gridDim.x - 1) {
      a.err[2] = 0ull;
      a.err[4] = 0ull;
      if (step_ends) atomicAdd(&a.err[1], 1ull);
    }
  }
}

}  // namespace vt
