// Many steps of a small problem in one launch.
//
// A problem with at most one tile per SM leaves the stage kernel with nothing
// to overlap: at 8 x 8 cells, p = 3 (two tiles) a stage took 6.2 us, of which
// the tile's own work is 4 and the rest the end of one launch, the start of the
// next and the tile's way to HBM and back. Here every block keeps its tile for
// all the steps of a call: state, geometry and face list stay in shared memory,
// U_n and the RK accumulator in registers, and a tile waits only for the tiles
// it shares a face with. Alone on its SM a tile is bound by latency, so with
// the folded operators it has two threads per element and component, one for
// the even and one for the odd parts, and twice the threads for the faces:
//
//                                    stage kernel  256 threads  512 threads
//   250 RK4 steps,  8 x 8,   p = 3       6.2 ms       4.7 ms      4.15 ms
//   50 RK4 steps,   64 x 64, p = 2       1.12         0.97        0.86
//   100 Euler steps, 27 x 18, p = 1      0.51         0.42        0.37
//
// (3.96, 0.826 and 0.351 since the loop for faces without a slot has kernels of
// its own.)
// (768 threads, which leave 80 registers each: 4.43, 0.93 and 0.40 ms.) What is
// left of a stage at 8 x 8, p = 3, in cycles of 7900: lift and volume, with the
// wait for the slowest faces, 2300, faces 2000, waiting for the neighbours and
// copying their nodes 1300, the rest 2300. The numbers are the stage kernel's,
// bit for bit: the same functions in the same order (vt_tile.cuh).
//
// Stage s of a launch (counted over its steps):
//   1. one warp of each half waits until the neighbours' tiles have published s
//      stages (flags, below);
//   2. meanwhile the nodal flux into a buffer of its own; then the neighbours'
//      side nodes are requested (cp.async) and the own traces formed;
//   3. barrier; faces; barrier;
//   4. lift, volume, update: the new stage state goes to shared memory and to
//      the stage's vector in HBM, where the neighbours find it;
//   5. barrier; one thread makes the block's writes visible and publishes.
// A vector that a tile overwrites in stage s was last read by its neighbours in
// a stage before s, and they have published that stage before this tile passes
// its own wait of stage s; so two stage vectors and U are enough. That needs
// every tile that reads this one to be one that it waits for, that is, reads
// itself: use_resident (vt_solver.cu) takes the kernel for such meshes only.
//
// All blocks are resident at once (a cooperative launch). Every wait is bounded;
// one that gives up sets bit 1 of err[3], the block leaves, and the others give
// up in turn.
#pragma once

#include <type_traits>

#include "vt_tile.cuh"

namespace vt {

struct ResidentArgs {
  double2 *U, *Sa, *Sb;
  unsigned* flags;  // per tile: stages published, modulo 2^32
  unsigned flag0;   // what they hold when the launch starts
  int nsteps;
  unsigned long long step0;  // steps of the call done before this launch (error reports)
  double dt;
  int euler;  // forward Euler instead of RK4
};

// The stage kernel's buffers, with the nodal flux apart from the face buffer.
template <int P, int NFQ>
struct ResidentLayout {
  using B = TileLayout<P, NFQ>;
  static constexpr int kG = (B::kBytes + 127) / 128 * 128;  // double2 [NP][4][E]
  static constexpr int kBytes = kG + 4 * B::NP * kTileElems * 16;
};

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr unsigned kMaxFlagTries = 1u << 20;

// A flag per tile, each in a line of its own: with all of them in a few lines,
// and every thread that copies a neighbour's rows polling, the polls of 128
// blocks queued at those lines (a stage at 64 x 64 cells, p = 2 took 7.7 us).
constexpr int kFlagStride = 32;

// false when the tile has not published `target` stages within the bound.
__device__ __forceinline__ bool wait_for_tile(const unsigned* flags, int tile, unsigned target, unsigned tries) {
  for (unsigned n = 0; n < tries; ++n)
    if (static_cast<int>(load_acquire(flags + tile * kFlagStride) - target) >= 0) return true;
  return false;
}

// N points of one face, from point q on (`own`, `oth`: its rows of this and the
// partner's column): all traces, then all fluxes, then all results.
template <int P, int NFQ, int N, typename Outer, typename OnError>
__device__ __forceinline__ void face_points(double2* own, double2* oth, bool mirror, double2 n, int q, Outer&& outer,
                                            OnError&& on_error) {
  constexpr int E = kTileElems;
  double up[N][4], um[N][4], f[N][4];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double2 x0 = own[2 * k * E], x1 = own[(2 * k + 1) * E];
    up[k][0] = x0.x, up[k][1] = x0.y, up[k][2] = x1.x, up[k][3] = x1.y;
    if (mirror) {
      const double2 y0 = oth[-2 * k * E], y1 = oth[(1 - 2 * k) * E];
      um[k][0] = y0.x, um[k][1] = y0.y, um[k][2] = y1.x, um[k][3] = y1.y;
    }
  }
  if (!mirror) outer(q, um);
  RoeAverages r[N];
  int usual = 1;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    roe_averages(up[k], um[k], n.x, n.y, r[k]);
    usual = min(usual, r[k].usual);
  }
  if (__builtin_expect(usual <= 0, 0)) {
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (r[k].usual <= 0) roe_unusual(up[k], um[k], r[k], [&](int err) { on_error(q + k, err); });
  }
#pragma unroll
  for (int k = 0; k < N; ++k) roe_sum(up[k], um[k], n.x, n.y, r[k], f[k]);
#pragma unroll
  for (int k = 0; k < N; ++k) {
    own[2 * k * E] = make_double2(f[k][0], f[k][1]);
    own[(2 * k + 1) * E] = make_double2(f[k][2], f[k][3]);
    if (mirror) {
      oth[-2 * k * E] = make_double2(-f[k][0], -f[k][1]);
      oth[(1 - 2 * k) * E] = make_double2(-f[k][2], -f[k][3]);
    }
  }
}

// Threads of a block: with the folded operators two per element and component,
// one for the even and one for the odd parts.
constexpr int resident_threads(int map) { return (map == kMapFolded ? 8 : 4) * kTileElems; }

// The even (ODD = 0), the odd (1) or all (-1) parts of the update, and the nodes
// whose new values this thread forms from them: the first ones of the mirrored
// pairs and the fixed nodes, the second ones, or all.
template <int P, int PART>
struct ResidentPart {
  static constexpr int kParts = PART < 0 ? np_of_p(P) : (PART == 0 ? fold_nodes(P) : fold_pairs(P));
  static constexpr int kArray = PART < 0 ? np_of_p(P) : fold_nodes(P);
  __device__ static constexpr int node(int a) {
    return PART < 0 ? a : (PART == 0 ? fold_node(P, a) : mirror_node(P, fold_node(P, a)));
  }
};

// Barrier of the THREADS threads that hold one half's columns.
template <int THREADS>
__device__ __forceinline__ void half_sync(int which) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + which), "n"(THREADS) : "memory");
}
// Barrier of the two warps with the same elements and components.
__device__ __forceinline__ void pair_sync(int t) {
  asm volatile("bar.sync %0, 64;" ::"r"(3 + ((t >> 5) & 7)) : "memory");
}

template <int P, int NFQ, int MAP, bool FAR>
__global__ void __launch_bounds__(resident_threads(MAP), 1)
    resident_steps_kernel(const __grid_constant__ StageArgs a, const __grid_constant__ ResidentArgs ra,
                          const OpsOf<P, NFQ, MAP> ops) {
  using L = TileLayout<P, NFQ>;
  constexpr int E = L::E;
  constexpr int NP = L::NP;
  constexpr int NE = L::NE;
  constexpr int T = resident_threads(MAP);
  constexpr int G = T / E;  // groups of a thread per column
  constexpr bool FOLD = MAP == kMapFolded;
  extern __shared__ __align__(128) unsigned char smem[];
  double2* S = reinterpret_cast<double2*>(smem + L::kS);
  double2* H = reinterpret_cast<double2*>(smem + L::kH);
  double* FB = reinterpret_cast<double*>(smem + L::kFB);
  double2* FB2 = reinterpret_cast<double2*>(smem + L::kFB);
  double* GB = reinterpret_cast<double*>(smem + ResidentLayout<P, NFQ>::kG);
  double2* GB2 = reinterpret_cast<double2*>(smem + ResidentLayout<P, NFQ>::kG);
  double2* GE = reinterpret_cast<double2*>(smem + L::kGE);
  double* TM = reinterpret_cast<double*>(smem + L::kTM);
  const int* EL = reinterpret_cast<const int*>(smem + L::kEL);
  const unsigned short* items = reinterpret_cast<const unsigned short*>(smem + L::kItems);
  FaceCounts* counts = reinterpret_cast<FaceCounts*>(smem + L::kItems + kListCount);
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + L::kBar);
  // abort_flag is set only between a stage's start and its first barrier, and
  // read by all behind that barrier, so that all leave together; late_flag is
  // what the face phase sets, for the next stage
  int* abort_flag = reinterpret_cast<int*>(smem + L::kBar + 8);
  int* late_flag = reinterpret_cast<int*>(smem + L::kBar + 12);

  const int t = threadIdx.x;
  const int lane = t & 31;
  const int which = (t >> 5) & 1;  // this warp's half of the tile
  const int grp = t >> 6;          // and its number among the half's G
  const int col = t % E;           // nodal flux phase
  const int el = work_column(t % (4 * E)), c = work_component(t % (4 * E));
  const int tile = blockIdx.x;
  const long long blk = 2ll * tile + which;
  const unsigned max_tries = a.wait_tries ? a.wait_tries : kMaxWaitTries;
  const unsigned flag_tries = a.wait_tries ? a.wait_tries : kMaxFlagTries;

  {
    const double* tm = &ops.tm[0][0][0];
    for (int l = t; l < 3 * NFQ * NE; l += T) TM[l] = tm[l];
  }
  __shared__ unsigned least;
  if (t == 0) {
    mbar_init(bar, 2);
    *abort_flag = *late_flag = 0;
    least = ~0u;
  }
  const unsigned code = neighbour_code(a.lists, tile, which, lane);
  __syncthreads();
  if (grp == 0 && lane == 0) {
    issue_mesh_copies<P, NFQ>(a, tile, which, smem);
    issue_state_copy<P, NFQ>(ra.U, tile, which, smem, a.test_flags);
  }
  {
    bool ok = false;
    for (unsigned n = 0; n < max_tries && !ok; ++n) ok = mbar_try_wait(bar, 0);
    if (!ok) {
      atomicOr(&a.err[3], 2ull);
      *abort_flag = 1;
    }
  }
  if constexpr (T != 4 * E) {  // points per work item for this number of threads
    const int n0 = counts->n & 0xff, n1 = (counts->n >> 8) & 0xff, i = 1 + t / NFQ, j = 1 + t % NFQ;
    if (t < NFQ * NFQ) atomicMin(&least, static_cast<unsigned>(face_cost(n0, n1, NFQ, i, j, T) << 8 | (NFQ * NFQ - 1 - t)));
    __syncthreads();
    if (t == 0) {
      const int best = NFQ * NFQ - 1 - (least & 0xff);
      *counts = face_counts(n0, n1, counts->n >> 16, NFQ, 1 + best / NFQ, 1 + best % NFQ);
    }
  }
  __syncthreads();

  // a lane polls for its slot's tile unless the slot before it has the same one
  const unsigned before = __shfl_up_sync(0xffffffffu, code, 1);
  const bool polls = grp == G - 1 && code != kNoNeighbour &&
                     (lane == 0 || (before >> 2) / kTileElems != (code >> 2) / kTileElems);

  constexpr int kStep = 4 * kTileRun;  // doubles between node rows of the same pair
  const long long off0 = blk * (4 * NP * kTileRun) + (c >> 1) * (2 * kTileRun) + (el & 31) * 2 + (c & 1);
  double* Sd = reinterpret_cast<double*>(S) + sidx<NP>(c >> 1, el) * 2 + (c & 1);  // this thread's cells of the state
  const int at = ((c >> 1) * E + el) * 2 + (c & 1);  // its component and column in the face and flux buffers
  const int nstages = ra.euler ? ra.nsteps : 4 * ra.nsteps;
  constexpr int kOwn = FOLD ? fold_nodes(P) : NP;
  double base[kOwn], X[kOwn];
#pragma unroll
  for (int i = 0; i < kOwn; ++i) base[i] = X[i] = 0.0;

  for (int s = 0; s < nstages; ++s) {
    const int stage = ra.euler ? static_cast<int>(kStageEuler) : s & 3;
    // where this stage reads its neighbours and writes its result
    const double2* in = ra.euler ? (s & 1 ? ra.Sa : ra.U) : (stage == 0 ? ra.U : (stage == 2 ? ra.Sb : ra.Sa));
    double2* out2 = ra.euler ? (s & 1 ? ra.U : ra.Sa) : (stage == 3 ? ra.U : (stage == 1 ? ra.Sb : ra.Sa));
    const unsigned long long epoch = ra.euler ? (ra.step0 + s) * 4ull : (ra.step0 + (s >> 2)) * 4ull + stage;

    // ---- 1. the neighbours' tiles, one warp of each half ---------------------------
    if (polls && !wait_for_tile(ra.flags, static_cast<int>((code >> 2) / kTileElems), ra.flag0 + s, flag_tries)) {
      atomicOr(&a.err[3], 2ull);
      *abort_flag = 1;
    }
    if (FAR && t == 0 && *late_flag) *abort_flag = 1;

    // ---- 2. nodal flux; the neighbours' side nodes; own traces ----------------------
    if (P > 0) {
      const double2* ge = GE + which * kGeoRows * kTileRun + lane;
      const double2 j0 = ge[0], j1 = ge[kTileRun];
      if constexpr (FOLD) folded_nodal_flux<P, G>(S, GB2, col, grp, j0, j1);
      else plain_nodal_flux<P>(S, GB2, col, grp, j0, j1);
    }
    half_sync<T / 2>(which);  // the half's neighbours have published
    copy_neighbours<P>(H, in, code, which, G - 1 - grp, lane);
    if constexpr (FOLD) {
      if (t < 4 * E) own_traces<P, NFQ, 0, 3 * NFQ / 2>(ops, S, FB, el, c);
      else own_traces<P, NFQ, 3 * NFQ / 2, 3 * NFQ>(ops, S, FB, el, c);
    } else {
      own_traces<P, NFQ>(ops, S, FB, el, c);
    }
    cp_async_wait_all();
    __syncthreads();
    if (*abort_flag) break;

    // ---- 3. faces ------------------------------------------------------------------
    // Points side by side, to hide each other's latency where there are the
    // registers: 512 threads have them for one (two: 5.2 ms at 8 x 8, spilling).
    constexpr int kSide = FOLD || NFQ < 3 ? 1 : 3;
    const FaceCounts faces = *counts;
    int entry, q, q1;
    for (int w = t; face_work<NFQ>(faces, w, &entry, &q, &q1); w += T) {
      const int it = items[entry];
      const int fl = it & 63, sd = (it >> 6) & 3, x = it >> 9;
      const bool mirror = (it >> 8) & 1;
      const double2 n = GE[((fl >> 5) * kGeoRows + 4 + sd) * kTileRun + (fl & 31)];
      double2* own = FB2 + (sd * NFQ + q) * 2 * E + fl;
      double2* oth = FB2 + (sd * NFQ + NFQ - 1 - q) * 2 * E + (mirror ? x : 0);
      auto outer = [&](int q0, auto& um) {
        constexpr int N = sizeof(um) / sizeof(um[0]);
#pragma unroll
        for (int k = 0; k < N; ++k) um[k][0] = um[k][1] = um[k][2] = um[k][3] = 0.0;
        const double* cm = TM + (sd * NFQ + q0) * NE;
#pragma unroll
        for (int j = 0; j < NE; ++j) {
          const double2 n0 = H[2 * j * 2 * kSlots + x], n1 = H[(2 * j + 1) * 2 * kSlots + x];
#pragma unroll
          for (int k = 0; k < N; ++k) {
            um[k][0] = fma(cm[k * NE + j], n0.x, um[k][0]);
            um[k][1] = fma(cm[k * NE + j], n0.y, um[k][1]);
            um[k][2] = fma(cm[k * NE + j], n1.x, um[k][2]);
            um[k][3] = fma(cm[k * NE + j], n1.y, um[k][3]);
          }
        }
      };
      auto on_error = [&](int point, int err) { record_error_at(a.err, epoch, NFQ, EL[fl], point, sd, err); };
      while (q < q1) {
        const int done = q1 - q >= kSide ? kSide : 1;
        if (done == kSide) face_points<P, NFQ, kSide>(own, oth, mirror, n, q, outer, on_error);
        else face_points<P, NFQ, 1>(own, oth, mirror, n, q, outer, on_error);
        q += done;
        own += done * 2 * E;
        oth -= done * 2 * E;
      }
    }
    if constexpr (FAR) {
      FarFace x;
      for (int w = t; far_face<NFQ>(faces, items, a.nbr, tile, w, &x); w += T) {
        if (!wait_for_tile(ra.flags, x.nb / kTileElems, ra.flag0 + s, flag_tries)) {
          atomicOr(&a.err[3], 2ull);
          *late_flag = 1;
        }
        const double2 n = GE[((x.col >> 5) * kGeoRows + 4 + x.s) * kTileRun + (x.col & 31)];
        face_points<P, NFQ, 1>(FB2 + (x.s * NFQ + x.q) * 2 * E + x.col, nullptr, false, n, x.q,
                               [&](int q0, auto& um) {
                                 far_trace<P>(in, x, TM + (x.s * NFQ + q0) * NE, um[0],
                                              [](const double2* p) { return __ldcg(p); });
                               },
                               [&](int point, int err) {
                                 record_error_at(a.err, epoch, NFQ, EL[x.col], point, x.s, err);
                               });
      }
    }
    __syncthreads();

    // ---- 4. lift, volume, update ---------------------------------------------------
    auto update = [&](auto part) {
      constexpr int PART = decltype(part)::value;
      using R = ResidentPart<P, PART>;
      double r[R::kArray], u[R::kArray];
      {
        const double2* ge = GE + which * kGeoRows * kTileRun + (el & 31);
        if constexpr (PART < 0) lift_term<P, NFQ>(ops, FB + at, ge[2 * kTileRun], ge[3 * kTileRun], r);
        else lift_term<P, NFQ, PART == 0, PART == 1>(ops, FB + at, ge[2 * kTileRun], ge[3 * kTileRun], r);
      }
#pragma unroll
      for (int i = 0; i < R::kParts; ++i) u[i] = Sd[R::node(i) * kStep];  // the stage's input
      const double c_out = (stage == 0 || stage == 1 ? 0.5 : (stage == 3 ? 1.0 / 6 : 1.0)) * ra.dt;
      if (stage == 3) {
        const double f = kThird / c_out;
        if constexpr (PART < 0) {
#pragma unroll
          for (int i = 0; i < NP; ++i) r[i] = fma(f, u[i], r[i]);
        } else {
          folded_state<P, PART == 0, PART == 1>(S, el, c, f, r);
        }
      }
      if constexpr (PART < 0) {
        if (P > 0) volume_term<P, NFQ>(ops, GB + at, r);
      } else {
        if (P > 0) volume_term<P, NFQ, PART == 0, PART == 1>(ops, GB + at, r);
        // the other thread's parts, through the flux rows that only this thread has read
        double* G = GB + at;
        constexpr int NO = fold_pairs(P);
#pragma unroll
        for (int a = 0; a < NO; ++a) G[(a * 8 + 4 * PART) * E] = r[a];
        pair_sync(t);
#pragma unroll
        for (int a = 0; a < NO; ++a) {
          const double o = G[(a * 8 + 4 - 4 * PART) * E];
          r[a] = PART == 0 ? r[a] + o : o - r[a];
        }
      }
      if (stage == 0 || stage == kStageEuler) {
#pragma unroll
        for (int i = 0; i < R::kParts; ++i) base[i] = u[i];
      }
      if (stage == 1) {
        const double c_acc = (1.0 / 3) * ra.dt;
#pragma unroll
        for (int i = 0; i < R::kParts; ++i) X[i] = fma(c_acc, r[i], (base[i] + u[i]) * kThird);
      }
      if (EL[el] >= 0) {
        double* out = reinterpret_cast<double*>(out2) + off0;
#pragma unroll
        for (int i = 0; i < R::kParts; ++i) {
          const double v = fma(c_out, r[i], stage == 3 ? X[i] : base[i]);
          Sd[R::node(i) * kStep] = v;
          out[R::node(i) * kStep] = v;
        }
      }
    };
    if constexpr (FOLD) {
      if (t < 4 * E) update(std::integral_constant<int, 0>{});
      else update(std::integral_constant<int, 1>{});
    } else {
      update(std::integral_constant<int, -1>{});
    }

    // ---- 5. publish ----------------------------------------------------------------
    __syncthreads();
    if (t == 0) {  // a release at GPU scope, of all the block's writes behind the barrier
      store_release(ra.flags + tile * kFlagStride, ra.flag0 + s + 1);
    }
  }
  cp_async_wait_all();  // none may land after the block has left
  if (*abort_flag) {
    // the bulk copies of a wait that gave up may still land: wait for them once
    // more, with the same bound, before the block leaves
    for (unsigned n = 0; n < max_tries; ++n)
      if (mbar_try_wait(bar, 0)) break;
  }
}

}  // namespace vt
