// The solver context behind the opaque vt_ctx handle, shared by the forward
// solver (vt_solver.cu) and the discrete adjoint (vt_adjoint.cu).
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <vector>

#include "../../include/vortex_b200.h"
#include "vt_launch.h"

namespace vt {
struct AdjointState;  // vt_adjoint.cu
}

struct vt_ctx {
  std::mutex mu;
  int device = 0, p = 0, Np = 0, nfq = 0, K = 0;
  vt::Numbering num;
  long long ncols = 0;  // columns: 64 per tile
  int sms = 0, max_blocks = 0;  // persistent grid: SMs x resident blocks per SM
  cudaStream_t stream = nullptr;
  double2 *U = nullptr, *A = nullptr, *Sa = nullptr, *Sb = nullptr, *R = nullptr;
  double2* geo = nullptr;
  int4* nbr = nullptr;
  int* elem = nullptr;              // element of each column
  unsigned char* lists = nullptr;   // per-tile face lists
  bool far = false;                 // a tile has more leaving faces than slots (launch_build_tile_lists)
  int ntiles = 0;
  unsigned long long* err = nullptr;
  double2* aos = nullptr;
  double *W = nullptr, *partial = nullptr, *tot = nullptr;
  std::vector<double> ops;    // operator block (StageOps)
  std::vector<double> block;  // the stage kernel's form of it
  std::vector<double> minv_ref;  // Np x Np, for the projected initial condition
  vt::LaunchFn launch = nullptr;
  // many steps in one launch, for a problem of few tiles (null otherwise): the
  // kernel, the tiles' flags and what they hold (unknown after an error);
  // flag_launches: steps whose outcome finish() has still to see
  decltype(vt::StageKernel::resident) resident = nullptr;
  unsigned* flags = nullptr;
  unsigned flag_base = 0;
  bool flags_known = false, flag_launches = false;
  int counted = 0;  // tiles of steps under way that this context is counted with (take_resident)
  int map = vt::kDefaultMap;  // form of the stage kernel
  double time = 0.0;
  vt_error_info last{};
  int pending_steps = 0;
  double pending_dt = 0.0;
  // asynchronous steps by launches of a graph (enqueue_graphs, vt_solver.cu):
  // the graph, and what its launches were made with
  struct StepsGraph {
    cudaGraphExec_t exec = nullptr;
    double dt = 0.0;
    const double2* U = nullptr;
    int map = 0, flags = 0;
    unsigned tries = 0;
  } steps;
  bool side_pairing = false;  // nbr(nbr(e, s), s) == e for every element and side
  bool mutual_tiles = false;  // a tile that reads another is read by it (implied by side_pairing)
  // Per-tile time steps (a batch group's view; null otherwise): stage and
  // adjoint coefficients are then fractions scaled on the device.
  const double* tile_dt = nullptr;
  // A batch group's view: the numbering of each instance, at its first column,
  // and where its block starts in a caller's array (doubles), when that holds
  // the group's instances in order (`at`) or all instances of the batch in
  // order (`at_all`, used while `all_instances` is set). Else empty: num numbers
  // everything.
  struct Part {
    vt::Numbering num;
    long long column, at, at_all;
  };
  std::vector<Part> parts;
  bool all_instances = false;
  vt::AdjointState* adj = nullptr;
  // vt_test_bulk_wait: the stage kernels' wait bound and test flags
  unsigned test_wait_tries = 0;
  int test_flags = 0;
};

namespace vt {

std::string cuda_msg(const char* what, cudaError_t e);

// The column of every element of a numbering.
std::vector<int> element_columns(const Numbering& num);
// A mesh's geometry rows and side-ordered neighbour columns (StageArgs), its
// columns starting at `column` of the arrays.
void pack_mesh(const vt_mesh_desc& d, const std::vector<int>& col, double2* geo, int4* nbr, long long column);

// Arguments of one stage launch on this context's mesh and schedule.
StageArgs stage_args(vt_ctx* c, const double2* in, const double2* base, double2* acc, double2* out, int stage,
                     double c_acc, double c_out);
// The four stage launches of one RK4 step of U in place (A, Sa, Sb scratch).
cudaError_t enqueue_rk4_step(vt_ctx* c, double dt);
// Clears the first-error key and the step counters.
cudaError_t reset_error_words(vt_ctx* c);
// Builds the tiles' face lists, waits for them and sets c->far.
cudaError_t build_lists(vt_ctx* c);
// Takes the context's stage kernel of form `map` (and, where it may, the
// resident one) into use.
cudaError_t use_kernel(vt_ctx* c, int map);
// Waits for the stream, decodes the first-error key, advances the clock by
// nsteps * dt and returns the status.
int finish(vt_ctx* c, int nsteps, double dt);
// Device AoS staging buffer (K x Np x 4 doubles), allocated on first use.
int ensure_aos(vt_ctx* c);
// AoS (K x Np x 4, device memory) <-> the columns of a state vector.
cudaError_t to_columns(vt_ctx* c, const double* src, double2* dst);
cudaError_t from_columns(vt_ctx* c, const double2* src, double* dst);

// The context's steps are no longer under way (take_resident, vt_solver.cu).
void steps_are_done(vt_ctx* c);

// Frees the adjoint's buffers (no-op without them).
void adjoint_release(vt_ctx* c);

}  // namespace vt
