// Dispatch to the stage kernel instantiation for (p, nfq), and the tile
// schedule builders; one translation unit (vt_launch.cu) instantiates them.
#pragma once

#include <cuda_runtime.h>

#include "vt_device.cuh"

namespace vt {

struct ResidentArgs;  // vt_resident.cuh
struct JvpArgs;       // vt_jvp_tile.cuh

// Launches a kernel that may be scheduled while the stream's previous kernel is
// still running (let_next_start and wait_for_previous, vt_tile.cuh).
template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t st,
                             Args&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

using LaunchFn = cudaError_t (*)(const StageArgs&, const double*, int, cudaStream_t);
using PackFn = void (*)(const double*, double*);
using ConfigFn = cudaError_t (*)(int*);

constexpr int kBlockExtra = 2;

struct StageKernel {
  // Launches one stage with at most `max_blocks` persistent blocks; its second
  // argument is the kernel's own form of the operators, written by `pack`.
  LaunchFn launch = nullptr;
  // Writes that form (at most stage_ops_doubles(p, nfq) + kBlockExtra doubles)
  // from the operator block.
  PackFn pack = nullptr;
  // Sets the dynamic shared-memory attribute on the current device and
  // reports resident blocks per SM. Call before any launch or capture.
  ConfigFn configure = nullptr;
  // The kernel of many steps of a small problem (vt_resident.cuh): launches it
  // for a.ntiles tiles, all resident at once; its configure reports how many
  // fit an SM (0: it cannot run). Same form of the operators.
  cudaError_t (*resident)(const StageArgs&, const ResidentArgs&, const double*, cudaStream_t) = nullptr;
  ConfigFn configure_resident = nullptr;
  // The derivative of a stage along a direction (vt_jvp_tile.cuh), at most
  // `max_blocks` blocks. Same form of the operators.
  cudaError_t (*jvp)(const StageArgs&, const JvpArgs&, const double*, int, cudaStream_t) = nullptr;
  ConfigFn configure_jvp = nullptr;
  // The mapping it was selected for (kMapComponent or kMapDefault).
  int map = 0;
};

// The mapping a context uses unless told otherwise.
constexpr int kDefaultMap = kMapDefault;

// The kernel for the operator block `ops` (stage_ops_doubles(p, nfq) doubles):
// kMapDefault takes the folded form where operators_reflect says so, else the
// same kernel as kMapComponent.
// `far`: a tile of the mesh may have a face without a slot (launch_build_tile_lists
// tells; the kernels for such meshes are right for any, and a little slower).
// Empty (null members) for p outside 0..3, nfq outside 1..10.
StageKernel select_kernel(int p, int nfq, const double* ops, bool far, int map = kDefaultMap);
StageKernel select_kernel_component(int p, int nfq);
StageKernel select_kernel_folded(int p, int nfq);
StageKernel select_kernel_component_far(int p, int nfq);
StageKernel select_kernel_folded_far(int p, int nfq);

// Whether the operator block has the reference triangle's reflection symmetry
// (vt_device.cuh) to 1e-13 of each operator's largest entry, a few roundings
// of the tables it is folded from. The tables of the reference do (at most
// 1e-14 apart wherever the area rule makes the mass matrix regular); a caller's own tables
// need not.
bool operators_reflect(int p, int nfq, const double* ops);

// Number of doubles of the StageOps<P, NFQ> block for (p, nfq).
int stage_ops_doubles(int p, int nfq);

// Writes the StageOps<P, NFQ> block (stage_ops_doubles(p, nfq) doubles) into
// `ops`: M_ref^-1 folded into the volume operators (D = M_ref^-1 S_xi, S_eta)
// and the lift (M_ref^-1 phi+_s w), with long-double accumulation, and the own /
// neighbour face tables restricted to each side's p + 1 nodes. The inputs are
// the reference-space tables of vt_mesh_desc (Preevolve.cpp:15-144,
// Evolve.cpp:76-132). Host only; allocates nothing.
void fold_stage_operators(int p, int nfq, const double* minv, const double* stiff, const double* line,
                          const double* phi_plus, const double* phi_minus, double* ops);

// Column numberings (vt_device.cuh): of a mesh (the reference's structured
// mesh is recognised by its connectivity), of the reference's mesh of nx x ny
// cells, and without knowledge of the mesh.
Numbering number_mesh(int K, const int32_t* type, const int32_t* conn);
Numbering number_grid(int nx, int ny);
Numbering number_contiguous(int K);

// elem[x0 + x] = e0 + element of the numbering's column x (-1: empty).
cudaError_t launch_number_columns(const Numbering& num, int* elem, int x0, int e0, cudaStream_t st);
// The tiles' face lists (kTileListBytes each, 16-byte aligned) from the columns'
// neighbours and elements (elem null: contiguous numbering of K elements). Bit 0
// of `far` (when given) is set if a tile has more leaving faces than slots.
cudaError_t launch_build_tile_lists(const int4* nbr, const int* elem, int K, int ntiles, int nfq, unsigned char* lists,
                                    unsigned long long* far, cudaStream_t st);
// The callers' layout (K x Np x 4 doubles, 16-byte aligned) <-> a state vector's columns.
cudaError_t launch_to_columns(const double* aos, double2* columns, const Numbering& num, int Np, cudaStream_t st);
cudaError_t launch_from_columns(const double2* columns, double* aos, const Numbering& num, int Np, cudaStream_t st);

}  // namespace vt
