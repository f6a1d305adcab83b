// Launch and configuration of the tiled stage kernel for one form of the operators,
// and one form of the face phase, instantiated for p = 0..3 and nfq = 1..10 by
// vt_stage_component.cu, vt_stage_folded.cu, vt_stage_component_far.cu and
// vt_stage_folded_far.cu (compiled in parallel).
#pragma once

#include <cstring>

#include "vt_jvp_tile.cuh"
#include "vt_launch.h"
#include "vt_resident.cuh"
#include "vt_tile.cuh"

namespace vt {
namespace stage_inst {

template <int P, int NFQ, int MAP, bool FAR>
cudaError_t configure_stage(int* blocks_per_sm) {
  using Lay = TileLayout<P, NFQ>;
  cudaError_t e = cudaFuncSetAttribute(tile_stage_kernel<P, NFQ, MAP, FAR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       Lay::kBytes);
  if (e) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, tile_stage_kernel<P, NFQ, MAP, FAR>,
                                                       4 * kTileElems, Lay::kBytes);
}

template <int P, int NFQ, int MAP>
void pack_operators(const double* ops, double* block) {
  using Ops = OpsOf<P, NFQ, MAP>;
  static_assert(sizeof(Ops) % sizeof(double) == 0 && sizeof(Ops) <= sizeof(StageOps<P, NFQ>) + kBlockExtra * sizeof(double),
                "a block of doubles");
  if constexpr (MAP == kMapFolded) {
    Ops o;
    fold_operators(*reinterpret_cast<const StageOps<P, NFQ>*>(ops), &o);
    std::memcpy(block, &o, sizeof(o));
  } else {
    std::memcpy(block, ops, sizeof(Ops));
  }
}

// Persistent launch: at most `max_blocks` blocks (SMs x resident blocks) over
// all tiles (take_tile, vt_tile.cuh).
template <int P, int NFQ, int MAP, bool FAR>
cudaError_t launch_stage(const StageArgs& a, const double* block, int max_blocks, cudaStream_t st) {
  using Lay = TileLayout<P, NFQ>;
  const int grid = a.ntiles < max_blocks ? a.ntiles : max_blocks;
  return launch_dependent(tile_stage_kernel<P, NFQ, MAP, FAR>, grid, 4 * kTileElems, Lay::kBytes, st, a,
                          *reinterpret_cast<const OpsOf<P, NFQ, MAP>*>(block));
}

template <int P, int NFQ, int MAP, bool FAR>
cudaError_t configure_resident(int* blocks_per_sm) {
  constexpr int bytes = ResidentLayout<P, NFQ>::kBytes;
  *blocks_per_sm = 0;
  if (bytes > 227 * 1024) return cudaSuccess;  // more than a block may have
  const cudaError_t e = cudaFuncSetAttribute(resident_steps_kernel<P, NFQ, MAP, FAR>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, resident_steps_kernel<P, NFQ, MAP, FAR>,
                                                       resident_threads(MAP), bytes);
}

template <int P, int NFQ, int MAP, bool FAR>
cudaError_t launch_resident(const StageArgs& a, const ResidentArgs& r, const double* block, cudaStream_t st) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(a.ntiles));
  cfg.blockDim = dim3(resident_threads(MAP));
  cfg.dynamicSmemBytes = ResidentLayout<P, NFQ>::kBytes;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, resident_steps_kernel<P, NFQ, MAP, FAR>, a, r,
                            *reinterpret_cast<const OpsOf<P, NFQ, MAP>*>(block));
}

template <int P, int NFQ, int MAP, bool FAR>
cudaError_t configure_jvp(int* blocks_per_sm) {
  constexpr int bytes = JvpLayout<P, NFQ>::kBytes;
  static_assert(bytes <= 227 * 1024, "one block per SM");
  const cudaError_t e = cudaFuncSetAttribute(jvp_tile_kernel<P, NFQ, MAP, FAR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             bytes);
  if (e) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, jvp_tile_kernel<P, NFQ, MAP, FAR>, 4 * kTileElems,
                                                       bytes);
}

template <int P, int NFQ, int MAP, bool FAR>
cudaError_t launch_jvp(const StageArgs& a, const JvpArgs& j, const double* block, int max_blocks, cudaStream_t st) {
  const int grid = a.ntiles < max_blocks ? a.ntiles : max_blocks;
  return launch_dependent(jvp_tile_kernel<P, NFQ, MAP, FAR>, grid, 4 * kTileElems, JvpLayout<P, NFQ>::kBytes, st, a, j,
                          *reinterpret_cast<const OpsOf<P, NFQ, MAP>*>(block));
}

template <int P, int NFQ, int MAP, bool FAR>
StageKernel kernel_of() {
  return StageKernel{launch_stage<P, NFQ, MAP, FAR>, pack_operators<P, NFQ, MAP>, configure_stage<P, NFQ, MAP, FAR>,
                     launch_resident<P, NFQ, MAP, FAR>, configure_resident<P, NFQ, MAP, FAR>,
                     launch_jvp<P, NFQ, MAP, FAR>, configure_jvp<P, NFQ, MAP, FAR>};
}

template <int P, int MAP, bool FAR>
StageKernel kernel_for_nfq(int nfq) {
  switch (nfq) {
    case 1: return kernel_of<P, 1, MAP, FAR>();
    case 2: return kernel_of<P, 2, MAP, FAR>();
    case 3: return kernel_of<P, 3, MAP, FAR>();
    case 4: return kernel_of<P, 4, MAP, FAR>();
    case 5: return kernel_of<P, 5, MAP, FAR>();
    case 6: return kernel_of<P, 6, MAP, FAR>();
    case 7: return kernel_of<P, 7, MAP, FAR>();
    case 8: return kernel_of<P, 8, MAP, FAR>();
    case 9: return kernel_of<P, 9, MAP, FAR>();
    case 10: return kernel_of<P, 10, MAP, FAR>();
    default: return StageKernel{};
  }
}

template <int MAP, bool FAR>
StageKernel select_for_map(int p, int nfq) {
  switch (p) {
    case 0: return kernel_for_nfq<0, MAP, FAR>(nfq);
    case 1: return kernel_for_nfq<1, MAP, FAR>(nfq);
    case 2: return kernel_for_nfq<2, MAP, FAR>(nfq);
    case 3: return kernel_for_nfq<3, MAP, FAR>(nfq);
    default: return StageKernel{};
  }
}

}  // namespace stage_inst
}  // namespace vt
