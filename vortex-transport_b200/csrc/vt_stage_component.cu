// The stage kernel instantiations with the operators as they are (vt_tile.cuh).
#include "vt_stage_inst.cuh"

namespace vt {
StageKernel select_kernel_component(int p, int nfq) { return stage_inst::select_for_map<kMapComponent, false>(p, nfq); }
}  // namespace vt
