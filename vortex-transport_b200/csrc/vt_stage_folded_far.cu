// The stage kernel instantiations of the folded mapping (vt_tile.cuh).
#include "vt_stage_inst.cuh"

namespace vt {
StageKernel select_kernel_folded_far(int p, int nfq) { return stage_inst::select_for_map<kMapFolded, true>(p, nfq); }
}  // namespace vt
