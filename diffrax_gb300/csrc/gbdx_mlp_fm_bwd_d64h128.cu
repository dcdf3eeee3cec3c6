// gbdx_mlp_fm_bwd_d64h128.cu -- feature-major MLP backward instantiations for state
// dim 64, hidden width 128.
#include "gbdx_mlp_fm_bwd.cuh"

namespace gbdx {
BwdEntry find_mlp_fm_bwd_entry_d64h128(int solver) { return fm_bwd_entry<64, 128, false>(solver); }
}  // namespace gbdx
