// gbdx_mlp_fm_d64h128.cu -- feature-major MLP integrator instantiations for state
// dim 64, hidden width 128.
#include "gbdx_mlp_fm.cuh"

namespace gbdx {
OdeEntry find_mlp_fm_entry_d64h128(int solver) { return fm_entry<64, 128, false>(solver); }
}  // namespace gbdx
