// gbdx_mlp_fm_d64h256.cu -- feature-major MLP integrator instantiations for state
// dim 64, hidden width 256.
#include "gbdx_mlp_fm.cuh"

namespace gbdx {
OdeEntry find_mlp_fm_entry_d64h256(int solver) { return fm_entry<64, 256, false>(solver); }
}  // namespace gbdx
