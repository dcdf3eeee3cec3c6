// gbdx_mlp_fm_d32h64.cu -- feature-major MLP integrator instantiations for state
// dim 32, hidden width 64.
#include "gbdx_mlp_fm.cuh"

namespace gbdx {
OdeEntry find_mlp_fm_entry_d32h64(int solver) { return fm_entry<32, 64, false>(solver); }
}  // namespace gbdx
