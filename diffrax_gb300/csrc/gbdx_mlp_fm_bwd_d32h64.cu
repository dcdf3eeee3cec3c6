// gbdx_mlp_fm_bwd_d32h64.cu -- feature-major MLP backward instantiations for state
// dim 32, hidden width 64.
#include "gbdx_mlp_fm_bwd.cuh"

namespace gbdx {
BwdEntry find_mlp_fm_bwd_entry_d32h64(int solver, bool sde) {
  return sde ? fm_bwd_entry<32, 64, true>(solver) : fm_bwd_entry<32, 64, false>(solver);
}
}  // namespace gbdx
