// gbdx_mlp_bwd_d32h64.cu -- MLP-field backward instantiations for state dim 32,
// hidden width 64.
#include "gbdx_mlp_bwd_impl.cuh"

namespace gbdx {
BwdEntry find_mlp_bwd_entry_d32h64(int solver, bool sde) {
  return mlp_bwd_entry<32, 64, true>(solver, sde);
}
}  // namespace gbdx
