// gbdx_mlp_bwd_d64h128.cu -- MLP-field backward instantiations for state dim 64,
// hidden width 128.
#include "gbdx_mlp_bwd_impl.cuh"

namespace gbdx {
BwdEntry find_mlp_bwd_entry_d64h128(int solver, bool sde) {
  return mlp_bwd_entry<64, 128, false>(solver, sde);
}
}  // namespace gbdx
