// gbdx_mlp_fm_xo_d64h256.cu -- feature-major MLP integrator instantiations with the
// extended outputs (SaveAt(steps=n), SaveAt(dense=True), the clip controller, events,
// resume records) for state dim 64, hidden width 256.
#include "gbdx_mlp_fm.cuh"

namespace gbdx {
OdeEntry find_mlp_fm_xo_entry_d64h256(int solver) { return fm_entry<64, 256, true>(solver); }
}  // namespace gbdx
