// gbdx_mlp_fm_xo_d32h64.cu -- feature-major MLP integrator instantiations with the
// extended outputs (SaveAt(steps=n), SaveAt(dense=True), the clip controller, events,
// resume records) for state dim 32, hidden width 64.
#include "gbdx_mlp_fm.cuh"

namespace gbdx {
OdeEntry find_mlp_fm_xo_entry_d32h64(int solver) { return fm_entry<32, 64, true>(solver); }
}  // namespace gbdx
