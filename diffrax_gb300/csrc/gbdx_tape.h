// gbdx_tape.h -- sizes of the recursive adjoint's tape (MLP fields): the host lays the
// workspace out by them, the kernels index within them.
#pragma once

namespace gbdx {

// State slots a trajectory for a requested count.  An even count keeps the online
// thinning exact: when the slots fill at step n = C s, n is a multiple of the doubled
// stride 2 s.
inline int tape_slots(int checkpoints) {
  return checkpoints >= 4 ? (checkpoints / 2) * 2 : 2;
}

// Recomputed states a trajectory between two slots.  With C slots the stride stays
// below 2 max_steps / C + 1, and the segment's first state is the slot's.
inline int tape_segment(int max_steps, int slots) {
  const long long seg = (2ll * max_steps + slots - 1) / slots + 1;
  return int(seg < max_steps + 1ll ? seg : max_steps + 1ll);
}

}  // namespace gbdx
