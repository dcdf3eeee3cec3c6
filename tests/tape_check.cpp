// The recursive adjoint's tape sizes (diffrax_gb300/csrc/gbdx_tape.h) against the walk
// that fills them: every accepted state while the slots last, then every 2nd, 4th, ...
// step; a segment's states after its slot in the scratch.  Exits 1 where an index would
// pass its buffer.
#include <stdio.h>

#include "gbdx_tape.h"

int main() {
  long bad = 0;
  for (int checkpoints = 0; checkpoints <= 130; checkpoints++) {
    const int C = gbdx::tape_slots(checkpoints);
    bad += C < 2 || C % 2 || C > (checkpoints > 2 ? checkpoints : 2);
    for (int max_steps = 1; max_steps <= 4500; max_steps += max_steps < 1300 ? 1 : 37) {
      const int seg = gbdx::tape_segment(max_steps, C);
      // the accepted steps of one trajectory, and after each the tape as it would end
      int stride = 1;
      for (int n = 1; n <= max_steps; n++) {
        if (n % stride == 0) {
          int slot = n / stride;
          if (slot >= C) {
            stride *= 2;
            bad += n % stride != 0;  // the slot would hold another step's state
            slot = n / stride;
          }
          bad += slot >= C;
        }
        // the longest segment of n steps: states of the steps after its slot
        const int longest = stride < n ? stride : n;
        bad += longest - 1 > seg;
      }
    }
  }
  printf("%ld indexes outside\n", bad);
  return bad ? 1 : 0;
}
