"""The default number of tape states: enough for an ordinary solve, and the log2 count
once the tape of the batch would pass 16 GiB; never more than the steps."""
import pytest

from diffrax_gb300._integrate import _TAPE_BYTES, _default_checkpoints


@pytest.mark.parametrize("max_steps,small,large", [
    (1, 2, 1), (2, 2, 1), (3, 2, 2), (16, 16, 4), (127, 126, 7), (128, 128, 7),
    (4096, 128, 12)])
def test_default_checkpoints(max_steps, small, large):
    assert _default_checkpoints(max_steps) == small
    fits = _TAPE_BYTES // small
    assert _default_checkpoints(max_steps, fits) == small
    assert _default_checkpoints(max_steps, fits + 1) == large
