"""The default count of tape states: all of an ordinary solve's where the tape is small,
and never more memory than the log2 count's, with the segments it recomputes, where it is
large."""
import math

import pytest
import torch

import diffrax_gb300 as dfx
from diffrax_gb300 import _lib
from diffrax_gb300._integrate import _TAPE_BYTES, _tape_count, _tape_states

STEPS = list(range(1, 1400)) + [2048, 4096, 4097, 10 ** 5, 2 ** 31 - 2]


def few(max_steps):
    return max(1, math.ceil(math.log2(max(max_steps, 2))))


def test_memory_of_the_default():
    for m in STEPS:
        assert _tape_count(m, 1) == min(128, max(2, m // 2 * 2))
        large = _tape_count(m, _TAPE_BYTES)
        assert _tape_states(m, large) <= _tape_states(m, few(m))
        assert few(m) - 1 <= large <= 128
    # the default max_steps: a large batch keeps the count of a small one
    assert _tape_count(4096, _TAPE_BYTES) == 128


@pytest.mark.gpu
@pytest.mark.parametrize("max_steps", [16, 100, 400, 4096])
def test_workspace_of_a_large_batch(max_steps):
    B, w = 2 ** 19, (64, 128, 128, 64)
    field = dfx.MLPField([torch.zeros(w[i + 1], w[i]) for i in range(3)],
                         [torch.zeros(w[i + 1]) for i in range(3)])

    def size(count):
        fields = dfx.lower(dfx.ODETerm(field), dfx.Tsit5(), dfx.PIDController(1e-5, 1e-7),
                           dfx.SaveAt(t1=True), dim=64, dtype=torch.float32,
                           max_steps=max_steps, n_ts=0,
                           adjoint=dfx.RecursiveCheckpointAdjoint(checkpoints=count))
        return _lib.get_problem(fields).workspace_size(B)

    assert size(_tape_count(max_steps, B * 64 * 4)) <= size(few(max_steps))
