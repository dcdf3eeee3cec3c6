"""The tensor-core parameter pass of the BF16 BacksolveAdjoint against the FP64 oracle, on
constant steps (both sides take the same ones), for every shape and solver that it serves
and a full, a ragged and a single-row tile.  The products of stage differences are BF16:
with steps of 1/32 a difference is some 5 % of its vector, so their rounding is at most
2 * 2^-9 * 0.05^2 = 1e-5 of a gradient, and FP32 rounding stays below that; a tile of
another block, a swapped fragment or a missing term is 1e-3 and more."""
import numpy as np
import pytest

import diffrax_gb300 as dfx
from test_gpu_backsolve import backsolve_case, rel

pytestmark = pytest.mark.gpu

CASES = [((32, 64, 64, 32), s) for s in (dfx.Euler(), dfx.Heun(), dfx.Dopri5(), dfx.Tsit5())]
CASES += [((64, 128, 128, 64), dfx.Tsit5())]
CASES += [((64, 256, 256, 64), s) for s in (dfx.Tsit5(), dfx.Dopri5())]


@pytest.mark.parametrize("widths,solver", CASES)
@pytest.mark.parametrize("batch", [1, 16, 33])
def test_gradients_on_constant_steps(widths, solver, batch):
    c = backsolve_case(list(widths), solver, dfx.ConstantStepSize(), np.array([0.3, 0.55, 1.0]),
                       batch, "bf16", seed=batch, dt0=1 / 32)
    r = c["oracle"]
    assert np.array_equal(c["stats"], r["stats"])
    e0, ep = rel(c["g_y0"], r["grad_y0"]), rel(c["g_params"], r["grad_params"])
    assert e0 < 1e-4 and ep < 1e-4, (e0, ep)
    # every parameter block by its own size
    at = 0
    for i in range(3):
        for n in (widths[i] * widths[i + 1], widths[i + 1]):
            part = slice(at, at + n)
            e = rel(c["g_params"][part], r["grad_params"][part])
            assert e < 1e-4, (i, n, e)
            at += n
    assert at == c["g_params"].size
