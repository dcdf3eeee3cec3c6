"""The feature-major tcgen05 backward (RecursiveCheckpointAdjoint, BF16 products) at
the edges of its tiles and paths, against the FP64 oracle's discretise-then-optimise
gradient: ragged tiles of 32 rows, more rows than the first tiles hold, every solver and
shape, saves inside steps (the last stage of an SSAL tableau then has a cotangent) and
none, few checkpoints (recompute iterations), more iterations than sums are kept for, an
interval of length zero, parameters that are not 16-byte aligned."""
import numpy as np
import pytest
import torch

import diffrax_gb300 as dfx
from test_gpu_grad import grad_case, rel

pytestmark = pytest.mark.gpu

ODE = [64, 128, 128, 64]
SMALL = [32, 64, 64, 32]
SOLVERS = [dfx.Euler(), dfx.Heun(), dfx.Dopri5(), dfx.Tsit5()]
# constant steps, so the same grid as the oracle's: FP32 rounding of some 20 to 60 steps
# and their VJPs, a few 1e-6 at most; the tolerance of the FP32 form's tests
TOL = 1e-4


def check(*args, **kw):
    g_y0, g_p, r, _ = grad_case(*args, **kw)
    assert rel(g_y0, r["grad_y0"]) < TOL
    assert rel(g_p, r["grad_params"]) < TOL


@pytest.mark.parametrize("widths", [ODE, SMALL])
@pytest.mark.parametrize("solver", SOLVERS)
@pytest.mark.parametrize("saves", [False, True])
def test_solvers(widths, solver, saves):
    saveat = dfx.SaveAt(t0=True, ts=np.array([0.3, 0.52, 0.54, 1.0]), t1=True) if saves else \
        dfx.SaveAt(t1=True)
    check(widths, solver, dfx.ConstantStepSize(), saveat, 1.0, 0.05, 33, "bf16", checkpoints=64,
          seed=1)


@pytest.mark.parametrize("B", [1, 31, 32, 64])
@pytest.mark.parametrize("widths,sde", [(ODE, False), (SMALL, False), (SMALL, True)])
def test_tiles(B, widths, sde):
    check(widths, dfx.Heun(), dfx.ConstantStepSize(), dfx.SaveAt(t1=True), 1.0, 0.05, B, "bf16",
          checkpoints=64, seed=2, sde=sde)


@pytest.mark.parametrize("checkpoints", [2, 5, 16, None])
@pytest.mark.parametrize("sde", [False, True])
def test_recompute(checkpoints, sde):
    check(SMALL, dfx.Heun() if sde else dfx.Tsit5(), dfx.ConstantStepSize(),
          dfx.SaveAt(t1=True, ts=np.array([0.5])), 1.0, 0.02, 40, "bf16",
          checkpoints=checkpoints, seed=3, sde=sde)


@pytest.mark.parametrize("widths", [ODE, SMALL])
def test_uneven_intervals_and_refill(widths):
    # 4901 rows: more than 152 tiles of 32, refilled from the queue; one step each
    rng = np.random.default_rng(4)
    t1 = rng.uniform(0.05, 0.25, 4901)
    t1[::9] = 0.0
    check(widths, dfx.Heun(), dfx.ConstantStepSize(), dfx.SaveAt(t1=True), t1, 0.05, 4901,
          "bf16", checkpoints=8, seed=4)


def test_unaligned_parameters():
    from diffrax_gb300._integrate import Lowered
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(0)
    Ws = [torch.randn(ODE[i + 1], ODE[i], device=dev, generator=g) / ODE[i] ** 0.5
          for i in range(3)]
    bs = [torch.randn(ODE[i + 1], device=dev, generator=g) for i in range(3)]
    y0 = torch.randn(40, 64, device=dev, generator=g)
    low = Lowered(dfx.ODETerm(dfx.MLPField(Ws, bs)), dfx.Heun(), 0.0, 1.0, 0.1, y0, None,
                  dfx.SaveAt(t1=True), dfx.ConstantStepSize(), dfx.RecursiveCheckpointAdjoint(),
                  4096, "auto", 0, 0, want_grad=True)
    out = []
    for shift in (0, 1):
        p = torch.empty(low.params.numel() + shift, device=dev)[shift:]
        p.copy_(low.params)
        ys, _, _, _, ws = low.run_forward(params=p, keep_workspace=True)
        out.append(low.run_backward(ws, 2 * ys, y0, p))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
