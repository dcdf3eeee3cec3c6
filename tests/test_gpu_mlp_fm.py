"""The feature-major tcgen05 form of the MLP integrator (BF16 ODE forward solves)
against the FP64 oracle at the edges of its tiles: ragged tiles of 32 rows, one
trajectory, more rows than the first tiles hold (the queue refills them), every
solver and shape, save counts around a pass of 8, both directions of time, per
trajectory intervals with an empty one, and parameters that are not 16-byte
aligned."""
import numpy as np
import pytest
import torch

import diffrax_gb300 as dfx
import oracle as O
from diffrax_gb300._integrate import Lowered

pytestmark = pytest.mark.gpu

SHAPES = [(64, 128), (64, 256), (32, 64)]
SOLVERS = {"euler": dfx.Euler(), "heun": dfx.Heun(), "dopri5": dfx.Dopri5(), "tsit5": dfx.Tsit5()}


def bf16(a):
    return torch.tensor(a, dtype=torch.float32).to(torch.bfloat16).double().numpy()


def make(shape, seed):
    D, H = shape
    rng = np.random.default_rng(seed)
    w = [D, H, H, D]
    Ws = [bf16(rng.standard_normal((w[i + 1], w[i])) / np.sqrt(w[i])) for i in range(3)]
    bs = [np.float32(0.1 * rng.standard_normal(w[i + 1])).astype(np.float64) for i in range(3)]
    return rng, Ws, bs


def solve(shape, solver, ctrl, t0, t1, dt0, B, ts=None, seed=0, shift=0, n_chk=200):
    """Largest error against the oracle, per trajectory relative to its largest value
    (the first and last n_chk trajectories)."""
    rng, Ws, bs = make(shape, seed)
    dev = torch.device("cuda")
    f32 = lambda a: torch.tensor(a, dtype=torch.float32, device=dev)  # noqa: E731
    y0 = np.float32(rng.standard_normal((B, shape[0]))).astype(np.float64)
    saveat = dfx.SaveAt(ts=ts, t1=True)
    terms = dfx.ODETerm(dfx.MLPField([f32(W) for W in Ws], [f32(b) for b in bs]))
    tt = lambda x: torch.tensor(x, dtype=torch.float64, device=dev) if isinstance(  # noqa: E731
        x, np.ndarray) else x
    low = Lowered(terms, solver, tt(t0), tt(t1), dt0, f32(y0), None, saveat, ctrl, None, 4096,
                  "auto", 0, 0)
    if shift:
        moved = torch.empty(low.params.numel() + shift, dtype=torch.float32, device=dev)[shift:]
        moved.copy_(low.params)
        low.params = moved
    ys, _, res, _ = low.run_forward()
    assert (res == 0).all()
    pick = np.unique(np.r_[np.arange(min(B, n_chk)), np.arange(max(0, B - n_chk), B)])
    sub = lambda x: x[pick] if isinstance(x, np.ndarray) else x  # noqa: E731
    params = np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in zip(Ws, bs)])
    r = O.solve(O.make_desc(**O.oracle_fields(low.fields)), sub(t0), sub(t1), dt0, y0[pick],
                params=params, ts=ts, nthreads=8)
    a, b = ys.double().cpu().numpy()[pick], r["ys"]
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    a, b = np.where(np.isfinite(b), a, 0), np.where(np.isfinite(b), b, 0)
    return (np.abs(a - b).max(axis=(1, 2)) / np.abs(b).max(axis=(1, 2))).max()


# constant steps: the same grid as the oracle's, so FP32 rounding alone: 20 steps of
# a field with Lipschitz constant of order one, 6e-8 a step and a few of it within
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("solver", list(SOLVERS))
@pytest.mark.parametrize("B", [1, 33])
def test_solvers(shape, solver, B):
    assert solve(shape, SOLVERS[solver], dfx.ConstantStepSize(), 0.0, 1.0, 0.05, B) < 1e-5


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("B", [31, 32, 64, 9727, 9729])
def test_tiles(shape, B):
    assert solve(shape, dfx.Heun(), dfx.ConstantStepSize(), 0.0, 1.0, 0.05, B) < 1e-5


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("solver", ["dopri5", "tsit5"])
def test_adaptive(shape, solver):
    # FP32 and FP64 controllers part at the tolerance level of 1e-5
    err = solve(shape, SOLVERS[solver], dfx.PIDController(rtol=1e-5, atol=1e-7), 0.0, 1.0, None,
                77, ts=np.linspace(0.0, 1.0, 5))
    assert err < 5e-5


@pytest.mark.parametrize("solver", list(SOLVERS))
@pytest.mark.parametrize("n", [1, 8, 9, 17])
@pytest.mark.parametrize("back", [False, True])
def test_saves(solver, n, back):
    # all of the times inside one step; the interpolant's value too is FP32 rounding
    ts = np.linspace(0.51, 0.74, n)
    t0, t1, dt0 = (1.0, 0.0, -0.25) if back else (0.0, 1.0, 0.25)
    err = solve((64, 128), SOLVERS[solver], dfx.ConstantStepSize(), t0, t1, dt0, 35,
                ts=ts[::-1].copy() if back else ts)
    assert err < 1e-5


@pytest.mark.parametrize("shape", SHAPES)
def test_uneven_intervals_and_refill(shape):
    rng = np.random.default_rng(3)
    B = 20011
    t1 = rng.uniform(0.1, 1.0, B)
    t1[::7] = 0.0
    assert solve(shape, dfx.Heun(), dfx.ConstantStepSize(), np.zeros(B), t1, 0.05, B) < 1e-5


@pytest.mark.parametrize("shape", SHAPES)
def test_unaligned_parameters(shape):
    assert solve(shape, dfx.Heun(), dfx.ConstantStepSize(), 0.0, 1.0, 0.05, 40, shift=1) < 1e-5


def test_nan_row_stays_alone():
    # a row that overflows ends at max_steps without touching its tile's other rows
    rng, Ws, bs = make((64, 128), 1)
    dev = torch.device("cuda")
    f32 = lambda a: torch.tensor(a, dtype=torch.float32, device=dev)  # noqa: E731
    terms = dfx.ODETerm(dfx.MLPField([f32(W) for W in Ws], [f32(b) for b in bs]))
    y0 = f32(rng.standard_normal((32, 64)))
    pid = dfx.PIDController(rtol=1e-5, atol=1e-7)
    good = dfx.diffeqsolve(terms, dfx.Tsit5(), 0.0, 1.0, None, y0, stepsize_controller=pid)
    bad0 = y0.clone()
    bad0[5, 3] = float("nan")
    bad = dfx.diffeqsolve(terms, dfx.Tsit5(), 0.0, 1.0, None, bad0, stepsize_controller=pid,
                          max_steps=64, throw=False)
    keep = torch.arange(32, device=dev) != 5
    assert torch.equal(bad.ys[keep], good.ys[keep])
    assert int(bad.result[5]) == int(dfx.RESULTS.max_steps_reached)
