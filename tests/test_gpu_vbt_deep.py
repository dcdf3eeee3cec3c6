"""Virtual Brownian trees deeper than a 32-bit path: one level around the word size, and
tolerances far below what an FP32 time resolves, against the FP64 oracle on the same
integer stream.  Step times are multiples of 59999 / 2^20 (20 bits, exact in FP32), so
the path turns on every upper level and both sides descend the same one; every level
below the 20th ends at the time itself, where the bridge has no width left, and FP32
rounding of the increments remains (2e-5 of the largest value, as on shallower trees)."""
import numpy as np
import pytest
import torch

import diffrax_gb300 as dfx
import oracle as O

pytestmark = pytest.mark.gpu

TOLS = [2.0 ** -30, 2.0 ** -31, 2.0 ** -32, 2.0 ** -33, 1e-10, 2.0 ** -40, 1e-12]
N, H = 16, 59999 / 2 ** 20


def span(back):
    return (N * H, 0.0, -H) if back else (0.0, N * H, H)


def solve(terms, back, y0, args):
    t0, t1, dt0 = span(back)
    saveat = dfx.SaveAt(ts=np.arange(N + 1)[::-1 if back else 1] * H)
    f32 = lambda a: None if a is None else torch.tensor(  # noqa: E731
        a, dtype=torch.float32, device="cuda")
    return dfx.diffeqsolve(terms, dfx.Heun(), t0, t1, dt0, f32(y0), f32(args),
                           saveat=saveat), saveat


def check(terms, back, y0, args, params):
    sol, saveat = solve(terms, back, y0, args)
    t0, t1, dt0 = span(back)
    fields = dfx.lower(terms, dfx.Heun(), dfx.ConstantStepSize(), saveat, dim=y0.shape[1],
                       dtype=torch.float32, max_steps=4096, n_ts=saveat.ts.size)
    r = O.solve(O.make_desc(**O.oracle_fields(fields)), t0, t1, dt0, y0, args=args,
                params=params, ts=saveat.ts, nthreads=8)
    err = np.abs(sol.ys.cpu().double().numpy() - r["ys"]).max() / np.abs(r["ys"]).max()
    assert err < 2e-5, err


def ou(tol, dim, key=2 ** 40 + 7, t1=1.0):
    bm = dfx.VirtualBrownianTree(0.0, t1, tol, (dim,), key=key)
    return dfx.MultiTerm(dfx.ODETerm(dfx.OrnsteinUhlenbeck()),
                         dfx.ControlTerm(dfx.OrnsteinUhlenbeck(), bm))


@pytest.mark.parametrize("tol", TOLS)
@pytest.mark.parametrize("dim", [2, 4])
@pytest.mark.parametrize("back", [False, True])
def test_pairs(tol, dim, back):
    y0 = np.random.default_rng(5).uniform(-2, 2, (33, dim))
    check(ou(tol, dim), back, y0, np.array([1.5, 0.5, 0.6]), None)


def test_tolerance_relative_to_the_interval():
    # 1e-7 of [0, 1024]: 34 levels, the times divided by 1024 exactly
    y0 = np.random.default_rng(7).uniform(-2, 2, (33, 2))
    check(ou(1e-7, 2, t1=1024.0), False, y0, np.array([1.5, 0.5, 0.6]), None)


@pytest.mark.parametrize("tol", TOLS)
@pytest.mark.parametrize("back", [False, True])
def test_quads(tol, back):
    # zero drift and a constant diffusion 0.1 tanh(b): the path itself
    rng = np.random.default_rng(6)
    w = [32, 64, 64, 32]
    Ws = [np.zeros((w[i + 1], w[i])) for i in range(3)]
    bs = [np.zeros(w[i + 1]) for i in range(3)]
    Wd, bd = np.zeros((32, 32)), np.float32(rng.uniform(1, 2, 32)).astype(np.float64)
    f32 = lambda a: torch.tensor(a, dtype=torch.float32, device="cuda")  # noqa: E731
    bm = dfx.VirtualBrownianTree(0.0, 1.0, tol, (32,), key=3)
    terms = dfx.MultiTerm(
        dfx.ODETerm(dfx.MLPField([f32(W) for W in Ws], [f32(b) for b in bs])),
        dfx.ControlTerm(dfx.TanhDiagonalDiffusion(f32(Wd), f32(bd)), bm))
    params = np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in zip(Ws, bs)] +
                            [Wd.reshape(-1), bd])
    check(terms, back, rng.uniform(-2, 2, (37, 32)), None, params)


@pytest.mark.parametrize("tol", [1e-30, 1e-44, 1e-60])
def test_below_the_smallest_float(tol):
    # more levels than FP64 can follow in the oracle: the value at an exact time is that
    # of any tree that resolves it
    y0, args = np.ones((33, 2)), np.array([1.5, 0.5, 0.6])
    got = solve(ou(tol, 2), False, y0, args)[0].ys
    want = solve(ou(2.0 ** -28, 2), False, y0, args)[0].ys
    assert float((got - want).abs().max()) < 2e-5 * float(want.abs().max())


def neural(tol, precision, grad):
    """A neural SDE on the path of a tree of tolerance tol, at exact times."""
    dev, w = torch.device("cuda"), (32, 64, 64, 32)
    gen = torch.Generator(device=dev).manual_seed(9)
    leaf = lambda *s: torch.randn(*s, device=dev, generator=gen).div_(  # noqa: E731
        s[-1] ** 0.5).requires_grad_(grad)
    Ws, bs = [leaf(w[i + 1], w[i]) for i in range(3)], [leaf(w[i + 1]) for i in range(3)]
    Wd, bd, y0 = leaf(32, 32), leaf(32), leaf(45, 32)
    terms = dfx.MultiTerm(dfx.ODETerm(dfx.MLPField(Ws, bs, precision=precision)), dfx.ControlTerm(
        dfx.TanhDiagonalDiffusion(Wd, bd), dfx.VirtualBrownianTree(0.0, 1.0, tol, (32,), key=3)))
    return terms, y0, [y0, *Ws, *bs, Wd, bd]


@pytest.mark.parametrize("precision", ["bf16", "fp32"])
@pytest.mark.parametrize("tol", [2.0 ** -31, 1e-10, 1e-60])
def test_gradients(tol, precision):
    # the path at the steps' times is that of a tree that resolves them (2e-5, above)
    grads = []
    for t in (tol, 2.0 ** -28):
        terms, y0, leaves = neural(t, precision, True)
        sol = dfx.diffeqsolve(terms, dfx.Heun(), 0.0, N * H, H, y0)
        grads.append(torch.autograd.grad(sol.ys.square().sum(), leaves))
    for a, b in zip(*grads):
        assert float((a - b).norm()) <= 2e-5 * float(b.norm())


@pytest.mark.parametrize("precision", ["bf16", "fp32"])
def test_extended_outputs(precision):
    ys = []
    for t in (1e-10, 2.0 ** -28):
        terms, y0, _ = neural(t, precision, False)
        ys.append(dfx.diffeqsolve(terms, dfx.Heun(), 0.0, N * H, H, y0, max_steps=N,
                                  saveat=dfx.SaveAt(steps=True)).ys)
    assert float((ys[0] - ys[1]).abs().max()) <= 2e-5 * float(ys[1].abs().max())
