"""The virtual Brownian tree at the sizes where its descent can go wrong, against
the FP64 oracle on the same integer stream: depth 0 and 1, odd and even depths (the
levels' normals are drawn in pairs, the leaf's with the last), the deepest cached
tree and one deeper than the cache, times on the tree's midpoints, both
directions of time, both widths of the draw (a pair of dimensions uncached, a quad
from the cached path)."""
import numpy as np
import pytest
import torch

import diffrax_gb300 as dfx
import oracle as O

pytestmark = pytest.mark.gpu

TOLS = [1.5, 0.7, 0.3, 2.0 ** -3, 0.99 * 2.0 ** -3, 2.0 ** -24, 2.0 ** -26]


def check(terms, t0, t1, dt0, y0, args, params):
    ts = np.linspace(t0, t1, 9)
    saveat = dfx.SaveAt(ts=ts)
    dev = torch.device("cuda")
    sol = dfx.diffeqsolve(terms, dfx.Heun(), t0, t1, dt0,
                          torch.tensor(y0, dtype=torch.float32, device=dev),
                          None if args is None else torch.tensor(args, dtype=torch.float32,
                                                                 device=dev), saveat=saveat)
    fields = dfx.lower(terms, dfx.Heun(), dfx.ConstantStepSize(), saveat, dim=y0.shape[1],
                       dtype=torch.float32, max_steps=4096, n_ts=ts.size)
    r = O.solve(O.make_desc(**O.oracle_fields(fields)), t0, t1, dt0, y0, args=args,
                params=params, ts=ts, nthreads=8)
    ys = sol.ys.cpu().double().numpy()
    # the times are multiples of 1/16, exact in FP32, so both descend the same
    # path; FP32 rounding of the increments remains
    err = np.abs(ys - r["ys"]).max() / np.abs(r["ys"]).max()
    assert err < 2e-5, err


@pytest.mark.parametrize("tol", TOLS)
@pytest.mark.parametrize("dim", [2, 4])
@pytest.mark.parametrize("back", [False, True])
def test_pairs(tol, dim, back):
    rng = np.random.default_rng(5)
    t0, t1, dt0 = (1.0, 0.0, -1 / 16) if back else (0.0, 1.0, 1 / 16)
    bm = dfx.VirtualBrownianTree(0.0, 1.0, tol, (dim,), key=2 ** 40 + 7)
    terms = dfx.MultiTerm(dfx.ODETerm(dfx.OrnsteinUhlenbeck()),
                          dfx.ControlTerm(dfx.OrnsteinUhlenbeck(), bm))
    check(terms, t0, t1, dt0, rng.uniform(-2, 2, (33, dim)), np.array([1.5, 0.5, 0.6]), None)


@pytest.mark.parametrize("tol", TOLS)
@pytest.mark.parametrize("back", [False, True])
def test_quads(tol, back):
    # zero drift and a constant diffusion 0.1 tanh(b): the path itself
    rng = np.random.default_rng(6)
    dev = torch.device("cuda")
    w = [32, 64, 64, 32]
    Ws = [np.zeros((w[i + 1], w[i])) for i in range(3)]
    bs = [np.zeros(w[i + 1]) for i in range(3)]
    Wd, bd = np.zeros((32, 32)), np.float32(rng.uniform(1, 2, 32)).astype(np.float64)
    f32 = lambda a: torch.tensor(a, dtype=torch.float32, device=dev)  # noqa: E731
    t0, t1, dt0 = (1.0, 0.0, -1 / 16) if back else (0.0, 1.0, 1 / 16)
    bm = dfx.VirtualBrownianTree(0.0, 1.0, tol, (32,), key=3)
    terms = dfx.MultiTerm(
        dfx.ODETerm(dfx.MLPField([f32(W) for W in Ws], [f32(b) for b in bs])),
        dfx.ControlTerm(dfx.TanhDiagonalDiffusion(f32(Wd), f32(bd)), bm))
    params = np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in zip(Ws, bs)] +
                            [Wd.reshape(-1), bd])
    check(terms, t0, t1, dt0, rng.uniform(-2, 2, (37, 32)), None, params)
