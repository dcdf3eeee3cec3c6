"""The analytic RecursiveCheckpoint backward reads a step's record one step ahead, from
lines asked for eight steps ahead: solves of fewer, as many and more steps than that,
forward and reverse in time, against torch autograd through the same FP64 Heun steps.
Both run the same recurrences in FP64; 17 steps of some 50 roundings each, amplified at
most e^3 by the field over the interval, stay below 1e-11 of the largest component."""
import pytest
import torch

import diffrax_gb300 as dfx

pytestmark = pytest.mark.gpu


def heun(y, mu, h, n):
    def f(y):
        return torch.stack([y[:, 1], mu[:, 0] * (1 - y[:, 0] ** 2) * y[:, 1] - y[:, 0]], 1)

    for _ in range(n):
        k1 = f(y)
        y = y + h / 2 * (k1 + f(y + h * k1))
    return y


@pytest.mark.parametrize("steps", [0, 1, 2, 7, 8, 9, 17])
@pytest.mark.parametrize("sign", [1, -1])
def test_records_read_ahead(steps, sign):
    gen = torch.Generator().manual_seed(steps)
    y0 = torch.rand(37, 2, dtype=torch.float64, generator=gen) + 0.5
    mu = torch.rand(37, 1, dtype=torch.float64, generator=gen) + 0.2
    G = torch.randn(37, 2, dtype=torch.float64, generator=gen)
    ref = [x.clone().requires_grad_(True) for x in (y0, mu)]
    (heun(*ref, sign / 8, steps) * G).sum().backward()
    got = [x.cuda().requires_grad_(True) for x in (y0, mu)]
    sol = dfx.diffeqsolve(dfx.ODETerm(dfx.VanDerPol()), dfx.Heun(), 0.0, sign * steps / 8,
                          sign / 8, *got, stepsize_controller=dfx.ConstantStepSize(),
                          adjoint=dfx.RecursiveCheckpointAdjoint())
    (sol.ys[:, -1] * G.cuda()).sum().backward()
    for g, r in zip(got, ref):
        want = torch.zeros_like(r) if r.grad is None else r.grad
        assert float((g.grad.cpu() - want).abs().max()) <= 1e-11 * max(1.0, float(want.abs().max()))
