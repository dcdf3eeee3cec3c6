"""A BF16 neural ODE solved for a recursive gradient (the row-tile integrator, which
records the tape) against the same solve without one (the feature-major integrator), over
full and ragged tiles.  Both keep the local error of each of their some five steps within
rtol |y| + atol, and the field's Lipschitz constant over [0, 1] amplifies it at most
tenfold: the saved states agree within 1e-3 of the largest component."""
import pytest
import torch

import diffrax_gb300 as dfx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [dfx.Tsit5(), dfx.Dopri5()])
@pytest.mark.parametrize("d,h", [(64, 128), (32, 64)])
@pytest.mark.parametrize("batch", [1, 31, 33, 97])
def test_taped_and_untaped_solves_agree(batch, d, h, solver):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(d + batch)
    w = (d, h, h, d)
    Ws = [torch.randn(w[i + 1], w[i], device=dev, generator=gen) / w[i] ** 0.5 for i in range(3)]
    bs = [0.1 * torch.randn(w[i + 1], device=dev, generator=gen) for i in range(3)]
    y0 = torch.randn(batch, d, device=dev, generator=gen)
    ys = []
    for grad in (True, False):
        y = y0.clone().requires_grad_(grad)
        sol = dfx.diffeqsolve(
            dfx.ODETerm(dfx.MLPField(Ws, bs, precision="bf16")), solver, 0.0, 1.0, None, y,
            stepsize_controller=dfx.PIDController(rtol=1e-5, atol=1e-7),
            adjoint=dfx.RecursiveCheckpointAdjoint())
        if grad:
            sol.ys.square().sum().backward()
            assert torch.isfinite(y.grad).all() and bool((y.grad != 0).any())
        ys.append(sol.ys.detach())
    assert float((ys[0] - ys[1]).abs().max()) <= 1e-3 * float(ys[1].abs().max())
