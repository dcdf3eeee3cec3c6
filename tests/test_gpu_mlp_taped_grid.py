"""BF16 neural ODEs with and without a recursive gradient, which run different kernels (the
row-tile integrator records the tape, the feature-major one serves the rest): on a constant
grid their saved states agree to FP32 rounding, and under the PID controller, where the
error estimates' rounding chooses the steps, their step counts stay close."""
import pytest
import torch

import diffrax_gb300 as dfx

pytestmark = pytest.mark.gpu


def solves(batch, d, h, solver, **kw):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(d + batch)
    w = (d, h, h, d)
    Ws = [(torch.randn(w[i + 1], w[i], device=dev, generator=gen) / w[i] ** 0.5)
          .bfloat16().float() for i in range(3)]
    bs = [0.1 * torch.randn(w[i + 1], device=dev, generator=gen) for i in range(3)]
    y0 = torch.randn(batch, d, device=dev, generator=gen)
    return [dfx.diffeqsolve(dfx.ODETerm(dfx.MLPField(Ws, bs, precision="bf16")), solver, 0.0, 1.0,
                            y0=y0.clone().requires_grad_(grad), saveat=dfx.SaveAt(
                                ts=torch.linspace(0, 1, 9, dtype=torch.float64)),
                            adjoint=dfx.RecursiveCheckpointAdjoint(), **kw)
            for grad in (True, False)]


@pytest.mark.parametrize("solver", [dfx.Euler(), dfx.Heun(), dfx.Tsit5(), dfx.Dopri5()])
@pytest.mark.parametrize("d,h", [(64, 128), (32, 64)])
@pytest.mark.parametrize("batch", [1, 33])
def test_equal_grids(batch, d, h, solver):
    # 16 steps; a sum of at most 128 products of size 1 is within 128 * 2^-24 = 8e-6 of
    # its terms' size, each step adds 1/16 of that
    taped, other = solves(batch, d, h, solver, dt0=1 / 16)
    assert torch.equal(taped.stats["num_steps"], other.stats["num_steps"])
    a, b = taped.ys.detach(), other.ys
    assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("d,h", [(64, 128), (32, 64)])
def test_adaptive_step_counts(d, h):
    taped, other = solves(997, d, h, dfx.Tsit5(), dt0=None,
                          stepsize_controller=dfx.PIDController(rtol=1e-5, atol=1e-7))
    n, m = (s.stats["num_accepted_steps"].double() for s in (taped, other))
    assert float((n - m).abs().max()) <= 2
    assert abs(float(n.mean() - m.mean())) <= 0.5
