"""The parameter pass of the BF16 BacksolveAdjoint, over the layers' run lengths and full
and ragged tiles of rows: its scaled errors are formed one way for every tolerance, so
absolute tolerances that no component can see lead to the same steps and to the same
gradients, up to the FP32 rounding of sums over rows (bounded here by 1e-5 of the
largest component)."""
import pytest
import torch

import diffrax_gb300 as dfx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,h", [(64, 256), (64, 128), (32, 64)])
@pytest.mark.parametrize("batch", [1, 33])
def test_invisible_tolerances_agree(d, h, batch):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(d + h + batch)
    w = (d, h, h, d)
    Ws = [torch.randn(w[i + 1], w[i], device=dev, generator=gen) / w[i] ** 0.5 for i in range(3)]
    bs = [0.1 * torch.randn(w[i + 1], device=dev, generator=gen) for i in range(3)]
    y0 = torch.randn(batch, d, device=dev, generator=gen)
    G = torch.randn(batch, 5, d, device=dev, generator=gen)
    ts = torch.linspace(0.0, 1.0, 5, dtype=torch.float64, device=dev)

    def grads(atol):
        leaves = [x.clone().requires_grad_(True) for x in Ws + bs + [y0]]
        ctrl = dfx.PIDController(rtol=1e-2, atol=atol)
        sol = dfx.diffeqsolve(
            dfx.ODETerm(dfx.MLPField(leaves[:3], leaves[3:6], precision="bf16")), dfx.Tsit5(),
            0.0, 1.0, None, leaves[6], saveat=dfx.SaveAt(ts=ts),
            stepsize_controller=dfx.PIDController(rtol=1e-5, atol=1e-7),
            adjoint=dfx.BacksolveAdjoint(stepsize_controller=ctrl))
        (sol.ys * G).sum().backward()
        return [x.grad for x in leaves], sol.lowered.bwd_stats

    fast, s_fast = grads(1e-29)
    full, s_full = grads(1e-31)
    assert torch.equal(s_fast, s_full)
    for a, b in zip(fast, full):
        assert torch.isfinite(a).all()
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
