"""Run by test_gpu_lost_products.py with a library whose waits for a product all run out:
argv: the library, "fwd" or "bwd"."""
import sys

import torch

from diffrax_gb300 import _build

_build.LIB_PATH = sys.argv[1]
_build.is_stale = lambda bounds=False: False
import diffrax_gb300 as dfx  # noqa: E402

ERR = int(dfx.RESULTS.internal_error)
dev = torch.device("cuda")
W = (32, 64, 64, 32)


def mlp(grad):
    g = torch.Generator(device=dev).manual_seed(1)
    leaf = lambda *s: torch.randn(*s, device=dev, generator=g).div_(8).requires_grad_(grad)  # noqa: E731
    Ws = [leaf(W[i + 1], W[i]) for i in range(3)]
    bs = [leaf(W[i + 1]) for i in range(3)]
    return dfx.MLPField(Ws, bs), Ws + bs, leaf


def sound():
    # the context still serves: the same field's FP32 products, which wait for none
    field, _, leaf = mlp(False)
    field = dfx.MLPField(field.weights, field.biases, precision="fp32")
    sol = dfx.diffeqsolve(dfx.ODETerm(field), dfx.Tsit5(), 0.0, 1.0, 0.25, leaf(3, W[0]))
    assert bool(torch.isfinite(sol.ys).all())


def fwd(batch, solver, dt0, controller=dfx.ConstantStepSize(), **kw):
    field, _, leaf = mlp(False)
    y0 = leaf(batch, W[0])
    kw.update(stepsize_controller=controller)
    sol = dfx.diffeqsolve(dfx.ODETerm(field), solver, 0.0, 1.0, dt0, y0, throw=False, **kw)
    assert bool((sol.result == ERR).all()), sol.result.unique()
    try:
        dfx.diffeqsolve(dfx.ODETerm(field), solver, 0.0, 1.0, dt0, y0, **kw)
    except RuntimeError as e:
        assert f"({batch} of {batch} trajectories failed)" in str(e), e
    else:
        raise AssertionError("no error raised")


def bwd(batch, sde, steps):
    field, leaves, leaf = mlp(True)
    terms = dfx.ODETerm(field)
    if sde:
        Wd, bd = leaf(W[0], W[0]), leaf(W[0])
        leaves = leaves + [Wd, bd]
        terms = dfx.MultiTerm(terms, dfx.ControlTerm(
            dfx.TanhDiagonalDiffusion(Wd, bd),
            dfx.VirtualBrownianTree(0.0, 1.0, 1e-2, (W[0],), key=1)))
    y0 = leaf(batch, W[0])
    # (the forward that records the tape waits for no such product)
    sol = dfx.diffeqsolve(terms, dfx.Heun(), 0.0, 1.0, 1.0 / steps, y0)
    assert bool(torch.isfinite(sol.ys).all())
    for g in torch.autograd.grad(sol.ys.square().sum(), [y0] + leaves):
        assert bool(torch.isnan(g).all())


for B in (1, 33, 5000, 20000):
    if sys.argv[2] == "fwd":
        pid = dfx.PIDController(rtol=1e-5, atol=1e-7)
        # rows that end with the first step, later, with adaptive steps; saves; extended
        # outputs; an event whose condition is evaluated after the stages
        fwd(B, dfx.Tsit5(), 1.0)
        fwd(B, dfx.Euler(), 0.25, saveat=dfx.SaveAt(t0=True, ts=[0.5, 1.0]))
        fwd(B, dfx.Dopri5(), None, pid)
        fwd(B, dfx.Tsit5(), 0.5, saveat=dfx.SaveAt(steps=True), max_steps=8)
        fwd(B, dfx.Heun(), 1.0, event=dfx.Event(dfx.steady_state_event(rtol=1e3, atol=1e3)))
    else:
        for steps in (1, 3, 20):
            bwd(B, False, steps)
            bwd(B, True, steps)
    sound()
print("ok")
