"""The recursive adjoint's tape for every count of states, odd ones among them: its sizes
hold the walk that fills it (compiled for the host), and gradients do not depend on it."""
import os
import shutil
import subprocess

import pytest
import torch

import diffrax_gb300 as dfx

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "diffrax_gb300", "csrc")


def test_sizes_hold_the_walk(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "tape_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "tape_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["bf16", "fp32"])
@pytest.mark.parametrize("checkpoints,steps", [(1, 5), (3, 17), (3, 16), (5, 33), (7, 97),
                                               (8, 97)])
def test_gradients_do_not_depend_on_the_count(checkpoints, steps, precision):
    # the recomputed states come from other kernels than the tape's, in FP32
    dev, w = torch.device("cuda"), (32, 64, 64, 32)
    gen = torch.Generator(device=dev).manual_seed(steps)
    leaf = lambda *s: torch.randn(*s, device=dev, generator=gen).div_(  # noqa: E731
        s[-1] ** 0.5).requires_grad_()
    Ws, bs = [leaf(w[i + 1], w[i]) for i in range(3)], [leaf(w[i + 1]) for i in range(3)]
    y0 = leaf(37, w[0])
    grads = []
    for count in (checkpoints, 2 * steps):
        sol = dfx.diffeqsolve(dfx.ODETerm(dfx.MLPField(Ws, bs, precision=precision)), dfx.Heun(),
                              0.0, 1.0, 1.0 / steps, y0, max_steps=steps,
                              adjoint=dfx.RecursiveCheckpointAdjoint(checkpoints=count))
        grads.append(torch.autograd.grad(sol.ys.square().sum(), [y0, *Ws, *bs]))
    for a, b in zip(*grads):
        assert float((a - b).norm()) <= 2e-5 * float(b.norm())
