"""A solve's outcome in one launch (gbdx_solve_status): failed trajectories are counted
and the first one's code raised, saveat.ts on the device is checked in either direction
of time and against every trajectory's interval, at batches around the kernel's block
and grid sizes, on streams and threads of their own."""
import threading

import pytest
import torch

import diffrax_gb300 as dfx

pytestmark = pytest.mark.gpu

PID = dfx.PIDController(rtol=1e-6, atol=1e-8)


def solve(B, t0=0.0, t1=1.0, ts=None, max_steps=4096, throw=True):
    y0 = torch.ones(B, 2, device="cuda")
    mu = torch.ones(B, 1, device="cuda")
    saveat = dfx.SaveAt(t1=True) if ts is None else dfx.SaveAt(
        ts=torch.tensor(ts, dtype=torch.float64, device="cuda"))
    return dfx.diffeqsolve(dfx.ODETerm(dfx.VanDerPol()), dfx.Tsit5(), t0, t1, None, y0, mu,
                           saveat=saveat, stepsize_controller=PID, max_steps=max_steps,
                           throw=throw)


@pytest.mark.parametrize("B", [1, 255, 1024, 1025, 70001])
def test_counts_failures(B):
    t1 = torch.full((B,), 1e-3, dtype=torch.float64, device="cuda")
    solve(B, t1=t1)
    t1[B // 2:] = 20.0  # out of steps
    with pytest.raises(RuntimeError, match=rf"max.*\({B - B // 2} of {B} trajectories"):
        solve(B, t1=t1, max_steps=16)
    solve(B, t1=torch.full_like(t1, 1e-3))  # the scratch is clean again
    assert int((solve(B, t1=t1, max_steps=16, throw=False).result != 0).sum()) == B - B // 2


@pytest.mark.parametrize("throw", [True, False])
@pytest.mark.parametrize("back", [False, True])
@pytest.mark.parametrize("n", [2, 256, 257, 700])
def test_times(throw, back, n):
    t0, t1 = (1.0, 0.0) if back else (0.0, 1.0)
    good = torch.linspace(t0, t1, n, dtype=torch.float64).tolist()
    solve(3, t0, t1, good, throw=throw)
    swapped = list(good)
    swapped[-1], swapped[-2] = swapped[-2], swapped[-1]
    with pytest.raises(RuntimeError, match="increasing or decreasing"):
        solve(3, t0, t1, swapped, throw=throw)
    for at, x in ((0, t0 + 1e-9 * (t0 - t1)), (-1, t1 + 1e-9 * (t1 - t0))):
        outside = list(good)
        outside[at] = x
        with pytest.raises(RuntimeError, match="between t0 and t1"):
            solve(3, t0, t1, outside, throw=throw)
    solve(3, t0, t1, [0.5])
    with pytest.raises(RuntimeError, match="between t0 and t1"):
        solve(3, t0, t1, [1.5], throw=throw)


def test_times_against_every_interval():
    t1 = torch.ones(5000, dtype=torch.float64, device="cuda")
    solve(5000, t1=t1, ts=[0.25, 0.5])
    t1[4321] = 0.4
    with pytest.raises(RuntimeError, match="between t0 and t1"):
        solve(5000, t1=t1, ts=[0.25, 0.5])


def test_threads_and_streams():
    bad = []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    if k % 2:
                        solve(100 + k, ts=[0.1, 0.9])
                    else:
                        try:
                            solve(100 + k, ts=[0.9, 0.1])
                            bad.append(k)
                        except RuntimeError as e:
                            if "increasing or decreasing" not in str(e):
                                bad.append(str(e))
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
