"""Invalid save times are refused before the solve is launched where the host holds every
time, where the solve has no step bound, and where it would allocate dense records; and
the sign of dt0 is checked for any number that a time may be."""
from decimal import Decimal

import numpy as np
import pytest
import torch

import diffrax_gb300 as dfx
from diffrax_gb300 import _integrate

pytestmark = pytest.mark.gpu

OUT, MIXED = "between t0 and t1", "increasing or decreasing"
BAD = [([0.5, 1.5], OUT), ([-1e-9, 0.5], OUT), ([0.5, 0.25], MIXED), ([1.5], OUT)]
FORMS = {"list": list, "array": np.array, "tensor": lambda x: torch.tensor(
    x, dtype=torch.float64), "device": lambda x: torch.tensor(x, dtype=torch.float64,
                                                              device="cuda")}


def solve(ts, sign=1, t0=0.0, t1=1.0, dt0=None, **kw):
    y0 = torch.ones(3, 2, device="cuda")
    if sign < 0:
        t0, t1 = -t0, -t1
    return dfx.diffeqsolve(dfx.ODETerm(dfx.VanDerPol()), dfx.Tsit5(), t0, t1, dt0, y0,
                           torch.ones(3, 1, device="cuda"), saveat=dfx.SaveAt(
                               ts=ts, dense=kw.pop("dense", False)),
                           stepsize_controller=dfx.PIDController(rtol=1e-6, atol=1e-8), **kw)


@pytest.mark.parametrize("form,kw", [
    ("list", {}), ("array", {}), ("tensor", {}), ("list", {"throw": False}),
    ("device", {"max_steps": None}), ("device", {"dense": True, "max_steps": 16}),
    ("list", {"t1": torch.ones(3, dtype=torch.float64), "max_steps": None})])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("bad,message", BAD)
def test_refused_before_the_launch(monkeypatch, form, kw, sign, bad, message):
    def launched(*a, **k):
        raise AssertionError("the solve was launched")
    make = FORMS[form]
    if not (form == "tensor" and kw):
        solve(make([sign * t for t in (0.0, 0.25, 0.25, 1.0)]), sign, **kw)  # a valid one
    monkeypatch.setattr(_integrate.Lowered, "run_forward", launched)
    monkeypatch.setattr(_integrate.Lowered, "run_forward_ex", launched)
    with pytest.raises(RuntimeError, match=message):
        solve(make([sign * t for t in bad]), sign, **kw)


def test_equal_times():
    # t0 == t1 counts as backwards: only that time lies inside
    solve([2.0, 2.0], t0=2.0, t1=2.0)
    with pytest.raises(RuntimeError, match=OUT):
        solve([2.0 + 1e-9], t0=2.0, t1=2.0)


@pytest.mark.parametrize("number", [float, Decimal, np.float64, np.float32])
def test_sign_of_dt0(number):
    solve([0.5], dt0=number("0.125") if number is Decimal else number(0.125),
          t0=number(0), t1=number(1))
    with pytest.raises(ValueError, match="dt0"):
        solve([0.5], dt0=-0.125, t0=number(0), t1=number(1))
