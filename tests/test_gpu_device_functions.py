"""The kernels' hand-written functions on the device against FP64: tanh of pairs over its
whole range, at the join of its two forms and at special values; Box-Muller on uniform,
smallest and largest words; the place of a save in its step from the approximate
reciprocal.  Bounds are sums of each form's roundings and of the approximate instructions'
documented errors; the mean errors are held against the CUDA library's functions."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

from diffrax_gb300 import _build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("device") / "functions.so")
    subprocess.run([_build.nvcc(), *_build.NVCC_FLAGS, "-shared", "-cudart", "shared", "-I",
                    _build.CSRC, "-I", os.path.join(_build.ROOT, "include"), "-o", out,
                    os.path.join(HERE, "device_functions.cu")], check=True)
    torch.cuda.init()
    return ctypes.CDLL(out)


def run(f, ins, out_dtype, n_out, count):
    dev = [torch.from_numpy(a).cuda() for a in ins]
    out = torch.empty(n_out, dtype=out_dtype, device="cuda")
    assert f(*(ctypes.c_void_p(t.data_ptr()) for t in (*dev, out)), count) == 0
    return out.cpu().numpy()


def rms(x):
    return np.sqrt(np.mean(np.square(x.astype(np.float64))))


def test_tanh(lib):
    rng = np.random.default_rng(1)
    n = 1 << 20
    join = np.float32(0.65)
    near = join.view(np.int32) + np.arange(-512, 512, dtype=np.int32)
    x = np.concatenate([
        rng.standard_normal(n), 0.1 * rng.standard_normal(n), rng.uniform(-12, 12, n),
        np.exp(rng.uniform(np.log(1e-38), np.log(1e38), n)) * rng.choice([-1, 1], n),
        near.view(np.float32), -near.view(np.float32),
        [0.0, -0.0, 1e-45, -1e-45, 1e-40, 3e38, -3e38, 9.0, -9.0, 44.0]]).astype(np.float32)
    y = run(lib.run_tanh2, [x], torch.float32, x.size, x.size // 2)
    exact = np.tanh(x.astype(np.float64))
    err = np.abs(y - exact)
    # 1 - 2 / (1 + e) at the join: 2^-22 of e and its argument's rounding over 1.7, 2^-23
    # of the reciprocal, the last rounding; the polynomial's side stays below
    assert (err <= 3.5e-7 * np.abs(exact)).all(), (err / np.maximum(np.abs(exact), 1e-45)).max()
    assert (np.abs(y) <= 1).all()
    lib_err = run(lib.run_tanh_lib, [x], torch.float32, x.size, x.size // 2) - exact
    for k in range(2):  # N(0, 1), N(0, 0.01)
        part = slice(k * n, (k + 1) * n)
        assert rms(y[part] - exact[part]) <= rms(lib_err[part])
    special = np.array([np.inf, -np.inf, np.nan, 1.0, 2.0, np.nan], dtype=np.float32)
    y = run(lib.run_tanh2, [special], torch.float32, 6, 3)
    assert y[0] == 1 and y[1] == -1 and np.isnan(y[[2, 5]]).all()
    assert np.abs(y[3:5] - np.tanh([1.0, 2.0])).max() < 3.5e-7  # not touched by the NaNs


def test_box_muller(lib):
    rng = np.random.default_rng(2)
    n = 1 << 21
    u, v = (rng.integers(0, 2 ** 32, 2 * n, dtype=np.uint32) for _ in range(2))
    ends = np.array([0, 255, 256, 2 ** 31 - 1, 2 ** 31, 2 ** 32 - 1, 2 ** 30, 3 * 2 ** 30],
                    dtype=np.uint32)
    u[:64], v[:64] = np.repeat(ends, 8), np.tile(ends, 8)
    # the uniforms as the kernels hold them, in FP32
    a, b = (((w >> 8).astype(np.float64) + 0.5).astype(np.float32) / 2.0 ** 24 for w in (u, v))
    a, b = a.astype(np.float64), b.astype(np.float64)
    rad = np.sqrt(-2 * np.log(a))
    exact = np.stack([rad * np.cos(2 * np.pi * b), rad * np.sin(2 * np.pi * b)], 1).reshape(-1)
    words = [u.view(np.int32), v.view(np.int32)]
    z = run(lib.run_box, words, torch.float32, 4 * n, n)
    # half the logarithm's 2^-23, the root's 2^-23, 2^-23 of sine and cosine, the product
    bound = 3.5e-7 * np.repeat(rad, 2) + 1e-15
    assert (np.abs(z - exact) <= bound).all()
    assert rms(z - exact) <= 1.25 * rms(run(lib.run_box_lib, words, torch.float32, 4 * n, n) -
                                        exact)


def test_quotient(lib):
    rng = np.random.default_rng(3)
    n = 1 << 20
    b = np.exp2(rng.uniform(-80, 50, n)) * rng.choice([-1, 1], n)
    th = rng.uniform(0, 1, n)
    k = np.arange(n) % 4
    th = np.where(k == 1, np.exp2(-50 * th), np.where(k == 2, 1 - np.exp2(-50 * th), np.where(
        k == 3, th.astype(np.float32), th)))
    a = b * th
    q = run(lib.run_quotient, [a, b], torch.float32, n, n).astype(np.float64)
    x = a / b
    # one rounding to FP32 of a value within 2^-40, and of the FP64 quotient here
    assert (np.abs(q - x) <= (1 + 2.0 ** -12) * 2.0 ** -24 * np.abs(x)).all()
    assert (q <= 1).all()
    assert (run(lib.run_quotient, [b, b], torch.float32, n, n) == 1).all()
    assert (run(lib.run_quotient, [0 * b, b], torch.float32, n, n) == 0).all()
    ends = np.array([1e-300, 1e-45, 1e-30, 1e20, 1e300, 1.0, np.inf, np.nan])
    a, b = np.repeat(ends, 8), np.tile(ends, 8)
    q = run(lib.run_quotient, [a, b], torch.float32, 64, 64)
    with np.errstate(all="ignore"):
        assert np.array_equal(q, (a / b).astype(np.float32), equal_nan=True)
