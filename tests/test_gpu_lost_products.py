"""A tensor-core product whose completion does not show within the wait's limit: every
trajectory that it, or its group's early end, could touch reports an internal error, every
gradient is NaN, and the context goes on.  The feature-major 32-64 kernels are built with a
limit of no polls at all, so that each wait runs out; their products do complete, and the
kernels wait for that before they leave."""
import os
import subprocess
import sys

import pytest

from diffrax_gb300 import _build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def impatient(tmp_path_factory):
    _build.build()
    out = tmp_path_factory.mktemp("impatient")
    units = ["gbdx_mlp_fm_d32h64", "gbdx_mlp_fm_xo_d32h64", "gbdx_mlp_fm_bwd_d32h64"]
    jobs = [subprocess.Popen([_build.nvcc(), *_build.NVCC_FLAGS, "-DGBDX_FM_POLLS=0u", "-I",
                              os.path.join(_build.ROOT, "include"), "-c",
                              os.path.join(_build.CSRC, u + ".cu"), "-o", str(out / (u + ".o"))])
            for u in units]
    assert [j.wait() for j in jobs] == [0] * len(units)
    objs = [str(out / (u + ".o")) for u in units]
    objs += [os.path.join(_build.OBJ_DIR, os.path.basename(s)[:-3] + ".o")
             for s in _build.sources() if os.path.basename(s)[:-3] not in units]
    lib = str(out / "libgbdx_impatient.so")
    subprocess.run([_build.nvcc(), "-shared", "-cudart", "shared", *_build.ARCH, "-o", lib, *objs],
                   check=True)
    return lib


@pytest.mark.parametrize("way", ["fwd", "bwd"])
def test_lost_products(impatient, way):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(
        [os.path.dirname(HERE), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, os.path.join(HERE, "lost_products_child.py"), impatient,
                        way], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout[-3000:] + r.stderr[-3000:]
