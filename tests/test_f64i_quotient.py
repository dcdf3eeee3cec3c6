"""The division-free place of a save inside its step (f64i_quotient_f32 in
diffrax_gb300/csrc/gbdx_f64i.cuh), compiled for the host: within one rounding
of the long-double quotient, exact at a step's ends."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "diffrax_gb300", "csrc")


@pytest.mark.parametrize("seed", [1, 2])
def test_f64i_quotient(tmp_path, seed):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "f64i_quotient_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                    os.path.join(HERE, "f64i_quotient_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "2000000", str(seed)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
