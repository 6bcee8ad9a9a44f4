"""The stretch of the 3-D bond kernels and the state-based passes
(pd_gpu1_gb300/csrc/bondtpl.h), compiled for the host and held to quadruple
precision from bond vectors of one subtraction a component."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_stretch_against_quad_precision(tmp_path):
    exe = tmp_path / "stretch_check"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "pd_gpu1_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "stretch_check.cpp"), "-o", str(exe), "-lquadmath"],
                       capture_output=True, text=True)
    if r.returncode != 0 and "quadmath" in (r.stderr + r.stdout):
        pytest.skip("no libquadmath on this host")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
