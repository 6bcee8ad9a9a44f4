"""The offset of a bond vector from its class with the class's scale
(pd_gpu1_gb300/csrc/bondtpl.h, offset_class), compiled for the host and held
bit for bit to the general form."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_offset_class_equals_offset_pair(tmp_path):
    exe = tmp_path / "offset_class_check"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "pd_gpu1_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "offset_class_check.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
