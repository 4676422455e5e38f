"""The integer product by a factor (mul_f64, csrc/fp64_int.cuh) has the bits of
the plain one also for factors outside the normal range."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_products_by_any_factor(tmp_path):
    exe = tmp_path / "mul_factor_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "implicit_dpd_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "mul_factor_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
