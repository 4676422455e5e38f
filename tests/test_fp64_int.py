"""The integer forms of FP64 operations (csrc/fp64_int.cuh) against the host's
own arithmetic, bit for bit: any bit patterns, ties, cancellation, subnormals,
zeros, infinities and NaN."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_integer_fp64_has_the_bits_of_the_plain_operation(tmp_path):
    exe = tmp_path / "fp64_int_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "implicit_dpd_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fp64_int_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
