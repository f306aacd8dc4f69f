"""
The FP64 kernels take most of their products on the integer pipes
(fsg_soft.cuh).  Each product must have the bits of the double product it
stands for wherever it says so, and the escape and stationarity thresholds
read from the exponents must agree with the double comparisons: the device
header is compiled for the host and checked on random and special operands.
"""
import os
import shutil
import subprocess

import pytest

from test_num_bits import HERE, _cuda_include


@pytest.mark.parametrize("opt", ["-O0", "-O2"])
def test_integer_products_match_double_products(tmp_path, opt):
    cxx = shutil.which("g++")
    inc = _cuda_include()
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path / "soft_mul_check")
    src = os.path.join(HERE, "native", "soft_mul_check.cpp")
    r = subprocess.run([cxx, opt, "-ffp-contract=off", "-std=c++17", "-I", inc, src, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe, "2000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert " 0 mismatches" in r.stdout
