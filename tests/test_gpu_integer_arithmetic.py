"""The FP64 products, reciprocals, square roots and sums that the kernels take
on the integer pipes (tests/integer_check.cu): mul_rn_alu, rcp_rn_alu and
add_alu give the FP64 unit's bits; mul_alu is as close to the exact product as
a rounding to nearest; rcp_alu and sqrt_alu stay within the 0.5001 and 0.52
ulp that their series leave with an FP32 seed two ulps off.  8M operand pairs:
binade edges, ties, exponent gaps up to 34, odd and even exponents, the ends
of the magnitudes they take, special values."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "benchmark-euler-kernels_gb300", "csrc")


@pytest.mark.gpu
def test_integer_arithmetic(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "integer_check"
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC,
                    os.path.join(ROOT, "tests", "integer_check.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    r = json.loads(out.strip().splitlines()[-1])
    assert r["n"] > 8_000_000
    assert all(r[k] == 0 for k in ("mul_rn", "rcp_rn", "add", "mul", "rcp_outside", "sqrt_outside")), r
    assert r["rcp_ulps"] <= 0.5001 and r["sqrt_ulps"] <= 0.52, r
