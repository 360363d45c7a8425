"""The FP64 kernels' quotients and square roots come from FP32 / integer seeds and
integer remainders (phd_fp64.cuh).  Against CUDA's IEEE operations: bit for bit equal on
15.5M pairs of each of six kinds, hard cases next to rounding boundaries among them; every
operand outside the window (zeros, infinities, NaN, subnormals, negative radicands)
declined."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_quotient_and_root_are_ieee(tmp_path):
    nvcc = next((c for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc"))
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "fp64_ieee_check")
    subprocess.run([nvcc, "-O3", "-std=c++17", "--fmad=false", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "phd-code_gb300", "csrc"),
                    os.path.join(HERE, "fp64_ieee_check.cu"), "-o", exe], check=True)
    lines = subprocess.run([exe, "100"], check=True, capture_output=True, text=True).stdout.splitlines()
    for mode, line in enumerate(lines[:6]):
        n, div_bad, div_declined, root_bad, root_declined, seed_off = map(int, line.split())
        assert (div_bad, root_bad, seed_off) == (0, 0, 0), (mode, line)
        if mode:
            assert (div_declined, root_declined) == (0, 0), (mode, line)
        else:                                   # 1,000 and 800 of 2,046 exponents are in the windows
            assert 0.7 * n < div_declined < 0.9 * n and 0.5 * n < root_declined < 0.7 * n
    assert int(lines[6]) == 0
