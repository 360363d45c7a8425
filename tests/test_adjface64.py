"""The lean reverse of the FP64 face (phd_adjface64.cuh) against the plain one
(phd_adjoint.cuh: gizmo_pair_adj, temporal_adj, hll_family_adj), compiled for the host with
nvcc, on a million seeded random faces of eight kinds: all 24 adjoints of each face the same to
rounding (both take the forward's branches).  No GPU needed."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_lean_reverse_matches_plain_reverse(tmp_path):
    nvcc = next((c for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc"))
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "adjface64_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "phd-code_gb300", "csrc"), "-x", "cu",
                    os.path.join(HERE, "adjface64_check.cu"), "-o", exe], check=True)
    n, n_open, worst, n_off, median_ulp = subprocess.run([exe, "1000000"], check=True, capture_output=True,
                                                         text=True).stdout.split()
    assert int(n) == 1000000
    assert int(n_open) < 0.1 * int(n)          # vacuum and other extremes: the plain path's
    assert int(n_off) == 0, worst
    assert float(median_ulp) < 10.0
