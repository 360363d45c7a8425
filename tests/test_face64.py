"""The lean FP64 face (phd_face64.cuh: states64, hll64) against the plain one
(face_spatial_f64, temporal, hll_family), compiled for the host with nvcc: every state and
flux equal on seeded random faces of eight kinds (equal cells up to the last bits, smooth
flow, simple waves, jumps, strong rarefactions, sign changes, supersonic), HLL and HLLC, with
and without boost, GIZMO limiter and slopes.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_lean_face_equals_plain_face(tmp_path):
    nvcc = next((c for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc"))
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "face64_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "phd-code_gb300", "csrc"), "-x", "cu",
                    os.path.join(HERE, "face64_check.cu"), "-o", exe], check=True)
    n, n_open, n_diff = map(int, subprocess.run([exe, "1000000"], check=True, capture_output=True,
                                                text=True).stdout.split())
    assert n == 1000000
    assert n_open < 0.03 * n          # vacuum and other extremes: the plain path's
    assert n_diff == 0
