"""The FP64 path's exact flux (phd_exact64.cuh) and its fixed-point powers (phd_fp64.cuh),
compiled for the host with nvcc: the powers against 80-bit (or wider) arithmetic on two million
seeded bases and exponents of the solver, off by at most 0.51 units of the last place and
rounded the wrong way in fewer than one of a thousand; the flux against the plain one
(exact_flux of phd_physics.cuh) on 500,000 seeded faces of eight kinds, the same convergence
flag and within 1e-12 of the component's scale.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def run(name, tmp_path, n):
    nvcc = next((c for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc"))
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / name)
    subprocess.run([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "phd-code_gb300", "csrc"), "-x", "cu",
                    os.path.join(HERE, name + ".cu"), "-o", exe], check=True)
    return subprocess.run([exe, str(n)], check=True, capture_output=True, text=True).stdout.split()


def test_powers_are_rounded_right(tmp_path):
    n, worst, wrong, of_one, declined = run("pow64_check", tmp_path, 2000000)
    assert float(worst) <= 0.51
    assert int(wrong) < 0.001 * int(n)
    assert int(of_one) == 0
    assert int(declined) < 0.1 * int(n)            # powers beyond 2^900


def test_lean_exact_flux_matches_plain(tmp_path):
    n, n_open, n_flag, worst, n_off = run("exact64_check", tmp_path, 500000)
    assert int(n_open) < 0.03 * int(n)             # vacuum and other extremes: the plain path's
    assert int(n_flag) == 0
    assert int(n_off) == 0, worst
