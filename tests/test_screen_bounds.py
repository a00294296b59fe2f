"""The bounds that rule starts out of the chi2 minimum, checked on the CPU.

The bounding arithmetic (gtls_b200/csrc/screen.cuh) builds for the host as
well; tests/csrc/screen_bounds.cu compares it with 64-bit sums over every
window, for widths at the edges of its tables, on exact and coarse prefix
values.
"""
import os
import subprocess

import pytest

from conftest import ROOT

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def test_bounds_enclose_the_exact_value_of_every_start(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "screen_bounds")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                    "-I", os.path.join(ROOT, "gtls_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "csrc", "screen_bounds.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("ok "), r.stdout
