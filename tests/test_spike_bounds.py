"""The bounds of starts whose curve has spikes, checked on the CPU: the
arithmetic that leaves a few samples out of the prefix sums and adds them to the
windows that hold them (gtls_b200/csrc/screen.cuh) against 64-bit sums, and the
rounding of prefix sums that are accumulated in FP64 and rounded once."""
import os
import subprocess

import pytest

from conftest import ROOT

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def test_bounds_enclose_the_exact_value_with_spikes(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "spike_bounds")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                    "-I", os.path.join(ROOT, "gtls_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "csrc", "spike_bounds.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("ok "), r.stdout
