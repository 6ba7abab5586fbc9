"""A buffer whose allocation failed is empty: neither its size nor a later request for as much passes for memory
that is not there (a kernel would write through a null pointer)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.join(HERE, "..")


def test_failed_allocation(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "alloc_state_check")
    subprocess.run([nvcc, "-std=c++17", "-x", "cu", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "stormbird_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "alloc_state_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], text=True, check=True, capture_output=True).stdout.split("\n")[:4]
    assert out == [f"{name} 1 0 0" for name in ("device", "device", "pinned", "pinned")]
