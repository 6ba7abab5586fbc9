"""launch_mlp_gemm refuses a call without an array that its mode reads or writes (the epilogue stores through
them unconditionally; only the transposed output may be left out)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.join(HERE, "..")
NEEDS = {0: {"A", "B", "bias", "z_out", "h_out"}, 1: {"A", "B", "h_out", "z_in"}, 2: {"A", "B", "part_out"}}


def test_arrays_of_each_mode(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "mlp_args_check")
    subprocess.run([nvcc, "-std=c++17", "-x", "cu", "-I", os.path.join(ROOT, "stormbird_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "mlp_args_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    lines = subprocess.run([exe], text=True, check=True, capture_output=True).stdout.split("\n")
    seen = [line.split() for line in lines if line]
    assert len(seen) == 27
    for mode, left_out, accepted in seen:
        assert (accepted == "1") == (left_out not in NEEDS[int(mode)]), (mode, left_out)
