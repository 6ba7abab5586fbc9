"""The rows that a CTA of the refined Linearized solve stores into the other CTAs of its cluster: the system's own,
each by one CTA, and none past the arrays they go to (the number of 16-row blocks need not be a multiple of the
cluster). On the GPU: sizes where it is not give the same bits every time."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from stormbird_gb300 import Batch, Simulation

from .test_linearized_refined import row

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.join(HERE, "..")
# 16-row blocks 1 to 48, their first and last sizes, and the sizes of the GPU test
SIZES = sorted({n for b in range(1, 49) for n in (16 * b - 15, 16 * b)} | {72, 190, 300, 570, 768})


def test_stored_rows(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "lin_rows_check")
    subprocess.run([nvcc, "-std=c++17", "-x", "cu", "-I", os.path.join(ROOT, "stormbird_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "lin_rows_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    cases = [(n, c) for n in SIZES for c in (1, 2, 4, 8, 16) if c <= (n + 15) // 16]
    out = subprocess.run([exe], input="".join(f"{n} {c}\n" for n, c in cases), text=True, check=True,
                         capture_output=True).stdout.split("\n")
    at = 0
    for n, c in cases:
        padded = (n + 15) // 16 * 16
        room = [int(v) for v in out[at].split()]
        rows = np.concatenate([np.array(out[at + 1 + r].split(), dtype=int) for r in range(c)])
        at += 1 + c
        assert rows.max() < min(room)  # nothing past the residual or the correction
        assert np.array_equal(np.sort(rows), np.arange(padded))  # every row once


@pytest.mark.gpu
@pytest.mark.parametrize("wings,panels", [(1, 72), (2, 95), (3, 100), (6, 95)])
def test_same_bits_every_time(gpu_lib, wings, panels):
    """Alone and in batches whose clusters are halved."""
    setup = row(wings, panels)
    sim = Simulation(setup)
    fs = np.tile([5.0, 8.0, 0.1], (sim.nr_freestream_points, 1))
    first = sim.do_step(time=0.0, time_step=0.1, freestream_velocity=fs).circulation_strength
    for _ in range(1000):
        assert np.array_equal(sim.do_step(time=0.0, time_step=0.1, freestream_velocity=fs).circulation_strength, first)
    for cases in (16, 48):
        b = Batch([setup] * cases)
        all_fs = np.tile(fs, (cases, 1))
        b.do_step(time=0.0, time_step=0.1, freestream_velocity=all_fs)
        g = b.circulation().reshape(cases, -1).copy()
        assert np.array_equal(g, np.tile(g[0], (cases, 1)))
        for _ in range(60):
            b.do_step(time=0.0, time_step=0.1, freestream_velocity=all_fs)
            assert np.array_equal(b.circulation().reshape(cases, -1), g)
