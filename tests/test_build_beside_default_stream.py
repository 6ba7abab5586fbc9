"""Simulations, batches and networks built and used while another thread keeps the default stream busy: their first
results are those of an idle GPU, bit for bit (what a handle zeroes at its start is zeroed on its own stream)."""
import threading

import numpy as np
import pytest

from stormbird_gb300 import Batch, Simulation
from stormbird_gb300 import setups as S

pytestmark = pytest.mark.gpu
SETUP = S.wing_sail_row(2, 24, 20, wind_speed=9.0, apparent_wind_angle_deg=50.0)


def steps():
    sim = Simulation(SETUP)
    fs = np.tile([7.0, 5.0, 0.0], (sim.nr_freestream_points, 1))
    out = [sim.do_step(time=0.05 * k, time_step=0.05, freestream_velocity=fs) for k in range(3)]
    b = Batch([SETUP] * 3)
    for k in range(3):
        b.do_step(time=0.05 * k, time_step=0.05, freestream_velocity=np.tile(fs, (3, 1)))
    return np.concatenate([r.circulation_strength for r in out] + [r.integrated_forces_sum() for r in out] + [b.circulation()])


def test_busy_default_stream(gpu_lib):
    torch = pytest.importorskip("torch")
    want = steps()
    stop = threading.Event()

    def busy():
        while not stop.is_set():
            torch.cuda._sleep(2_000_000)  # about 1 ms of the default stream
            torch.cuda.current_stream().synchronize()

    other = threading.Thread(target=busy)
    other.start()
    try:
        for _ in range(10):
            assert np.array_equal(steps(), want)
    finally:
        stop.set()
        other.join()
