"""The Linearized solve of one large case, its system built and its results evaluated by all SMs (from 448
lines): sizes around that line and around the four rows of a CTA, the settings that add or leave out a pass,
and the strengths handed to the wake; against the oracle, and against the same case in a batch (one cluster
for all steps).

1e-9, the bound of the Linearized tests: the same formulas in f64, sums in another order.
"""
import numpy as np
import pytest

from stormbird_gb300 import Batch, Simulation

from .helpers import rel_inf
from .test_linearized_refined import check, row, step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wings,panels", [(1, 447), (1, 448), (1, 449), (1, 451), (3, 155), (6, 95), (6, 128)])
def test_sizes(gpu_lib, oracle_mod, wings, panels):
    setup = row(wings, panels)
    g = Simulation(setup)
    a = step(g, [5.0, 8.0, 0.0])
    check(a, step(oracle_mod.OracleSimulation(setup), [5.0, 8.0, 0.0]))
    b = Batch([setup])
    b.do_step(time=0.0, time_step=0.1, freestream_velocity=np.tile([5.0, 8.0, 0.0], (g.nr_freestream_points, 1)))
    assert rel_inf(a.circulation_strength, b.circulation()) <= 1e-9


@pytest.mark.parametrize("solver", [{"Linearized": {"disable_viscous_corrections": True}},
                                    {"Linearized": {"induced_velocity_correction_method": "NoCorrection"}},
                                    {"Linearized": {"velocity_corrections": "FixedMagnitudeEqualToFreestream"}}])
def test_settings(gpu_lib, oracle_mod, solver):
    setup = row(2, 225, solver=solver)
    check(step(Simulation(setup), [5.0, 8.0, 0.0]), step(oracle_mod.OracleSimulation(setup), [5.0, 8.0, 0.0]))


def test_dynamic(gpu_lib, oracle_mod):
    """The FP32 unit matrix (1e-5, the bound of the FP32 sweeps), strengths into the wake's rows."""
    setup = row(4, 113, dynamic=True, rows=4)
    g, o = Simulation(setup), oracle_mod.OracleSimulation(setup)
    for k in range(5):
        a, b = step(g, [5.0, 8.0, 0.0], k), step(o, [5.0, 8.0, 0.0], k)
        assert rel_inf(a.circulation_strength, b.circulation_strength) <= 1e-5
