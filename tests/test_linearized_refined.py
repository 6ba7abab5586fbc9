"""The Linearized solve by an FP32 inverse and f64 refinement, at the edges of its blocks (16 rows) and
clusters, and what it leaves to the elimination, against the oracle.

Tolerance 1e-9, the bound of the other Linearized tests: the refinement stops at a correction of
2^-50 of the solution or at the rounding of an f64 residual, as far from the exact solution as an
f64 elimination.
"""
import json

import numpy as np
import pytest

from stormbird_gb300 import Batch, SbError, Simulation
from stormbird_gb300 import setups as S

from .helpers import rel_inf, rel_vec

pytestmark = pytest.mark.gpu


def row(wings, panels, dynamic=False, rows=12, solver=None, **wake):
    d = json.loads(S.wing_sail_row(wings, panels, rows, apparent_wind_angle_deg=60.0))
    if dynamic:
        d["simulation_settings"]["Dynamic"]["solver"] = solver or {"Linearized": {}}
        return json.dumps(d)
    return S.simulation(d["line_force_model"], False, solver, wake or None)


def step(sim, u, k=0):
    return sim.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=np.tile(u, (sim.nr_freestream_points, 1)))


def check(a, b, tol=1e-9):
    assert rel_inf(a.circulation_strength, b.circulation_strength) <= tol
    assert rel_vec(a.integrated_forces_sum(), b.integrated_forces_sum()) <= tol
    assert abs(a.residual - b.residual) <= tol * max(1.0, abs(b.residual))


# blocks of 16 rows on clusters of 1, 2, 4, 8, 16; 768 lines are the most that fit, 769 are eliminated
@pytest.mark.parametrize("panels", [1, 2, 15, 16, 17, 32, 33, 63, 65, 127, 129, 256, 257, 272, 768, 769])
def test_sizes(gpu_lib, oracle_mod, panels):
    setup = row(1, panels)
    check(step(Simulation(setup), [5.0, 8.0, 0.0]), step(oracle_mod.OracleSimulation(setup), [5.0, 8.0, 0.0]))


@pytest.mark.parametrize("solver", [{"Linearized": {"disable_viscous_corrections": True}},
                                    {"Linearized": {"induced_velocity_correction_method": "NoCorrection"}},
                                    {"Linearized": {"velocity_corrections": "FixedMagnitudeEqualToFreestream"}},
                                    {"Linearized": {"velocity_corrections": {"MaxInducedVelocityMagnitudeRatio": 0.05}}}])
def test_settings(gpu_lib, oracle_mod, solver):
    setup = row(2, 20, solver=solver)
    check(step(Simulation(setup), [5.0, 8.0, 0.1]), step(oracle_mod.OracleSimulation(setup), [5.0, 8.0, 0.1]))


def test_dynamic(gpu_lib, oracle_mod):
    """The unit matrix in FP32 (1e-5, the bound of the FP32 sweeps), strengths into the wake."""
    setup = row(2, 12, dynamic=True)
    g, o = Simulation(setup), oracle_mod.OracleSimulation(setup)
    for k in range(6):
        a, b = step(g, [5.0, 8.0, 0.0], k), step(o, [5.0, 8.0, 0.0], k)
        assert rel_inf(a.circulation_strength, b.circulation_strength) <= 1e-5


def test_what_it_leaves(gpu_lib, oracle_mod):
    """A matrix scaled below the pivot the reference calls singular is refused as before; a system too
    ill-conditioned for an FP32 inverse (a core wider than a panel) is eliminated: two f64
    eliminations of it agree to about 1e-5."""
    with pytest.raises(SbError):
        step(Simulation(row(1, 20)), [1e14, 1e13, 0.0])
    setup = row(1, 126, viscous_core_length={"Absolute": 0.4})
    a, b = step(Simulation(setup), [5.0, 8.0, 0.1]), step(oracle_mod.OracleSimulation(setup), [5.0, 8.0, 0.1])
    assert rel_inf(a.circulation_strength, b.circulation_strength) <= 1e-4
    # without wind the reference divides by zero: no number, and no error
    assert not np.any(np.isfinite(step(Simulation(row(1, 20)), [0.0, 0.0, 0.0]).circulation_strength))


def test_batch_of_uneven_systems(gpu_lib):
    """Clusters halved until all run side by side: the same solutions as each alone (another order of
    the FP32 inverse, the same refinement)."""
    sizes = [(1, 3), (1, 16), (2, 24), (3, 50), (4, 64), (6, 95), (1, 40)] * 4
    b = Batch([row(*s) for s in sizes])
    u = np.array([5.0, 8.0, 0.1])
    b.do_step(time=0.0, time_step=0.1, freestream_velocity=np.tile(u, (b.total_freestream, 1)))
    g = b.circulation()
    for i, s in enumerate(sizes[:7]):
        alone = step(Simulation(row(*s)), u).circulation_strength
        for k in range(i, len(sizes), 7):
            assert rel_inf(g[b.case_slice(k)], alone) <= 1e-10
