"""No wind, or wind along the spans: nothing flows past the lines in their planes. What the solvers and the forces make of
that, against the oracle: zeros are zeros (circulation, angles, forces, residual) and no numbers are no numbers."""
import json

import numpy as np
import pytest

from stormbird_gb300 import Batch, Simulation
from stormbird_gb300 import setups as S

pytestmark = pytest.mark.gpu


def setup(solver, panels=17, dynamic=False):
    d = json.loads(S.wing_sail_row(2, panels, 6, apparent_wind_angle_deg=40.0))
    return S.simulation(d["line_force_model"], dynamic, solver, S.dynamic_wake(6) if dynamic else None)


def outputs(r):
    s = r.sectional_forces
    return {"circulation": r.circulation_strength, "velocity": r.force_input.velocity, "angles": r.force_input.angles_of_attack,
            "circulatory": s.circulatory, "viscous": s.viscous_lift, "drag": s.sectional_drag, "total": s.total,
            "added": s.added_mass, "force": r.force_sum, "moment": r.moment_sum, "residual": np.array([r.residual])}


@pytest.mark.parametrize("wind", [(0.0, 0.0, 0.0), (0.0, 0.0, 5.0)])
@pytest.mark.parametrize("dynamic", [False, True])
@pytest.mark.parametrize("panels", [1, 17, 100])
def test_iterations(gpu_lib, oracle_mod, panels, dynamic, wind):
    js = setup(S.simple_iterative(5, 0.05, 0.0, 0.0), panels, dynamic)
    g, o = Simulation(js), oracle_mod.OracleSimulation(js)
    for k in range(3):
        fs = np.tile(wind, (g.nr_freestream_points, 1))
        a = outputs(g.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs))
        b = outputs(o.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs))
        for name in a:
            assert np.array_equal(a[name], b[name]), name
            assert not np.any(a[name]), name


def test_batch(gpu_lib):
    js = setup(S.simple_iterative(5, 0.05, 0.0, 0.0))
    b = Batch([js] * 3)
    for k in range(5):
        b.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=np.zeros((3 * 34, 3)))
        assert not np.any(b.circulation()) and not np.any(b.summary()[:, :7])


@pytest.mark.parametrize("wind", [(0.0, 0.0, 0.0), (0.0, 0.0, 5.0)])
@pytest.mark.parametrize("panels", [17, 100, 240])
def test_linearized(gpu_lib, oracle_mod, panels, wind):
    """Without wind in its plane a line has no Linearized solution: no number in all that follows from it, the drag
    included, and no error (which rounding beside the 0 would give: a singular matrix)."""
    js = setup(None, panels)
    g, o = Simulation(js), oracle_mod.OracleSimulation(js)
    for _ in range(3):  # accelerations from the third step
        fs = np.tile(wind, (g.nr_freestream_points, 1))
        a = outputs(g.do_step(time=0.0, time_step=0.1, freestream_velocity=fs))
        b = outputs(o.do_step(time=0.0, time_step=0.1, freestream_velocity=fs))
        for name in a:
            assert np.array_equal(a[name], b[name], equal_nan=True), name


def test_no_time(gpu_lib, oracle_mod):
    """Steps of no length have no acceleration: no added mass, not even of a foil without one."""
    js = setup(S.simple_iterative(5, 0.05, 0.0, 0.0))
    g, o = Simulation(js), oracle_mod.OracleSimulation(js)
    for k in range(4):
        fs = np.tile([8.0 + 0.3 * k * k, 5.0, 0.0], (g.nr_freestream_points, 1))
        a = outputs(g.do_step(time=0.0, time_step=0.0, freestream_velocity=fs))
        b = outputs(o.do_step(time=0.0, time_step=0.0, freestream_velocity=fs))
        for name in ("added", "total", "force"):
            assert np.array_equal(np.isnan(a[name]), np.isnan(b[name])), name
    assert np.all(np.isnan(b["added"]))
