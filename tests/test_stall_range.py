"""Stall ranges down to 0, where the stall is a step at the stall angle (the sigmoid's slope is infinite), and ranges
so narrow that FP32 cannot tell on which side of the step an angle lies; against the oracle.

Tolerance 1e-9, the bound of the other solver tests: away from the step its sigmoid is 0 or 1 on both sides,
and beside it the angle (1e-15 rad against an offset of 1e-9 and more) leaves no doubt. One iteration from zero
circulation there, so that the angle is the geometric one.
"""
import math

import numpy as np
import pytest

from stormbird_gb300 import Simulation
from stormbird_gb300 import setups as S

from .helpers import fixed_iterations, rel_inf, rel_vec

pytestmark = pytest.mark.gpu
STALL = 0.2


def wing(solver, stall=STALL, stall_range=0.0, viscous_lift=False, **foil):
    f = S.foil(mean_positive_stall_angle=stall, mean_negative_stall_angle=stall, cd_min=0.01, stall_range=stall_range, **foil)
    lfm = S.line_force_model([S.wing_builder([(0, 0, 0), (0, 0, 30.0)], [(10.0, 0, 0)] * 2, f)], 20)
    if viscous_lift:
        lfm["force_calculation_settings"] = {"include_viscous_lift_in_the_circulation": True}
    return S.simulation(lfm, False, solver, {"viscous_core_length": {"Absolute": 0.5}})


def check(oracle_mod, setup, angle):
    g, o = Simulation(setup), oracle_mod.OracleSimulation(setup)
    fs = np.tile([10.0 * math.cos(angle), 10.0 * math.sin(angle), 0.0], (g.nr_freestream_points, 1))
    for k in range(2):
        rg = g.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs)
        ro = o.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs)
        assert np.all(np.isfinite(ro.circulation_strength))
        assert rel_inf(rg.circulation_strength, ro.circulation_strength) <= 1e-9
        assert rel_vec(rg.integrated_forces_sum(), ro.integrated_forces_sum()) <= 1e-9
        assert abs(rg.residual - ro.residual) <= 1e-9 * max(1.0, ro.residual)


@pytest.mark.parametrize("stall_range", [0.0, 1e-300, 1e-40, 1e-36, 1e-30, 1e-12])
@pytest.mark.parametrize("angle", [0.05, -0.05, 0.6, -0.6])
@pytest.mark.parametrize("kind", ["iterative", "viscous_lift", "linearized", "offset"])
def test_step(gpu_lib, oracle_mod, kind, angle, stall_range):
    if kind == "linearized":
        check(oracle_mod, wing({"Linearized": {}}, stall_range=stall_range), angle)
        return
    foil = {"cd_stall_angle_offset": 0.1} if kind == "offset" else {}
    setup = wing(S.simple_iterative(10, 0.02, 0.0, 0.0), stall_range=stall_range, viscous_lift=kind == "viscous_lift", **foil)
    check(oracle_mod, fixed_iterations(setup, 10), angle)


@pytest.mark.parametrize("stall_range", [0.0, 1e-12, 1e-10])
@pytest.mark.parametrize("offset", [1e-9, -1e-9, 4e-9, -4e-9, 3e-8, -3e-8])
def test_beside_the_step(gpu_lib, oracle_mod, offset, stall_range):
    """A stall angle just above or below the angle of attack of every line, at angles spread over FP32's rounding."""
    for angle in np.linspace(0.1, 0.3, 24):
        setup = wing(S.simple_iterative(1, 0.02, 0.0, 0.0), stall=angle + offset, stall_range=stall_range)
        g, o = Simulation(fixed_iterations(setup, 1)), oracle_mod.OracleSimulation(fixed_iterations(setup, 1))
        fs = np.tile([10.0 * math.cos(angle), 10.0 * math.sin(angle), 0.0], (g.nr_freestream_points, 1))
        rg = g.do_step(time=0.0, time_step=0.1, freestream_velocity=fs)
        ro = o.do_step(time=0.0, time_step=0.1, freestream_velocity=fs)
        # 1e-9 of the unstalled strength's scale, chord x speed
        assert np.max(np.abs(rg.circulation_strength - ro.circulation_strength)) <= 1e-9 * 100.0
