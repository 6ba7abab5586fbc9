"""Geometry and forces at the edges of their blocks (62 lines a geometry block, a CTA per wing with 256
threads), with motion, coordinate systems and section models, against the oracle: every array of the
result.

The circulation comes from one iteration without induced velocities (a start scaled by 0), so that no
influence matrix and its rounding at fine panels takes part. Tolerance 1e-9 of each array's largest
value, far above f64 rounding and far below any wrong line; the accelerations are differences of
velocities over the time step (times 30 here): 1e-7.
"""
import math

import numpy as np
import pytest

from stormbird_gb300 import Simulation
from stormbird_gb300 import setups as S

from .helpers import rel_inf

pytestmark = pytest.mark.gpu


def setup(panels, foil=None, output="Global", rotation=(0.0, 0.0, 0.0), viscous=False):
    f = S.foil(**(foil or {}))
    wings = []
    for i, n in enumerate(panels):
        w = S.wing_builder([(40.0 * i, 0, 0), (40.0 * i + 2, 0.5, 12.0), (40.0 * i, 0, 30.0)],
                           [(10, 0, 0), (8, 0, 0), (5, 0, 0)], f, nr_sections=n)
        wings.append(w)
    lfm = S.line_force_model(wings, 8, local_wing_angles=[0.2 + 0.1 * i for i in range(len(panels))],
                             output_coordinate_system=output, rotation=rotation, translation=(1.0, 2.0, -0.5))
    if viscous:
        lfm["force_calculation_settings"] = {"include_viscous_lift_in_the_circulation": True}
    return S.simulation(lfm, False, S.simple_iterative(1, 0.1, 0.0, 0.0, correction_factor_initial_solution=0.0))


def arrays(r):
    out = {"circulation": r.circulation_strength, "aoa": r.force_input.angles_of_attack, "velocity": r.force_input.velocity,
           "input": r.solver_input_ctrl_points_velocity, "points": r.ctrl_points,
           "force": r.integrated_forces_sum(), "moment": r.integrated_moments_sum()}
    for part in ("circulatory", "viscous_lift", "sectional_drag", "added_mass", "gyroscopic", "total"):
        out["section " + part] = getattr(r.sectional_forces, part)
        out["force " + part] = np.stack([getattr(w, part) for w in r.integrated_forces])
        out["moment " + part] = np.stack([getattr(w, part) for w in r.integrated_moments])
    return out


def check(oracle_mod, js, u):
    g, o = Simulation(js), oracle_mod.OracleSimulation(js)
    rng = np.random.default_rng(2)
    for k in range(4):
        for s in (g, o):
            s.set_translation_and_rotation_with_finite_difference_for_the_velocity(
                0.1, [1.0 + 0.2 * k, 2.0, 0.1 * k], [0.02 * k, -0.01 * k, 0.03 * k])
        fs = np.tile(u, (g.nr_freestream_points, 1)) + rng.normal(0, 0.2, (g.nr_freestream_points, 3)) * [1.0, 1.0, 0.0]
        a = g.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs)
        b = o.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs)
        x, y = arrays(a), arrays(b)
        for name in x:
            assert rel_inf(x[name], y[name]) <= (1e-7 if "added" in name else 1e-9), (k, name)
        assert rel_inf(a.force_input.acceleration, b.force_input.acceleration) <= 1e-7


@pytest.mark.parametrize("panels", [(3,), (61,), (62,), (63,), (124,), (125,), (30, 31, 5), (40, 22, 70), (300,)])
def test_sizes(gpu_lib, oracle_mod, panels):
    check(oracle_mod, setup(panels), [9.0, 4.0, 0.0])


@pytest.mark.parametrize("case", ["body", "drag", "bump", "offset", "power", "added_mass", "viscous", "stalled", "reversed"])
def test_options(gpu_lib, oracle_mod, case):
    stall = dict(mean_positive_stall_angle=math.radians(15), mean_negative_stall_angle=math.radians(12))
    kw, u = {}, [9.0, 4.0, 0.0]
    if case == "body":
        kw = dict(output="Body", rotation=(0.1, -0.05, 0.2))
    elif case == "drag":
        kw = dict(foil=dict(stall, cd_min=0.01, cd_second_order_factor=0.3, angle_cd_min=0.02, cdi_correction_factor=0.05))
    elif case == "bump":
        kw = dict(foil=dict(stall, cd_bump_during_stall=0.2))
    elif case == "offset":
        kw = dict(foil=dict(stall, cd_stall_angle_offset=-0.05))
    elif case == "power":
        kw = dict(foil=dict(stall, cd_power_after_stall=2.5, cd_max_after_stall=1.8))
    elif case == "added_mass":
        kw = dict(foil=dict(stall, added_mass_factor=0.9))
    elif case == "viscous":
        kw = dict(foil=stall, viscous=True)
    elif case == "stalled":
        kw, u = dict(foil=stall), [2.0, 9.0, 0.0]
    elif case == "reversed":
        kw, u = dict(foil=stall), [-9.0, -3.0, 0.0]
    check(oracle_mod, setup((9, 14), **kw), u)
