"""The SimpleIterative solve's cluster sizes and its per-line arithmetic at the edges of their
ranges, against the oracle (a fixed number of iterations, so that a difference is the arithmetic's).

Tolerance 1e-9 (circulation and total force): the double-float matrix-vector product carries about
2^-44 per product, grown by at most the iterations' own condition (the f64 tests of this solver use
the same bound). The lift near a stall angle 1e-4 deg wide is as steep as 4e6 per radian, so that
case asks for 1e-5 (1e-9 of angle and velocity times 4e4, the slope times the lift's own scale).
"""
import json
import math

import numpy as np
import pytest

from stormbird_gb300 import Simulation
from stormbird_gb300 import setups as S

from .helpers import fixed_iterations, rel_inf, rel_vec

pytestmark = pytest.mark.gpu


def quasi_steady(panels=24, foil=None, points=None, chord=(10.0, 0.0, 0.0), wings=1, output="Global", rotation=(0, 0, 0),
                 iterations=12, viscous_lift=False, correction=None):
    f = S.foil(**(foil or dict(mean_positive_stall_angle=math.radians(15), mean_negative_stall_angle=math.radians(15),
                               cd_min=0.01)))
    w = [S.wing_builder([(40.0 * i + p[0], p[1], p[2]) for p in points or [(0, 0, 0), (0, 0, 30.0)]], [chord, chord], f)
         for i in range(wings)]
    lfm = S.line_force_model(w, panels, output_coordinate_system=output, rotation=rotation)
    if viscous_lift:
        lfm["force_calculation_settings"] = {"include_viscous_lift_in_the_circulation": True}
    extra = {"velocity_corrections": correction} if correction else {}
    # damping and core as fine panels need them for the iteration to contract (else it grows any rounding)
    wake = {"viscous_core_length": {"Absolute": 0.5}}
    return fixed_iterations(S.simulation(lfm, False, S.simple_iterative(iterations, 0.02, 0.0, 0.0, **extra), wake), iterations)


def check(oracle_mod, setup, u, tol=1e-9):
    g, o = Simulation(setup), oracle_mod.OracleSimulation(setup)
    fs = np.tile(u, (g.nr_freestream_points, 1))
    for k in range(2):
        rg = g.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs)
        ro = o.do_step(time=0.1 * k, time_step=0.1, freestream_velocity=fs)
        assert rg.iterations == ro.iterations
        assert rel_inf(rg.circulation_strength, ro.circulation_strength) <= tol
        assert rel_vec(rg.integrated_forces_sum(), ro.integrated_forces_sum()) <= tol


def wind(deg, speed=10.0):
    return speed * np.array([math.cos(math.radians(deg)), math.sin(math.radians(deg)), 0.0])


# clusters of 1, 8 and 16 CTAs: one row, the ends of each range, a cluster whose last CTA has no
# rows (129 lines: 9 to a CTA), a second pass over a CTA's rows, a matrix that no longer fits
# shared memory and is streamed (16 rows at a time, and with a remainder)
@pytest.mark.parametrize("panels", [1, 2, 3, 47, 48, 49, 129, 160, 161, 271, 420, 701])
def test_cluster_sizes(gpu_lib, oracle_mod, panels):
    check(oracle_mod, quasi_steady(panels, iterations=8), wind(8.0))


def test_four_rows_per_thread(gpu_lib, oracle_mod):
    """4,200 lines: more than 256 a CTA in the largest cluster; matrix rows from global memory."""
    check(oracle_mod, quasi_steady(4200, iterations=3), wind(8.0))


@pytest.mark.parametrize("deg", [-160.0, -60.0, -15.0, -3.0, 0.0, 0.5, 15.0, 40.0, 90.0, 135.0, 179.0, 180.0])
def test_angles(gpu_lib, oracle_mod, deg):
    check(oracle_mod, quasi_steady(), wind(deg))


@pytest.mark.parametrize("case", ["swept", "swept_rotated", "along_span", "no_chord", "viscous_lift", "uneven_stall",
                                  "cd_angle", "high_order", "narrow_stall", "body", "max_induced", "fixed_magnitude",
                                  "no_wind", "slow", "fast", "two_wings"])
def test_lines(gpu_lib, oracle_mod, case):
    stall = dict(mean_positive_stall_angle=math.radians(15), mean_negative_stall_angle=math.radians(15))
    kw, u, tol = {}, wind(9.0), 1e-9
    if case == "swept":
        kw = dict(points=[(0, 0, 0), (6.0, 1.0, 30.0)])
    elif case == "swept_rotated":
        kw = dict(points=[(0, 0, 0), (6.0, 1.0, 30.0)], rotation=(0.1, -0.2, 0.3))
    elif case == "along_span":
        kw = dict(chord=(0.0, 0.0, 10.0))
    elif case == "no_chord":
        kw = dict(chord=(0.0, 0.0, 0.0))
    elif case == "viscous_lift":
        kw, u = dict(viscous_lift=True), wind(25.0)
    elif case == "uneven_stall":
        kw, u = dict(foil=dict(mean_positive_stall_angle=0.2, mean_negative_stall_angle=0.3, cl_zero_angle=0.3)), wind(0.0)
    elif case == "cd_angle":
        kw = dict(foil=dict(stall, angle_cd_min=-0.15, cl_zero_angle=-0.2))
    elif case == "high_order":
        kw = dict(foil=dict(stall, cl_high_order_factor_positive=-0.4, cl_high_order_factor_negative=0.3,
                            cl_high_order_power=2.0))
    elif case == "narrow_stall":
        kw, tol = dict(foil=dict(stall, stall_range=math.radians(1e-4))), 1e-5
    elif case == "body":
        kw = dict(output="Body", rotation=(0.1, 0.2, -0.3))
    elif case == "max_induced":
        kw = dict(correction={"MaxInducedVelocityMagnitudeRatio": 0.02})
    elif case == "fixed_magnitude":
        kw = dict(correction="FixedMagnitudeEqualToFreestream")
    elif case == "no_wind":
        u = np.zeros(3)
    elif case == "slow":
        u = wind(9.0, 1e-20)
    elif case == "fast":
        u = wind(9.0, 1e20)
    elif case == "two_wings":
        kw = dict(wings=2, panels=33)
    check(oracle_mod, quasi_steady(**kw), u, tol)


def test_strength_tolerance_stops_as_the_oracle(gpu_lib, oracle_mod):
    """The largest |dGamma| decides, across the CTAs of a cluster and in one."""
    for panels in (24, 60, 200):
        d = json.loads(quasi_steady(panels))
        s = d["simulation_settings"]["QuasiSteady"]["solver"]["SimpleIterative"]
        s["max_iterations_per_time_step"], s["strength_difference_tolerance"] = 2000, 0.5
        setup = json.dumps(d)
        g, o = Simulation(setup), oracle_mod.OracleSimulation(setup)
        fs = np.tile(wind(8.0), (g.nr_freestream_points, 1))
        rg = g.do_step(time=0.0, time_step=0.1, freestream_velocity=fs)
        ro = o.do_step(time=0.0, time_step=0.1, freestream_velocity=fs)
        assert 1 < ro.iterations < 2000 and rg.iterations == ro.iterations and rg.converged == ro.converged
        assert rel_inf(rg.circulation_strength, ro.circulation_strength) <= 1e-9
