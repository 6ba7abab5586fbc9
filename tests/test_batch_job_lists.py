"""A batch's launches over lists of cases (wind, geometry, core lengths, horseshoe matrices) against the
same cases stepped alone: uneven quasi-steady cases at the edges of the geometry's 62-line blocks and the
horseshoe matrix's 127-point tiles, every core kind, symmetry, beside dynamic ones; gusts and inflow
corrections; first steps, and replayed graphs with the wind of the new step.

The list kernels run the single case's functions, so all that differs is the split of a solve's sums over
CTAs: 1e-9 of the largest value, the bound of the solves elsewhere.
"""
import json

import numpy as np
import pytest

from stormbird_gb300 import Simulation
from stormbird_gb300 import setups as S
from stormbird_gb300.batch import Batch

from . import wind_cases as W
from .helpers import rel_inf, small_row

pytestmark = pytest.mark.gpu


def _quasi_steady(sails, panels, core, symmetry="NoSymmetry", solver=None):
    d = json.loads(S.wing_sail_row(sails, panels, 1, apparent_wind_angle_deg=60.0))
    return S.simulation(d["line_force_model"], False, solver, {"viscous_core_length": core, "symmetry_condition": symmetry})


def _cases(with_dynamic):
    out = [_quasi_steady(1, 2, {"Relative": 0.1}, "Z"), _quasi_steady(2, 31, {"Absolute": 0.05}),
           _quasi_steady(1, 63, "NoViscousCore"), _quasi_steady(1, 127, {"Relative": 0.1}),
           _quasi_steady(3, 43, {"Relative": 0.05}, "Z"),
           _quasi_steady(2, 5, {"Relative": 0.1}, solver=S.simple_iterative(max_iterations=30))]
    if with_dynamic:
        out[3:3] = [small_row(2, 6, 5), small_row(1, 9, 4)]
    return out


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("with_dynamic", [False, True])
def test_lists_match_single_cases(gpu_lib, with_dynamic, graph):
    cases = _cases(with_dynamic)
    env = W.environment(inflow_corrections=True, nr_wings=3)
    conds = [W.condition(30.0 + 7.0 * i, ("power", "log", "constant")[i % 3], gusts=i % 2 == 0) for i in range(len(cases))]
    b = Batch(cases)
    b.use_graph(graph)
    sims = [Simulation(c) for c in cases]
    b.set_wind(env, conds)
    for s, c in zip(sims, conds):
        s.set_wind(env, c)
    for k in range(8):
        if k == 6:  # another wind in mid-run
            conds = conds[::-1]
            b.set_wind(env, conds)
            for s, c in zip(sims, conds):
                s.set_wind(env, c)
        ships = [1.0 + 0.2 * i + 0.1 * k for i in range(len(cases))]
        b.do_step_wind(time=0.2 * k, time_step=0.2, ship_velocities=ships)
        circ = b.circulation()
        for i, s in enumerate(sims):
            r = s.do_step_wind(time=0.2 * k, time_step=0.2, ship_velocity=ships[i])
            assert rel_inf(circ[b.case_slice(i)], r.circulation_strength) <= 1e-9, (k, i)
            f = b.read_case_output(i).integrated_forces_sum()
            assert rel_inf(f, r.integrated_forces_sum()) <= 1e-9, (k, i)
