"""The FP64 vortex elements at the edges of their formulas and the horseshoe matrix at the edges of its
tiles, against the oracle.

Sweep tolerance 1e-12 of the largest velocity: each f64 evaluation is good to a few 2^-53 times the
cancellation of r1.r2 against l1 l2 that both sides share (den above 1e-10 at distances of metres: at
most 1e3 of rounding). Solves: 1e-9, the bound of the other Linearized tests.
"""
import json

import numpy as np
import pytest

from stormbird_gb300 import Simulation
from stormbird_gb300 import setups as S
from stormbird_gb300.simulation import panel_sweep

from .helpers import rel_inf, rel_vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("symmetry", ["NoSymmetry", "Z"])
@pytest.mark.parametrize("core", [{"Relative": 0.1}, {"Absolute": 0.01}, "NoViscousCore"])
@pytest.mark.parametrize("wings,panels", [(1, 2), (1, 126), (1, 127), (2, 63), (3, 42), (2, 127)])
def test_horseshoe_tiles(gpu_lib, oracle_mod, wings, panels, core, symmetry):
    """128 span points to a block, the last of them only for its neighbour: one block exactly, one
    point more, wings that end inside and at the edge of one. (Cores below a panel's width: a wider
    one makes the system so ill-conditioned that any two roundings part.)"""
    d = json.loads(S.wing_sail_row(wings, panels, 1, apparent_wind_angle_deg=60.0))
    wake = {"viscous_core_length": core, "symmetry_condition": symmetry}
    setup = S.simulation(d["line_force_model"], False, None, wake)
    g, o = Simulation(setup), oracle_mod.OracleSimulation(setup)
    u = np.tile([5.0, 8.0, 0.1], (g.nr_freestream_points, 1))
    rg = g.do_step(time=0.0, time_step=0.1, freestream_velocity=u)
    ro = o.do_step(time=0.0, time_step=0.1, freestream_velocity=u)
    assert rel_inf(rg.circulation_strength, ro.circulation_strength) <= 1e-9
    assert rel_vec(rg.integrated_forces_sum(), ro.integrated_forces_sum()) <= 1e-9


@pytest.mark.parametrize("scale", [1e-4, 1e-2, 1.0])
@pytest.mark.parametrize("core", [0.0, 0.3])
def test_fp64_ring_and_doublet(gpu_lib, oracle_mod, core, scale):
    """Targets on corners, on edges, beside them, beyond the ends and far away; panels with a repeated
    corner; lengths below a metre, where the 1e-10 cut-off fires for more pairs (far above it, a target
    on a line is no longer cut off and its velocity is rounding)."""
    rng = np.random.default_rng(5)
    corners = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]], dtype=float) + rng.normal(0, 0.05, (40, 4, 3))
    corners += rng.uniform(-3, 3, (40, 1, 3))
    corners[3, 2] = corners[3, 1]  # a triangle
    c = corners[:8]
    edge = 0.3 * c[:, 0] + 0.7 * c[:, 1]
    targets = np.concatenate([c.reshape(-1, 3), edge, edge + 1e-6, 2.0 * c[:, 1] - c[:, 0], rng.normal(0, 4, (50, 3)),
                              rng.normal(0, 200, (50, 3))])
    g = rng.normal(0, 3, len(corners))
    args = corners * scale, g, np.full(len(corners), core * scale)
    ours = panel_sweep(*args, targets * scale, far_field_ratio=5.0, precision="fp64")
    ref = oracle_mod.bs_sweep(args[0], args[2], g, 5.0, targets * scale, nthreads=4)
    assert np.all(np.isfinite(ref))
    assert rel_inf(ours, ref) <= 1e-12
