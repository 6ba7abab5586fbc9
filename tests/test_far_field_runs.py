"""Far-field runs of the FP32 panel sweep: panel counts around the run of 8, the test's 32 and the tile of 64;
zero-strength panels singly and as whole runs; warps of targets far from every panel, amid them, and beside
their edge, so that runs are all far, mixed and all near.

Against the oracle, 1e-5 of the largest velocity: a term is good to some 30 roundings of 6e-8, and the terms'
magnitudes add up to a few times the largest velocity. The far field begins at 1.5 panel lengths, where a
doublet in place of a ring (or the other way round) is off by percents.
"""
import numpy as np
import pytest

from stormbird_gb300.simulation import panel_sweep

from .helpers import rel_inf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("symmetry", [0, 3])
@pytest.mark.parametrize("zeros", ["none", "some", "runs", "all but one"])
@pytest.mark.parametrize("panels", [1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 72, 200])
def test_runs(gpu_lib, oracle_mod, panels, zeros, symmetry):
    rng = np.random.default_rng(panels)
    k = np.arange(panels)
    # a strip two panels wide along x, somewhat crumpled
    quad = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]], dtype=float)
    corners = quad + np.stack([k // 2, k % 2, 20.0 + 0 * k], axis=1)[:, None, :] + rng.normal(0, 0.05, (panels, 4, 3))
    g = rng.normal(0, 1, panels) + 2.0
    if zeros == "some":
        g[3::7] = 0.0
    elif zeros == "runs":
        g[(k // 8) % 3 == 1] = 0.0
    elif zeros == "all but one":
        g[k != panels // 2] = 0.0
    centre = corners.mean(axis=1)

    def cluster(at, width):
        return at + rng.uniform(-width, width, (64, 3))

    end = centre[-1] + [0.5, 0.0, 0.6]
    targets = np.concatenate([cluster(centre[0] + [0, 0, 40.0], 3.0), cluster(centre[panels // 2] + [0, 0, 1.0], 0.4),
                              cluster(end, 0.4), cluster(centre[0] + [0, 0, 2.0], 0.1), centre[:1] + [[0, 0, 3.0]] * 5])
    core = np.full(panels, 0.05)
    ours = panel_sweep(corners, g, core, targets, far_field_ratio=1.5, symmetry=symmetry, precision="kahan")
    ref = oracle_mod.bs_sweep(corners, core, g, 1.5, targets, nthreads=4)
    if symmetry:
        mirrored = targets * [1.0, 1.0, -1.0]
        m = oracle_mod.bs_sweep(corners, core, g, 1.5, mirrored, nthreads=4)
        ref = ref + m * [1.0, 1.0, -1.0]
    assert rel_inf(ours, ref) <= 1e-5


@pytest.mark.parametrize("symmetry", [0, 3])
@pytest.mark.parametrize("targets", [1, 2, 3, 7, 8, 9, 31, 33, 64, 65, 130, 255, 256])
def test_few_targets(gpu_lib, targets, symmetry):
    """With few targets a warp takes 32 down to 1 or 2 of them: a target's velocity stays the one it has among
    256, bit for bit (its sums run over the same panels in the same order)."""
    rng = np.random.default_rng(8)
    panels = 150
    k = np.arange(panels)
    quad = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]], dtype=float)
    corners = quad + np.stack([k // 5, k % 5, 5.0 + 0 * k], axis=1)[:, None, :] + rng.normal(0, 0.05, (panels, 4, 3))
    g, core = rng.normal(0, 1, panels), np.full(panels, 0.05)
    x = rng.uniform([0, 0, 5.2], [30, 5, 8], (256, 3))
    every = panel_sweep(corners, g, core, x, far_field_ratio=3.0, symmetry=symmetry)
    assert np.array_equal(panel_sweep(corners, g, core, x[:targets], far_field_ratio=3.0, symmetry=symmetry), every[:targets])
