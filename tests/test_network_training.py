"""Training step of the network at the edges of its launches: a remainder in the last tile of 128 rows, one
and two column pieces per tile (as many tiles as SMs, and one more), input counts that are no multiple
of 8.

Gradients against the f64 restatement with the BF16 roundings emulated, 1e-2 of each block's norm (the
bound elsewhere: rare BF16 flips of 2^-8 and FP32 sums); targets well off the outputs, so that the residuals
do not cancel. After a step the network computes with the parameters it reports: a network set to them gives
the same bits forward and backward (the BF16 copies, row-major and transposed, follow the update).
"""
import numpy as np
import pytest

from tests import mlp_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in", [5, 16, 64])
@pytest.mark.parametrize("tiles,extra", [(0, 1), (0, 127), (0, 129), (0, 3000), (1, 0), (1, 1)])
def test_step(gpu_lib, n_in, tiles, extra):
    torch = pytest.importorskip("torch")
    from stormbird_gb300.warm_start import WarmStartNet

    rows = 128 * tiles * torch.cuda.get_device_properties(0).multi_processor_count + extra
    net = WarmStartNet(n_in, seed=6)
    rng = np.random.default_rng(rows + n_in)
    x = rng.normal(size=(rows, n_in)).astype(np.float32)
    t = (20.0 + rng.normal(size=rows)).astype(np.float32)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    g, loss = net.gradients(xd, td)
    p = net.get_params()
    loss_r, g_r = R.loss_and_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64), emulate=True)
    assert abs(loss - loss_r) <= 1e-3 * loss_r
    for name, sl in R.blocks():
        err = np.linalg.norm(g[sl].astype(np.float64) - g_r[sl]) / max(np.linalg.norm(g_r[sl]), 1e-30)
        assert err <= 1e-2, (name, err)

    net.train_step(xd, td, 1e-3)
    q = net.get_params()
    assert not np.array_equal(p, q)
    other = WarmStartNet(n_in, seed=7)
    other.set_params(q)
    assert torch.equal(net.forward(xd), other.forward(xd))
    a, b = net.gradients(xd, td), other.gradients(xd, td)
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]
