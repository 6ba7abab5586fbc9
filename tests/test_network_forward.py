"""Inference of the network in one kernel (tiles of 128 rows; one tile at a time per CTA while there
are no more tiles than SMs, two in turn beyond that): sizes around the edges of a tile, of one tile per
SM and of two, input counts with and without a remainder of 4 or 8, and rows that start off a
16-byte boundary.

Every row against the f64 restatement (BF16 roundings emulated) within 5e-3 of the largest output,
the bound of the forward pass elsewhere: FP32 accumulation order and rare BF16 flips. A row's result
depends on nothing but the row: calls over odd pieces give the same bits.
"""
import numpy as np
import pytest

from tests import mlp_ref as R

pytestmark = pytest.mark.gpu


def _rows(torch, spec):
    tiles, extra = spec
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 128 * int(tiles * sms) + extra if tiles else extra


@pytest.mark.parametrize("n_in,offset", [(16, 0), (5, 0), (20, 1), (64, 0), (64, 3)])
@pytest.mark.parametrize("spec", [(0, 1), (0, 127), (0, 128), (0, 129), (1, -1), (1, 0), (1, 1), (2, 0), (2, 1), (5, 77)])
def test_rows(gpu_lib, spec, n_in, offset):
    torch = pytest.importorskip("torch")
    from stormbird_gb300.warm_start import WarmStartNet

    rows = _rows(torch, spec)
    net = WarmStartNet(n_in, seed=4)
    rng = np.random.default_rng(rows + n_in)
    x = rng.normal(size=(rows, n_in)).astype(np.float32)
    flat = torch.empty(rows * n_in + offset, device="cuda")
    xd = flat[offset:].view(rows, n_in)
    xd.copy_(torch.from_numpy(x))
    y = net.forward(xd)
    yr, _, _ = R.forward(net.get_params().astype(np.float64), x[-4096:].astype(np.float64), emulate=True)
    assert np.max(np.abs(y.cpu().numpy()[-4096:] - yr)) <= 5e-3 * np.max(np.abs(yr))
    step = 4099
    alone = torch.cat([net.forward(xd[r:r + step].clone()) for r in range(0, rows, step)])
    assert torch.equal(alone, y)
