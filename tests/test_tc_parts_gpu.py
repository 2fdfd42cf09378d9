"""Work items of 32 and 64 columns in the tensor-core kernel (small grids) against whole chunks of 128, noise on,
bit for bit: ragged chunks, several in-splits, transposed outputs, bound management."""

import numpy as np
import pytest
import torch

from tests import helpers as H

pytestmark = pytest.mark.gpu


def _both(fn):
    from aihwkit_b200 import _cabi

    lib, out = _cabi.lib(), []
    try:
        for path in (2, 3):  # 2: parts where the grid is small; 3: single CTAs on whole chunks
            _cabi.check(lib.ab200_set_mvm_path(path))
            out.append(fn())
    finally:
        _cabi.check(lib.ab200_set_mvm_path(0))
    return out


@pytest.mark.parametrize("x_size,d_size,m,bm", [
    (64, 1, 1, False),       # one column, one row
    (100, 33, 130, True),    # a part with one column, two row blocks
    (130, 200, 128, False),  # a ragged second chunk: parts of 32, 32 and 8 columns
    (70, 1100, 1000, True),  # 9 chunks x 8 row blocks: parts of 64
    (65, 1300, 700, False),  # the same, no bound management
])
def test_single_tile(x_size, d_size, m, bm):
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(d_size)
    cfg = H.training_params(noise=True, pulse_det=False, bm=bm, out_bound=2.0)._config(
        x_size, d_size, H.device("cs", False), seed=3)
    w = torch.from_numpy(rng.uniform(-0.5, 0.5, (d_size, x_size)).astype(np.float32))
    x = torch.from_numpy(rng.uniform(-1, 1, (m, x_size)).astype(np.float32)).cuda()
    d = torch.from_numpy(rng.uniform(-1, 1, (m, d_size)).astype(np.float32)).cuda()

    def run():
        t = T.AnalogTile(cfg, cuda_device=0)
        t.set_weights(w)
        return t.forward(x), t.forward(x, False, False, True), t.backward(d), t.backward(d, False, False, True)

    for a, b in zip(*_both(run)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("out_size,in_size,max_tile,m", [(96, 200, 64, 40), (500, 700, 256, 300)])
def test_mapped_layer(out_size, in_size, max_tile, m):
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(out_size)
    cfg = H.inference_params(True)._config(max_tile, max_tile, H.D.IdealResistiveDeviceParameter(), seed=3)
    w = torch.from_numpy(rng.normal(0, 0.1, (out_size, in_size)).astype(np.float32))
    x = torch.from_numpy(rng.normal(0, 1, (m, in_size)).astype(np.float32)).cuda()

    def run():
        layer = T.TileArray(cfg, out_size, in_size, max_tile, max_tile, cuda_device=0)
        layer.set_seed(7)
        layer.set_weights(w, weight_scaling_omega=1.0)
        layer.set_bias(torch.linspace(-1, 1, out_size))
        return layer.forward(x)

    a, b = _both(run)
    assert torch.equal(a, b)
