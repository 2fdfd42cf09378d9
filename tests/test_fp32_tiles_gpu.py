"""The fp32 tile kernels (products beyond the small-batch kernel, floating-point update) at the edges of their
16 / 32 / 64-wide tiles, aligned and not, rows or lines contiguous, against float64; and the dense update for
implicit pulses against the oracle."""

import numpy as np
import pytest
import torch

from oracle import analog_tile_oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x_size,d_size,m", [
    (1, 1, 1), (15, 17, 3), (64, 64, 16), (65, 63, 17), (130, 200, 33),
    (700, 900, 31), (768, 1024, 64), (1023, 1025, 65)])
@pytest.mark.parametrize("trans", [False, True])
def test_floating_point_update(x_size, d_size, m, trans):
    from aihwkit_b200.rpu_base import tiles as T

    g = torch.Generator().manual_seed(x_size + m)
    t = T.FloatingPointTile(x_size, d_size, cuda_device=0)
    w = torch.rand(d_size, x_size, generator=g) - 0.5
    x, d = torch.rand(m, x_size, generator=g) - 0.5, torch.rand(m, d_size, generator=g) - 0.5
    t.set_weights(w)
    t.set_learning_rate(0.25)
    if trans:
        t.update(x.t().contiguous().cuda(), d.t().contiguous().cuda(), False, True, True)
    else:
        t.update(x.cuda(), d.cuda())
    want = w.double() - 0.25 * (d.double().t() @ x.double())
    # m products of at most 1/4, each sum rounded once, and the step on the weight
    assert (t.get_weights().double() - want).abs().max() <= (0.25 * m * m * 0.25 + 1.0) * 2.0 ** -24


@pytest.mark.parametrize("x_size,d_size,m", [
    (16, 64, 40000), (17, 200, 12000), (64, 70, 30000), (1100, 1030, 1000), (520, 33, 21000)])
@pytest.mark.parametrize("trans", [False, True])
def test_large_products(x_size, d_size, m, trans):
    from aihwkit_b200.rpu_base import tiles as T

    g = torch.Generator().manual_seed(x_size + m)
    t = T.FloatingPointTile(x_size, d_size, cuda_device=0)
    w = (torch.rand(d_size, x_size, generator=g) - 0.5).cuda()
    x, d = (torch.rand(m, n, generator=g).cuda() - 0.5 for n in (x_size, d_size))
    t.set_weights(w)
    if trans:
        y, gr = t.forward(x.t().contiguous(), False, True, True).t(), t.backward(d.t().contiguous(), False, True, True).t()
    else:
        y, gr = t.forward(x), t.backward(d)
    assert (y.double() - x.double() @ w.double().t()).abs().max() <= x_size ** 2 * 0.25 * 2.0 ** -24
    assert (gr.double() - d.double() @ w.double()).abs().max() <= d_size ** 2 * 0.25 * 2.0 ** -24


@pytest.mark.parametrize("kind", ["cs", "sb", "sbr"])
@pytest.mark.parametrize("x_size,d_size,m", [(1, 1, 1), (5, 63, 64), (17, 65, 65), (300, 520, 3)])
def test_implicit_pulses_without_noise(kind, x_size, d_size, m):
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(x_size * 7 + m)
    p = H.training_params(noise=False, pulse_det=True)
    dp = H.device(kind, False, dw_min=0.002, dw_min_dtod=0.3)
    cfg = p._config(x_size, d_size, dp, seed=5)
    t = T.AnalogTile(cfg, cuda_device=0)
    names, hp = t.get_hidden_parameter_names(), t.get_hidden_parameters().numpy()
    t.set_weights(torch.from_numpy(rng.uniform(-0.3, 0.3, (d_size, x_size)).astype(np.float32)))
    w = t.get_weights().numpy().copy()
    t.set_learning_rate(0.05)
    x = rng.uniform(-1, 1, (m, x_size)).astype(np.float32)
    d = rng.normal(0, 0.2, (m, d_size)).astype(np.float32)
    dev = O.DeviceArrays.from_hidden(
        {"cs": O.DEV_CONSTANT_STEP, "sb": O.DEV_SOFT_BOUNDS, "sbr": O.DEV_SOFT_BOUNDS_REFERENCE}[kind], names, hp,
        0.0, getattr(dp, "mult_noise", True))
    before = w.copy()
    O.update(w, x, d, 0.05, dp.dw_min, O.Up.from_c(cfg.update), dev, None)
    t.update(torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda())
    assert np.abs(t.get_weights().numpy() - w).max() <= 1e-6
    assert m * x_size < 5 or np.abs(w - before).max() > 0


def test_implicit_pulses_of_long_trains():
    """A train of ceil(lr / dw_min) = 2 million slots, past the length up to which the counts are rounded by adding
    2^23, with few pulses per pair."""
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(3)
    p = H.training_params(noise=False, pulse_det=True)
    p.update.fixed_bl = p.update.update_management = p.update.update_bl_management = False
    dp = H.device("sb", False, dw_min=5e-5, dw_min_dtod=0.3)
    x_size, d_size, m = 40, 70, 33
    cfg = p._config(x_size, d_size, dp, seed=5)
    t = T.AnalogTile(cfg, cuda_device=0)
    names, hp = t.get_hidden_parameter_names(), t.get_hidden_parameters().numpy()
    t.set_weights(torch.from_numpy(rng.uniform(-0.3, 0.3, (d_size, x_size)).astype(np.float32)))
    w = t.get_weights().numpy().copy()
    t.set_learning_rate(100.0)
    x = rng.uniform(-3e-3, 3e-3, (m, x_size)).astype(np.float32)
    d = rng.uniform(-3e-3, 3e-3, (m, d_size)).astype(np.float32)
    dev = O.DeviceArrays.from_hidden(O.DEV_SOFT_BOUNDS, names, hp, 0.0, getattr(dp, "mult_noise", True))
    before = w.copy()
    O.update(w, x, d, 100.0, dp.dw_min, O.Up.from_c(cfg.update), dev, None)
    t.update(torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda())
    assert np.abs(t.get_weights().numpy() - w).max() <= 1e-6
    assert np.abs(w - before).max() > 1e-3


@pytest.mark.parametrize("x_size,d_size", [(1024, 1024), (1023, 1025), (1500, 902)])
@pytest.mark.parametrize("m", [1, 15, 16, 17])
def test_floating_point_update_of_few_samples(x_size, d_size, m):
    """One step of samples on the 64-wide tiles, weights in fours and one by one; 17 samples take two steps."""
    from aihwkit_b200.rpu_base import tiles as T

    g = torch.Generator().manual_seed(x_size + m)
    t = T.FloatingPointTile(x_size, d_size, cuda_device=0)
    w = torch.rand(d_size, x_size, generator=g) - 0.5
    x, d = torch.rand(m, x_size, generator=g) - 0.5, torch.rand(m, d_size, generator=g) - 0.5
    t.set_weights(w)
    t.set_learning_rate(0.25)
    t.update(x.cuda(), d.cuda())
    want = w.double() - 0.25 * (d.double().t() @ x.double())
    # m products of at most 1/4, each sum rounded once, and the step on the weight
    assert (t.get_weights().double() - want).abs().max() <= (0.25 * m * m * 0.25 + 1.0) * 2.0 ** -24
