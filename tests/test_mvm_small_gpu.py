"""The CUDA-core kernel for small batches at the edges of its tiles: rows 4 / 8 / 16 per CTA, columns in 32s,
features in steps of 512, and the tiles of a mapped layer in one launch."""

import numpy as np
import pytest
import torch

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 4, 5, 8, 9, 16, 17])
@pytest.mark.parametrize("x_size,d_size", [(1, 33), (31, 1), (64, 32), (130, 785), (512, 96), (513, 31), (1030, 40)])
def test_perfect_io_against_float64(m, x_size, d_size):
    from aihwkit_b200.rpu_base import tiles as T

    g = torch.Generator().manual_seed(m * 10000 + x_size)
    t = T.FloatingPointTile(x_size, d_size, cuda_device=0)
    w = torch.rand(d_size, x_size, generator=g) - 0.5
    t.set_weights(w)
    x, d = torch.rand(m, x_size, generator=g) - 0.5, torch.rand(m, d_size, generator=g) - 0.5
    y, gr = t.forward(x.cuda()).cpu().double(), t.backward(d.cuda()).cpu().double()
    # K products of at most 1/4 and K - 1 additions in fp32, each rounded once
    for got, a, b, k in ((y, x, w.t(), x_size), (gr, d, w, d_size)):
        assert (got - a.double() @ b.double()).abs().max() <= k * k * 0.25 * 2.0 ** -24


@pytest.mark.parametrize("out_size,in_size,max_tile,m", [
    (96, 64, 64, 3), (33, 200, 70, 7), (700, 130, 64, 16), (1536, 384, 192, 21), (100, 2300, 64, 2)])
def test_mapped_layer_against_its_tiles_one_by_one(out_size, in_size, max_tile, m):
    """Scaled tiles, bias and all noise on: the layer in one launch of the fp32 kernel for small batches against the
    tensor-core path of the same layer, with the same weights and noise streams."""
    from aihwkit_b200 import _cabi
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(out_size + in_size)
    cfg = H.inference_params(True)._config(max_tile, max_tile, H.D.IdealResistiveDeviceParameter(), seed=3)
    w = torch.from_numpy(rng.normal(0, 0.1, (out_size, in_size)).astype(np.float32))
    x = torch.from_numpy(rng.normal(0, 1, (m, in_size)).astype(np.float32)).cuda()
    bias = torch.from_numpy(rng.normal(0, 0.1, out_size).astype(np.float32))
    out = []
    lib = _cabi.lib()
    try:
        for path in (0, 2):  # the fp32 kernel for small batches, the tensor-core kernel
            _cabi.check(lib.ab200_set_mvm_path(path))
            layer = T.TileArray(cfg, out_size, in_size, max_tile, max_tile, cuda_device=0)
            layer.set_seed(77)
            layer.set_weights(w, weight_scaling_omega=1.0)
            layer.set_bias(bias)
            layer.forward(x)
            out.append(layer.forward(x).cpu().double())  # second call: the call counters advanced alike
            scales = layer.get_tile_scales()
    finally:
        _cabi.check(lib.ab200_set_mvm_path(0))
    # the split-bf16 weights move a sum by less than an ADC step: a code differs by one where the sum is
    # next to a rounding tie, in the scale of the largest tile and input
    step = 2 * 10.0 / 254.0 * float(scales.max()) * float(x.abs().max())
    diff = (out[0] - out[1]).abs()
    assert diff.max() <= 2.01 * step
    assert (diff > 1e-4 * step).double().mean() <= 0.002 * scales.size(0) + 2.0 / diff.numel()


@pytest.mark.parametrize("size", [64, 100, 256, 300, 512, 600])
@pytest.mark.parametrize("w_noise", [0.0, 0.1])
@pytest.mark.parametrize("bm", [False, True])
def test_rows_of_very_small_numbers(size, w_noise, bm):
    """The abs-max scale of such a row is infinite: every input is +-1 after the DAC, and the zeros behind the last
    feature stay out of the product and of the norm. Against the same rows at the head of a batch that the general
    kernel takes."""
    from aihwkit_b200 import _cabi
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(size)
    p = H.training_params(noise=False, pulse_det=False, bm=bm)
    for io in (p.forward_io, p.backward_io):
        if w_noise:
            io.w_noise, io.w_noise_type = w_noise, H.D.WeightNoiseType.AdditiveConstant
    cfg = p._config(size, size, H.device("cs", False), seed=3)
    w = torch.from_numpy(rng.uniform(-0.1, 0.1, (size, size)).astype(np.float32))
    x = (rng.uniform(0.5, 1.5, (4096, size)) * rng.choice([-1, 1], (4096, size))).astype(np.float32)
    x[1], x[3] = x[1] * np.float32(1e-39), x[3] * np.float32(1e-42)
    assert (x != 0).all()
    out = []
    lib = _cabi.lib()
    try:
        _cabi.check(lib.ab200_set_mvm_path(1))  # CUDA cores for the large batch too
        for m in (5, 4096):
            t = T.AnalogTile(cfg, cuda_device=0)
            t.set_weights(w)
            rows = torch.from_numpy(x[:m]).cuda()
            out.append([v[:5].cpu().double() for v in (t.forward(rows), t.backward(rows))])
    finally:
        _cabi.check(lib.ab200_set_mvm_path(0))
    amax = torch.from_numpy(np.abs(x[:5]).max(1)).double()[:, None]
    for got, want in zip(*out):
        assert torch.isfinite(got).all() and torch.isfinite(want).all()
        # sums in another order: a code differs by one step (times the re-run's input reduction, at most 16
        # here) where the sum is next to a rounding tie; results of a tiny row are multiples of 2^-149
        diff = (got - want).abs() - 2.0 ** -149
        assert (diff <= 16.01 * 24.0 / 510.0 * amax).all()
        assert (diff > 1e-3 * 24.0 / 510.0 * amax).double().mean() <= 0.005
    assert out[0][1][1].abs().max() > 0


@pytest.mark.parametrize("m", [2, 4, 7, 16, 50])
@pytest.mark.parametrize("x_size,d_size", [(2, 33), (40, 3), (130, 785), (512, 64), (513, 31), (1030, 40)])
@pytest.mark.parametrize("bias", [False, True])
def test_transposed_inputs_bit_for_bit(m, x_size, d_size, bias):
    """[features][rows] inputs and outputs against the same rows the other way round, noise, bound management and
    weight noise on."""
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(m * 1000 + x_size)
    p = H.training_params(noise=True, pulse_det=False, out_bound=2.0)
    for io in (p.forward_io, p.backward_io):
        io.w_noise, io.w_noise_type = 0.02, H.D.WeightNoiseType.AdditiveConstant
    cfg = p._config(x_size, d_size, H.device("cs", False), seed=3)
    w = torch.from_numpy(rng.uniform(-0.5, 0.5, (d_size, x_size)).astype(np.float32))
    x = torch.from_numpy(rng.uniform(-1, 1, (m, x_size - int(bias))).astype(np.float32)).cuda()
    d = torch.from_numpy(rng.uniform(-1, 1, (m, d_size)).astype(np.float32)).cuda()
    out = []
    for trans in (False, True):
        t = T.AnalogTile(cfg, cuda_device=0)
        t.set_weights(w)
        if trans:
            y = t.forward(x.t().contiguous(), bias, True, True).t()
            out.append((y, t.backward(d.t().contiguous(), bias, True, True).t()))
        else:
            out.append((t.forward(x, bias), t.backward(d, bias)))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("x_size,d_size", [(40, 70), (600, 130)])
@pytest.mark.parametrize("trans", [False, True])
def test_noise_of_every_line(x_size, d_size, trans):
    """out_noise_std > 0: a standard deviation per output line. Against the general kernel on a batch with the same
    rows at its head."""
    from aihwkit_b200 import _cabi
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(x_size)
    p = H.training_params(noise=True, pulse_det=False)
    for io in (p.forward_io, p.backward_io):
        io.out_noise_std = 0.5
    p.forward_io.bound_management = H.D.BoundManagementType.None_
    cfg = p._config(x_size, d_size, H.device("cs", False), seed=3)
    w = torch.from_numpy(rng.uniform(-0.1, 0.1, (d_size, x_size)).astype(np.float32))
    x = rng.uniform(-1, 1, (8192, x_size)).astype(np.float32)
    d = rng.uniform(-1, 1, (8192, d_size)).astype(np.float32)
    out = []
    lib = _cabi.lib()
    try:
        _cabi.check(lib.ab200_set_mvm_path(1))
        for m in (9, 8192):
            t = T.AnalogTile(cfg, cuda_device=0)
            t.set_weights(w)
            xm, dm = torch.from_numpy(x[:m]).cuda(), torch.from_numpy(d[:m]).cuda()
            if trans:
                y = t.forward(xm.t().contiguous(), False, True, True).t()
                g = t.backward(dm.t().contiguous(), False, True, True).t()
            else:
                y, g = t.forward(xm), t.backward(dm)
            out.append((y[:9].cpu().double(), g[:9].cpu().double()))
    finally:
        _cabi.check(lib.ab200_set_mvm_path(0))
    for got, want, rows in zip(out[0], out[1], (x, d)):
        # sums in another order: a code differs by one where the sum is next to a rounding tie
        step = 24.0 / 510.0 * torch.from_numpy(np.abs(rows[:9]).max(1)).double()[:, None]
        diff = (got - want).abs()
        assert (diff <= 1.01 * step).all() and (diff > 1e-3 * step).double().mean() <= 0.005


@pytest.mark.parametrize("kind", ["plain", "weight noise", "line noise", "line chain", "worst case"])
@pytest.mark.parametrize("x_size,d_size", [(40, 33), (300, 70), (75, 300), (130, 520)])
def test_rerun_of_a_row_does_not_depend_on_the_other_rows(kind, x_size, d_size):
    """Bound management with 256, 512 and 1024 threads per row and up to five rows per CTA: a row has the same bits
    whether it is the only one of its CTA that clips or one of all."""
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(x_size)
    p = H.training_params(noise=True, pulse_det=False, out_bound=0.05 * x_size)
    io = p.forward_io
    if kind == "weight noise":
        io.w_noise, io.w_noise_type = 0.05, H.D.WeightNoiseType.AdditiveConstant
    elif kind == "line noise":
        io.out_noise_std = 0.3
    elif kind == "line chain":
        io.w_noise, io.w_noise_type = 0.02, H.D.WeightNoiseType.PCMRead
    elif kind == "worst case":
        io.bound_management = H.D.BoundManagementType.IterativeWorstCase
    cfg = p._config(x_size, d_size, H.device("cs", False), seed=3)
    w = rng.uniform(-0.5, 0.5, (d_size, x_size)).astype(np.float32)
    m = 1300  # up to five rows per CTA
    few = np.sort(rng.choice(m, 40, replace=False))
    x = (np.sign(w[rng.integers(0, d_size, m)]) * rng.uniform(0.8, 1, (m, x_size))).astype(np.float32)
    rest = 0.02 * rng.uniform(-1, 1, (m, x_size)).astype(np.float32)
    rest[:, 0] = 1.0
    rest[few] = x[few]
    out, served = [], []
    for rows in (x, rest):
        t = T.AnalogTile(cfg, cuda_device=0)
        t.set_weights(torch.from_numpy(w))
        out.append(t.forward(torch.from_numpy(rows).cuda())[torch.from_numpy(few).cuda()])
        served.append(t.last_bm_stats()[0])
    assert served[0] == m and 40 <= served[1] <= 60
    assert torch.equal(out[0], out[1])
