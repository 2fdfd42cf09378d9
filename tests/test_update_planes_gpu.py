"""The bit-plane update kernel against an event-by-event restatement, device noise on: trains, order of
the pulses and the Gaussian every pulse gets (pools of 256 per 32 weights, taken in rounds that start
once a weight holds more than 20 events after a group of four rows in which its input line pulsed)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TAG_X, TAG_D, TAG_DEVICE = 0x30000000, 0x40000000, 0x50000000


def _philox7(c, key):
    """Philox4x32 with seven rounds; ``c``: four uint32 arrays."""
    c = [np.asarray(v, np.uint64) & 0xFFFFFFFF for v in np.broadcast_arrays(*c)]
    k0, k1 = key
    for _ in range(7):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & np.uint64(0xFFFFFFFF),
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & np.uint64(0xFFFFFFFF)]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _managed(x, d, lr, dw_min, desired):
    """Train length and the factors of d and x per sample, update management on."""
    f = np.float32
    xm, dm = np.abs(x).max(1), np.abs(d).max(1)
    k = ((f(lr) * xm).astype(f) * dm).astype(f) / f(dw_min)
    bl = np.minimum(np.ceil(k), desired).astype(int)
    unit = np.sqrt(f(lr) / (f(dw_min) * bl.astype(f)).astype(f)).astype(f)
    dm = np.where(k > desired, (dm * (f(desired) / k)).astype(f), dm)
    return bl, (unit * np.sqrt(xm / dm).astype(f)).astype(f), (unit * np.sqrt(dm / xm).astype(f)).astype(f)


def _trains(v, strength, lengths, bl, key, tag):
    """Pulses ``[sample, line, slot]`` of a batch ``[sample, line]``."""
    m, n = v.shape
    p = (np.abs(v) * strength[:, None]).astype(np.float32)
    thr = np.ceil((p * np.float32(65536) - np.float32(0.5)).astype(np.float32))
    out = np.zeros((m, n, bl), bool)
    line, smp = np.arange(n)[None, :], np.arange(m)[:, None]
    for k in range(bl):
        seg, slot = divmod(k, 31)
        r = _philox7((line, smp, 0, tag + seg * 4 + slot // 8), key)[(slot % 8) >> 1]
        out[:, :, k] = ((r >> np.uint64(16 * (slot & 1))) & np.uint64(0xFFFF)).astype(np.float64) < thr
    return out & (np.arange(bl) < lengths[:, None])[:, None, :]


def _pool(task, refill, key):
    pair = (task * 32 + np.arange(32)).astype(np.uint64) | np.uint64(refill << 40)
    r = _philox7((pair & np.uint64(0xFFFFFFFF), pair >> np.uint64(32), 0, TAG_DEVICE), key)
    z = np.zeros((8, 32))
    for h in range(4):
        u1 = 1.0 - (r[h] >> np.uint64(16)).astype(np.float64) / 65536.0
        ang = 2 * np.pi * (r[h] & np.uint64(0xFFFF)).astype(np.float64) / 65536.0
        rad = np.sqrt(-2.0 * np.log(u1))
        z[2 * h], z[2 * h + 1] = rad * np.cos(ang), rad * np.sin(ang)
    return z.reshape(-1).astype(np.float32)


def _apply_task(w, hi, lo, up, down, counts, dirs, rows, std, task, key, rule=None):
    """One x-line and up to 32 d-lines: ``counts`` / ``dirs`` ``[row, lane]``, ``rows`` those in which the
    x-line pulsed; ``rule(lane, w, down, std * z)``: the weight after a pulse, ConstantStep by default.
    Returns the number of pulses of the busiest weight."""
    one, n_lanes = np.float32(1), w.size
    state = {"pool": None, "pos": 256, "refills": 0}

    def take(n):
        if state["pos"] + n > 256:
            state["pool"] = _pool(task, state["refills"], key)
            state["refills"] += 1
            state["pos"] = 0
        state["pos"] += n
        return state["pool"][state["pos"] - n : state["pos"]]

    def drain(q):
        for r in range(max(len(e) for e in q)):
            n = [e[r][0] if r < len(e) else 0 for e in q]
            for k in range(max(n)):
                lanes = [l for l in range(n_lanes) if k < n[l]]
                for l, z in zip(lanes, take(len(lanes))):
                    if rule is not None:
                        w[l] = rule(l, w[l], q[l][r][1], np.float32(std) * z)
                        continue
                    f = one + np.float32(std) * z
                    w[l] = w[l] - f * down[l] if q[l][r][1] else w[l] + f * up[l]
                    w[l] = max(min(w[l], hi[l]), lo[l])

    q = [[] for _ in range(n_lanes)]
    for g in range(0, len(rows), 4):
        for s in rows[g : g + 4]:
            for l in range(n_lanes):
                if counts[s, l]:
                    q[l].append((int(counts[s, l]), bool(dirs[s, l])))
        if max(len(e) for e in q) > 20:
            drain(q)
            q = [[] for _ in range(n_lanes)]
    drain(q)
    return int(counts.sum(0).max())


@pytest.mark.parametrize("x_size,d_size,m,bl,scale,layout", [
    (3, 33, 32, 1, 0.9, "rows"),     # one block, one slot, lines past a warp
    (5, 31, 33, 1, 1.0, "rows"),     # every row pulses: rounds start inside words
    (2, 64, 97, 2, 0.6, "trans"),    # ragged last block, two slots, transposed inputs
    (65, 7, 130, 3, 0.3, "rows"),    # sparse: a group of four rows spans words
    (4, 40, 70, 4, 0.8, "rows"),     # the first train of more than three slots
    (3, 32, 45, 31, 0.7, "trans"),   # longest train of one segment, many pulses per event
    (2, 35, 40, 40, 0.5, "rows"),    # two segments per sample
    (3, 33, 300, 20, 0.5, "managed"),  # lengths per sample: blocks with and without more than three slots
])
def test_pulses_and_noise_event_by_event(x_size, d_size, m, bl, scale, layout):
    from aihwkit_b200.rpu_base import devices as D
    from aihwkit_b200.rpu_base import tiles as T

    rng = np.random.default_rng(x_size * 1000 + m)
    p = D.AnalogTileParameter()
    p.update.pulse_type, p.update.desired_bl = D.PulseType.StochasticCompressed, bl
    p.update.update_management = p.update.update_bl_management = layout == "managed"
    p.update.fixed_bl = True
    dp = D.ConstantStepResistiveDeviceParameter()
    dp.dw_min, dp.dw_min_std, dp.construction_seed, dp.enforce_consistency = 0.002, 0.3, 11, True
    t = T.AnalogTile(p._config(x_size, d_size, dp, seed=17), cuda_device=0)
    seed = (5 << 32) | 1234567
    t.set_seed(seed)
    key = (seed & 0xFFFFFFFF, (seed >> 32) ^ 0x5BD1E995)
    lr = 0.01 if layout == "managed" else 0.002 * bl  # else: strength sqrt(lr / (dw_min * bl)) = 1
    t.set_learning_rate(lr)
    x = (rng.uniform(0.2, 1, (m, x_size)) * rng.choice([-1, 1], (m, x_size)) * scale).astype(np.float32)
    d = (rng.uniform(0.2, 1, (m, d_size)) * rng.choice([-1, 1], (m, d_size)) * scale).astype(np.float32)
    x[rng.random((m, x_size)) < 0.2] = 0.0
    lengths = np.full(m, bl)
    a = b = np.full(m, np.sqrt(np.float32(lr) / (np.float32(0.002) * np.float32(bl))), np.float32)
    if layout == "managed":
        x[:, 0], x[40:50] = np.where(x[:, 0] == 0, 0.5, x[:, 0]), x[40:50] * 4  # (no sample without a pulse)
        lengths, a, b = _managed(x, d, lr, 0.002, bl)
        assert (lengths <= 3).sum() > 200 and (lengths > 3).any()
    names = t.get_hidden_parameter_names()
    hp = t.get_hidden_parameters().numpy()
    hi, lo, up, down = (hp[names.index(k)] for k in ("max_bound", "min_bound", "dwmin_up", "dwmin_down"))
    w = np.clip(rng.uniform(-0.3, 0.3, (d_size, x_size)), lo, hi).astype(np.float32)
    t.set_weights(torch.from_numpy(w))
    xt, dt = torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda()
    if layout == "trans":
        t.update(xt.t().contiguous(), dt.t().contiguous(), False, True, True)
    else:
        t.update(xt, dt)
    got = t.get_weights().numpy()

    # rows: samples, or the segments of at most 31 slots of each
    n_seg = (bl + 30) // 31
    px, pd = _trains(x, b, lengths, bl, key, TAG_X), _trains(d, a, lengths, bl, key, TAG_D)
    busiest = 0
    for j in range(x_size):
        cut = [slice(31 * g, min(bl, 31 * g + 31)) for g in range(n_seg)]
        counts = np.stack([(px[:, j, None, c] & pd[:, :, c]).sum(-1) for c in cut], 1).reshape(m * n_seg, d_size)
        rows = np.flatnonzero(np.stack([px[:, j, c].any(-1) for c in cut], 1).reshape(-1))
        dirs = np.repeat((x[:, j, None] > 0) == (d > 0), n_seg, axis=0)  # equal signs: decrease
        for i0 in range(0, d_size, 32):
            s = slice(i0, min(i0 + 32, d_size))
            task = j * ((d_size + 31) // 32) + i0 // 32
            col = w[s, j].copy()
            busiest = max(busiest, _apply_task(col, hi[s, j], lo[s, j], up[s, j], down[s, j], counts[:, s],
                                               dirs[:, s], rows, 0.3, task, key))
            w[s, j] = col
    # one rounding of a value below 1 per pulse may fall the other way (the device's logarithm, sine and
    # cosine are approximations); a Gaussian given to another pulse moves a weight by about 6e-4
    assert np.abs(got - w).max() <= busiest * 2.0 ** -24
    assert busiest > 3


def _rule(kind, mult, col):
    """Linear step (SoftBounds) and SoftBoundsReference, noise multiplied with the step or added to it; ``col``: the
    parameters of the lanes by name."""
    one = np.float32(1)

    def linear(l, w, down, xi):
        sl, sc = (col["slope_down"][l], col["dwmin_down"][l]) if down else (col["slope_up"][l], col["dwmin_up"][l])
        dw = (sl * w + sc) * (one + xi) if mult else sl * w + sc * (one + xi)
        return max(min(w - dw if down else w + dw, col["max_bound"][l]), col["min_bound"][l])

    def reference(l, w, down, xi):
        sc, bound = ((col["dwmin_down"][l], col["min_bound"][l]) if down
                     else (col["dwmin_up"][l], col["max_bound"][l]))
        w = w + col["reference"][l]
        rest = one - w / bound
        dw = sc * rest * (one + xi) if mult else sc * (rest + xi)
        return max(min(w - dw if down else w + dw, col["max_bound"][l]), col["min_bound"][l]) - col["reference"][l]

    return linear if kind in ("ls", "sb") else reference


@pytest.mark.parametrize("kind", ["ls", "sb", "sbr"])
@pytest.mark.parametrize("mult", [False, True])
@pytest.mark.parametrize("x_size,d_size,m", [(3, 33, 70), (5, 31, 140)])
def test_noise_multiplied_or_added_event_by_event(kind, mult, x_size, d_size, m):
    from aihwkit_b200.rpu_base import devices as D
    from aihwkit_b200.rpu_base import tiles as T
    from tests import helpers as H

    rng = np.random.default_rng(m)
    bl, dw_min, std = 3, 0.01, 0.3
    p = D.AnalogTileParameter()
    p.update.pulse_type, p.update.desired_bl = D.PulseType.StochasticCompressed, bl
    p.update.update_management = p.update.update_bl_management = False
    p.update.fixed_bl = True
    dp = H.device(kind, True, dw_min=dw_min, dw_min_std=std, mult_noise=mult)
    if kind == "ls":
        dp.gamma_up, dp.gamma_down = 0.3, 0.4
    t = T.AnalogTile(p._config(x_size, d_size, dp, seed=17), cuda_device=0)
    t.set_seed(1234567)
    key = (1234567, 0x5BD1E995)
    t.set_learning_rate(dw_min * bl)  # strength 1
    x = (rng.uniform(0.4, 0.9, (m, x_size)) * rng.choice([-1, 1], (m, x_size))).astype(np.float32)
    d = (rng.uniform(0.4, 0.9, (m, d_size)) * rng.choice([-1, 1], (m, d_size))).astype(np.float32)
    names = t.get_hidden_parameter_names()
    hp = dict(zip(names, t.get_hidden_parameters().numpy()))
    w = np.clip(rng.uniform(-0.3, 0.3, (d_size, x_size)), hp["min_bound"], hp["max_bound"]).astype(np.float32)
    t.set_weights(torch.from_numpy(w))
    t.update(torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda())
    got = t.get_weights().numpy()

    unit = np.full(m, np.sqrt(np.float32(dw_min * bl) / (np.float32(dw_min) * np.float32(bl))), np.float32)
    lengths = np.full(m, bl)
    px, pd = _trains(x, unit, lengths, bl, key, TAG_X), _trains(d, unit, lengths, bl, key, TAG_D)
    busiest = 0
    for j in range(x_size):
        counts = (px[:, j, None] & pd).sum(-1)
        rows = np.flatnonzero(px[:, j].any(-1))
        dirs = (x[:, j, None] > 0) == (d > 0)
        for i0 in range(0, d_size, 32):
            s = slice(i0, min(i0 + 32, d_size))
            col = w[s, j].copy()
            rule = _rule(kind, mult, {n: v[s, j] for n, v in hp.items()})
            busiest = max(busiest, _apply_task(col, None, None, None, None, counts[:, s], dirs[:, s], rows, std,
                                               j * ((d_size + 31) // 32) + i0 // 32, key, rule))
            w[s, j] = col
    # two roundings of values below 2 per pulse (the weight, and the weight without its reference) may fall the other
    # way where the device's Gaussian differs in its last bits; one that belongs to another pulse, or the other form
    # of the noise, moves a weight by about 3e-3
    assert np.abs(got - w).max() <= busiest * 2.0 ** -22
    assert busiest > 20


@pytest.mark.parametrize("omega", [0.0, 0.6])
@pytest.mark.parametrize("kind", ["cs", "sb", "sbr"])
def test_noisy_tiles_of_a_layer_share_launches(kind, omega):
    """Device noise on: twelve tiles in shared launches against the same tiles as layers of one tile each."""
    from aihwkit_b200.rpu_base import tiles as T
    from tests import helpers as H

    g = torch.Generator().manual_seed(3)
    out_size, in_size, m = 200, 130, 65
    p = H.training_params(noise=False, pulse_det=False)
    cfg = p._config(64, 64, H.device(kind, True, dw_min=0.002, dw_min_dtod=0.3), seed=5)
    w = torch.rand(out_size, in_size, generator=g) - 0.5
    x = (torch.rand(m, in_size, generator=g) * 2 - 1).cuda()
    d = (torch.randn(m, out_size, generator=g) * 0.2).cuda()

    def run(**block):
        layer = T.TileArray(cfg, out_size, in_size, 64, 64, cuda_device=0, **block)
        layer.set_seed(9)
        layer.set_weights(w, weight_scaling_omega=omega)
        layer.set_learning_rate(0.05)
        for _ in range(2):
            layer.update(x, d)
        return layer.get_weights(), layer.num_in_splits, layer.num_out_splits

    whole, n_in, n_out = run()
    assert n_in * n_out == 12
    parts = torch.zeros_like(whole)
    for i in range(n_in):
        for o in range(n_out):
            parts += run(in_split_range=(i, i + 1), out_split_range=(o, o + 1))[0]
    assert torch.equal(whole, parts)
    assert (whole - w).abs().max() > 1e-3


@pytest.mark.parametrize("out_size,in_size,max_tile,m,omega", [
    (70, 33, 64, 32, 0.0),     # two ragged tiles in one launch
    (200, 130, 64, 65, 0.6),   # twelve tiles: a full launch and a rest, scaled gradients
    (96, 300, 100, 40, 0.0),   # three tiles along the inputs
])
def test_tiles_of_a_layer_share_launches(out_size, in_size, max_tile, m, omega):
    """Device noise off: the shared launches against the staged kernel tile by tile, bit for bit."""
    from aihwkit_b200 import _cabi
    from aihwkit_b200.rpu_base import tiles as T
    from tests import helpers as H

    g = torch.Generator().manual_seed(out_size + m)
    p = H.training_params(noise=False, pulse_det=False)
    cfg = p._config(max_tile, max_tile, H.device("sb", False, dw_min=0.002, dw_min_dtod=0.3), seed=5)
    w = torch.rand(out_size, in_size, generator=g) - 0.5
    x = (torch.rand(m, in_size, generator=g) * 2 - 1).cuda()
    d = (torch.randn(m, out_size, generator=g) * 0.2).cuda()
    out = []
    lib = _cabi.lib()
    try:
        for path in (0, 1):
            _cabi.check(lib.ab200_set_update_path(path))
            layer = T.TileArray(cfg, out_size, in_size, max_tile, max_tile, cuda_device=0)
            layer.set_seed(9)
            layer.set_weights(w, weight_scaling_omega=omega)
            layer.set_learning_rate(0.05)
            for _ in range(2):
                layer.update(x, d)
            out.append(layer.get_weights())
    finally:
        _cabi.check(lib.ab200_set_update_path(0))
    assert torch.equal(out[0], out[1])
    assert (out[0] - w).abs().max() > 1e-3


@pytest.mark.parametrize("path,m", [(1, 24), (2, 24), (0, 64), (1, 64)])
@pytest.mark.parametrize("every", [1, 5])
def test_noise_of_the_ranges_between_transfers(path, m, every):
    """A transfer compound whose transfers fall inside the batch applies it in ranges; a pulse on every weight for
    every row, so the spread of the weights tells whether the ranges draw their noise independently."""
    from aihwkit_b200 import _cabi
    from aihwkit_b200.rpu_base import devices as D
    from aihwkit_b200.rpu_base import tiles as T
    from tests import helpers as H

    x_size, d_size, dw_min, std = 40, 70, 1e-3, 0.3
    dp = D.TransferResistiveDeviceParameter()
    for _ in range(2):
        dp.append_parameter(H.device("cs", True, dw_min=dw_min, dw_min_std=std, dw_min_dtod=0.0, up_down_dtod=0.0,
                                     w_max=1.0, w_min=-1.0))
    dp.construction_seed, dp.gamma, dp.transfer_every, dp.units_in_mbatch = 21, 0.0, float(every), False
    dp.transfer_lr, dp.fast_lr = 0.0, 0.0  # the pulses take the learning rate; transfers cut the batch and write nothing
    p = H.training_params(noise=False, pulse_det=False)
    p.update.desired_bl, p.update.fixed_bl = 1, True
    p.update.update_management = p.update.update_bl_management = False
    lib = _cabi.lib()
    try:
        _cabi.check(lib.ab200_set_update_path(path))
        t = T.AnalogTile(p._config(x_size, d_size, dp, seed=3), cuda_device=0)
        t.set_learning_rate(dw_min)
        t.set_weights(torch.zeros(d_size, x_size))
        names = t.get_hidden_parameter_names()
        fast = next(i for i, n in enumerate(names) if n.startswith("hidden_weights"))
        before = t.get_hidden_parameters()[fast].double()
        t.update(torch.ones(m, x_size, device="cuda"), -torch.ones(m, d_size, device="cuda"))
        change = (t.get_hidden_parameters()[fast].double() - before) / dw_min
    finally:
        _cabi.check(lib.ab200_set_update_path(0))
    n = change.numel()
    # sums of m independent steps 1 + std * z over n weights: the mean of all, and their spread, each within five
    # standard errors (the same draws in every range of r rows spread the sums sqrt(m / r) times as far)
    assert abs(float(change.mean()) - m) <= 5 * std * (m / n) ** 0.5
    assert abs(float(change.std()) / (std * m ** 0.5) - 1) <= 5 * (0.5 / n) ** 0.5


def test_scaled_gradients_take_no_memory_of_their_own():
    """The shared launches divide by the mapping scales themselves: an update of a scaled layer holds no copy of the
    gradient per tile."""
    from aihwkit_b200.rpu_base import tiles as T
    from tests import helpers as H

    size, tile, m = 1024, 256, 4096  # sixteen tiles; a block of the gradient is 4 MB
    p = H.training_params(noise=False, pulse_det=False)
    layer = T.TileArray(p._config(tile, tile, H.device("sb", False), seed=5), size, size, tile, tile, cuda_device=0)
    layer.set_weights(torch.rand(size, size) - 0.5, weight_scaling_omega=0.6)
    layer.set_learning_rate(0.01)
    x, d = torch.rand(m, size, device="cuda"), 0.01 * torch.randn(m, size, device="cuda")
    layer.update(x[:64], d[:64])  # loads the kernels
    layer.forward(x)
    layer.backward(d)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    layer.update(x, d)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < m * tile * 4


@pytest.mark.parametrize("x_size,d_size,m,every", [(512, 512, 40, 1.0), (300, 1000, 37, 1.0), (300, 1000, 70, 7.0)])
def test_ranges_of_one_row_in_large_tiles(x_size, d_size, m, every):
    """A transfer after every row, in tiles whose lines are looked at before their weights are read, and longer ranges
    of the same: against the staged kernel, device noise off, bit for bit, the slow tile included."""
    from aihwkit_b200 import _cabi
    from aihwkit_b200.rpu_base import tiles as T
    from tests import helpers as H

    g = torch.Generator().manual_seed(m)
    p = H.training_params(noise=False, pulse_det=False)
    x = (torch.rand(m, x_size, generator=g) * 2 - 1).cuda()
    x[torch.rand(m, x_size, generator=g).cuda() < 0.3] = 0.0
    d = (torch.randn(m, d_size, generator=g) * 0.2).cuda()
    out = []
    lib = _cabi.lib()
    try:
        for path in (0, 1):
            _cabi.check(lib.ab200_set_update_path(path))
            t = T.AnalogTile(p._config(x_size, d_size, H.transfer_device(False, transfer_every=every,
                                                                         units_in_mbatch=False), seed=3), cuda_device=0)
            t.set_learning_rate(0.05)
            t.update(x, d)
            out.append((t.get_weights(), t.get_hidden_parameters()))
    finally:
        _cabi.check(lib.ab200_set_update_path(0))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert out[0][1].abs().sum() > 0
