"""The work that users of the analog tile have it do, as cases of one pass each.

A case names a kind of call and its sizes; every kind goes through the package's public classes
(``AnalogTile``, ``FloatingPointTile``, ``TileArray``) the way a training or serving loop does: inputs
on the GPU, calls enqueued on the current stream (``non_blocking``), weights of single tiles shared
with the caller as the layers above the tile share them.

Noise stays on where a user has it on. All draws are functions of the tile's seed, so a pass on the
same inputs gives the same numbers.
"""

import math

import torch
import torch.nn.functional as F

from aihwkit_b200.rpu_base import devices as D
from aihwkit_b200.rpu_base import tiles as T


def listed():
    return [
        # one vector through one physical tile: the smallest call, latency and launches only
        {"name": "tile_infer_512_m1", "kind": "tile_infer", "x": 512, "d": 512, "m": 1},
        # a handful of tokens through a mapped layer of a transformer block (a decode step)
        {"name": "infer_768x3072_m16", "kind": "infer", "x": 768, "d": 3072, "m": 16, "scaled": True},
        # the single-tile training step the reference documents: forward, backward, pulsed update
        {"name": "step_256_b64", "kind": "step", "x": 256, "d": 256, "m": 64, "device": "constant",
         "pulse": "stochastic", "bias": False},
        # a small fully connected layer with an analog bias column and ragged sizes, small batch
        {"name": "step_ragged_785x130_b10", "kind": "step", "x": 785, "d": 130, "m": 10,
         "device": "softbounds", "pulse": "stochastic", "bias": True},
        # noise switched off and implicit pulses: the reproducible runs of a debugging session
        {"name": "step_det_512_b128", "kind": "step", "x": 512, "d": 512, "m": 128, "device": "constant",
         "pulse": "implicit", "bias": False},
        # Tiki-Taka: two batches, so that one transfer falls into a pass
        {"name": "tiki_1024_b256", "kind": "tiki", "x": 1024, "d": 1024, "m": 256},
        # the floating-point tile that the analog ones are compared against in training
        {"name": "fp_1024_b512", "kind": "fp", "x": 1024, "d": 1024, "m": 512},
        # training step of a layer mapped onto 512 x 512 tiles
        {"name": "mapped_step_1024_b256", "kind": "mapped_step", "x": 1024, "d": 1024, "m": 256},
        # 3 x 3 convolution of an ordinary layer, odd image sides, through the indexed interface
        {"name": "conv_64ch_15x17_b12", "kind": "conv", "c": 64, "d": 64, "h": 15, "w": 17, "n": 12},
        # batched analog inference of a large mapped layer (64 tiles)
        {"name": "infer_4096_b8192", "kind": "infer", "x": 4096, "d": 4096, "m": 8192, "scaled": False},
        # the second MLP layer of a transformer block over a whole batch of sequences
        {"name": "infer_3072x768_b16384", "kind": "infer", "x": 3072, "d": 768, "m": 16384, "scaled": True},
        # 3 x 3 convolution, 256 channels, 128 images of 32 x 32: 131072 input columns per step
        {"name": "conv_256ch_32x32_b128", "kind": "conv", "c": 256, "d": 256, "h": 32, "w": 32, "n": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tile_infer", "infer", "infer", "step", "step", "tiki", "fp", "mapped_step", "conv", "conv"])
    if kind == "tile_infer":
        return {"kind": kind, "x": _log(rng, 32, 512), "d": _log(rng, 32, 512), "m": _log(rng, 1, 64)}
    if kind == "infer":
        x, d = _log(rng, 256, 4096), _log(rng, 256, 4096)
        m = _log(rng, 1, min(16384, max(2, (1 << 37) // (x * d))))
        return {"kind": kind, "x": x, "d": d, "m": m, "scaled": rng.random() < 0.5}
    if kind == "step":
        return {"kind": kind, "x": _log(rng, 24, 1024), "d": _log(rng, 10, 1024), "m": _log(rng, 4, 1024),
                "device": rng.choice(["constant", "softbounds", "softref"]),
                "pulse": rng.choice(["stochastic", "stochastic", "implicit"]), "bias": rng.random() < 0.3}
    if kind in ("tiki", "mapped_step"):
        return {"kind": kind, "x": _log(rng, 200, 1280), "d": _log(rng, 200, 1280), "m": _log(rng, 16, 512)}
    if kind == "fp":
        return {"kind": kind, "x": _log(rng, 64, 2048), "d": _log(rng, 64, 2048), "m": _log(rng, 8, 1024)}
    c, d = _log(rng, 16, 256), _log(rng, 16, 256)
    h, w = rng.randint(7, 32), rng.randint(7, 32)
    n = max(1, min(128, _log(rng, 4, 128), (1 << 36) // (9 * c * d * h * w)))
    return {"kind": kind, "c": c, "d": d, "h": h, "w": w, "n": n}


# ---- configurations ---------------------------------------------------------------------------


def _inference_parameter():
    # 8-bit DAC and ADC, output noise and additive weight noise, abs-max noise management
    p = D.AnalogTileParameter()
    io = p.forward_io
    io.inp_res = io.out_res = 1.0 / 254.0
    io.out_noise, io.w_noise = 0.04, 0.0175
    io.w_noise_type = D.WeightNoiseType.AdditiveConstant
    io.out_bound, io.inp_bound = 10.0, 1.0
    io.noise_management = D.NoiseManagementType.AbsMax
    io.bound_management = D.BoundManagementType.None_
    p.update.pulse_type = D.PulseType.None_
    return p


def _training_parameter(noisy=True, pulse="stochastic"):
    # 7-bit DAC, 9-bit ADC, output noise, iterative bound management, 31 pulse slots
    p = D.AnalogTileParameter()
    for io in (p.forward_io, p.backward_io):
        io.inp_res, io.out_res = 1.0 / 126.0, 1.0 / 510.0
        io.out_noise, io.out_bound, io.inp_bound = (0.06 if noisy else 0.0), 12.0, 1.0
        io.noise_management = D.NoiseManagementType.AbsMax
    p.forward_io.bound_management = D.BoundManagementType.Iterative
    p.update.pulse_type = (D.PulseType.StochasticCompressed if pulse == "stochastic"
                           else D.PulseType.DeterministicImplicit)
    p.update.desired_bl = 31
    return p


def _device(name, seed, noisy=True):
    dev = {"constant": D.ConstantStepResistiveDeviceParameter,
           "softbounds": D.SoftBoundsResistiveDeviceParameter,
           "softref": D.SoftBoundsReferenceResistiveDeviceParameter}[name]()
    dev.dw_min, dev.dw_min_dtod, dev.dw_min_std = 0.001, 0.3, (0.3 if noisy else 0.0)
    dev.w_max, dev.w_min = 0.6, -0.6
    if name == "softref":
        dev.dw_min, dev.w_max, dev.w_min, dev.reference_std = 0.002, 1.0, -1.0, 0.05
    dev.enforce_consistency = True
    dev.construction_seed = 1 + seed % 100003
    return dev


def _tile(config, seed, w_dx, lr):
    """A tile on the GPU whose weights ``[x, d]`` live in a tensor of the caller."""
    tile = T.AnalogTile(config, cuda_device=0)
    shared = torch.empty(w_dx.size(1), w_dx.size(0), device="cuda")
    tile.set_shared_weights(shared)
    tile.set_seed(seed)
    tile.set_weights(w_dx)
    tile.set_learning_rate(lr)
    return tile, shared


# ---- what a program has in hand ---------------------------------------------------------------


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda") * 2 - 1

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    kind = case["kind"]
    s = {"kind": kind}
    if kind == "conv":
        c, d, h, w, n = (case[k] for k in ("c", "d", "h", "w", "n"))
        x = 9 * c
        config = _training_parameter()._config(x, d, _device("softbounds", seed), seed=seed % 1000003)
        s["tile"], s["w"] = _tile(config, seed, 0.5 * rand(d, x), 0.01)
        # the index array a padded 3 x 3 convolution layer hands to its tile
        index = F.unfold(torch.arange(2, c * h * w + 2, dtype=torch.float64).reshape(1, c, h, w),
                         kernel_size=3, padding=1).flatten().round().to(torch.int32).cuda()
        s["tile"].set_matrix_indices(index)
        s["x"] = torch.relu(randn(n, c, h, w))
        s["d"] = 0.01 * randn(n, d, h, w)
        s["y"], s["g"] = torch.empty_like(s["d"]), torch.empty_like(s["x"])
        return s

    x, d, m = case["x"], case["d"], case["m"]
    if kind in ("infer", "tile_infer"):
        s["x"] = randn(m, x)
        w = randn(d, x) / math.sqrt(x)
        if kind == "tile_infer":
            config = _inference_parameter()._config(x, d, D.IdealResistiveDeviceParameter(), seed=seed % 1000003)
            s["tile"], s["w"] = _tile(config, seed, w, 0.0)
            return s
        config = _inference_parameter()._config(512, 512, D.IdealResistiveDeviceParameter(), seed=seed % 1000003)
        s["layer"] = T.TileArray(config, d, x, 512, 512, cuda_device=0)
        s["layer"].set_seed(seed)
        if case["scaled"]:
            # every tile fills its conductance range; digital output scales and a digital bias
            s["layer"].set_weights(w, weight_scaling_omega=1.0)
            s["layer"].set_bias(0.1 * randn(d))
        else:
            s["layer"].set_weights(w)
        return s

    if kind == "fp":
        s["x"], s["d"] = rand(m, x), 0.1 * randn(m, d)
        tile = T.FloatingPointTile(x, d, cuda_device=0)
        s["w"] = torch.empty(x, d, device="cuda")
        tile.set_shared_weights(s["w"])
        tile.set_weights(0.5 * rand(d, x))
        tile.set_learning_rate(0.01)
        s["tile"] = tile
        return s

    if kind == "tiki":
        dev = D.TransferResistiveDeviceParameter()
        for _ in range(2):
            dev.append_parameter(_device("softref", seed))
        dev.construction_seed = 1 + seed % 100003
        dev.gamma, dev.transfer_every, dev.units_in_mbatch = 0.0, 2.0, True
        dev.n_reads_per_transfer, dev.transfer_lr, dev.fast_lr = 1, 1.0, 1.0
        dev.transfer_forward.bound_management = D.BoundManagementType.Iterative
        config = _training_parameter()._config(x, d, dev, seed=seed % 1000003)
        s["tile"], s["w"] = _tile(config, seed, torch.zeros(d, x), 0.01)
        s["x"], s["d"] = rand(2, m, x), 0.05 * randn(2, m, d)
        return s

    if kind == "mapped_step":
        config = _training_parameter()._config(512, 512, _device("softbounds", seed), seed=seed % 1000003)
        layer = T.TileArray(config, d, x, 512, 512, cuda_device=0)
        layer.set_seed(seed)
        layer.set_weights(0.5 * rand(d, x))
        layer.set_learning_rate(0.01)
        s["layer"], s["x"], s["d"] = layer, rand(m, x), 0.05 * randn(m, d)
        return s

    noisy = case["pulse"] == "stochastic"
    config = _training_parameter(noisy, case["pulse"])._config(x, d, _device(case["device"], seed, noisy),
                                                               seed=seed % 1000003)
    s["tile"], s["w"] = _tile(config, seed, 0.5 * rand(d, x), 0.01)
    s["bias"] = bool(case["bias"])
    s["x"], s["d"] = rand(m, x - int(s["bias"])), 0.1 * randn(m, d)
    return s


# ---- one pass ---------------------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind == "infer":
        return s["layer"].forward(s["x"], is_test=True, non_blocking=True)
    if kind == "tile_infer":
        return s["tile"].forward(s["x"], is_test=True, non_blocking=True)
    if kind == "conv":
        t = s["tile"]
        t.forward_indexed(s["x"], s["y"], non_blocking=True)
        t.backward_indexed(s["d"], s["g"], non_blocking=True)
        t.update_indexed(s["x"], s["d"], non_blocking=True)
        return s["y"], s["g"], s["w"]
    if kind == "mapped_step":
        # the tiles of a mapped layer own their weights; the next pass reads the updated ones
        layer = s["layer"]
        y = layer.forward(s["x"], is_test=False, non_blocking=True)
        g = layer.backward(s["d"], non_blocking=True)
        layer.update(s["x"], s["d"], non_blocking=True)
        y2 = layer.forward(s["x"], is_test=False, non_blocking=True)
        return y, g, y2
    if kind == "tiki":
        t, out = s["tile"], []
        for k in range(2):
            out.append(t.forward(s["x"][k], non_blocking=True))
            out.append(t.backward(s["d"][k], non_blocking=True))
            t.update(s["x"][k], s["d"][k], non_blocking=True)
        return out + [s["w"]]
    t, bias = s["tile"], s.get("bias", False)
    y = t.forward(s["x"], bias, non_blocking=True)
    g = t.backward(s["d"], bias, non_blocking=True)
    t.update(s["x"], s["d"], bias, non_blocking=True)
    return y, g, s["w"]


def work(case):
    kind = case["kind"]
    if kind == "conv":
        x, d = 9 * case["c"], case["d"]
        cols = case["n"] * case["h"] * case["w"]
        io = 4 * cols * (case["c"] + d)  # images in or out once per pass, not the unfolded matrix
        return {"bytes": 3 * io + 4 * x * d * (2 + 2 + 6), "flops": 3 * 2.0 * cols * x * d}
    x, d, m = case["x"], case["d"], case["m"]
    one = {"bytes": 4 * m * (x + d) + 4 * x * d, "flops": 2.0 * m * x * d}
    if kind in ("infer", "tile_infer"):
        return one
    # forward, backward, update (weights read and written; analog devices: bounds and step sizes
    # of every element too)
    par = 0 if kind == "fp" else 16 if case.get("device") == "constant" else 24
    upd = {"bytes": 4 * m * (x + d) + x * d * (8 + par), "flops": 2.0 * m * x * d}
    passes = 3 if kind == "mapped_step" else 2
    step = {k: passes * one[k] + upd[k] for k in ("bytes", "flops")}
    return {k: 2 * v for k, v in step.items()} if kind == "tiki" else step


def tolerance(case):
    if case["kind"] == "fp":
        # 32-bit sums of up to 2048 terms: 6e-7 seen against 64 bits
        return {"rel": 3e-6}
    # Another order of the 32-bit sums in front of the ADC moves a few codes by one step: 1e-4 to
    # 7e-4 seen between the two kernels for the products (one step is up to 0.23 of the outputs'
    # root mean square). The draws are fixed by the seed and the updates change in the last bit only.
    return {"rel": 3e-3, "max": 0.9}


# ---- the same numbers in 64 bits --------------------------------------------------------------


def _quantise(v, res):
    return torch.round(v / res) * res


def _analog_mvm(inp, w, bm):
    """DAC with abs-max scaling, product, ADC with clipping; ``bm``: rows that clipped are repeated
    with half the input scale until they do not."""
    f32 = torch.float32
    bound = 12.0  # the resolutions are 32-bit parameters of the tile
    inp_res = float(torch.tensor(1.0 / 126.0, dtype=f32) * 2.0)
    out_res = float(torch.tensor(1.0 / 510.0, dtype=f32) * (2.0 * bound))
    amax = inp.abs().amax(dim=1, keepdim=True)
    scale = torch.where(amax > 0, 1.0 / amax, torch.zeros_like(amax))
    out, red = None, torch.ones_like(amax)
    for _ in range(10 if bm else 1):
        v = _quantise(inp * scale / red, inp_res).clamp(-1.0, 1.0)
        y = _quantise(v @ w, out_res)
        over = (y.to(f32).abs() > bound).any(dim=1, keepdim=True)
        out = y.clamp(-bound, bound) * torch.where(amax > 0, amax, torch.zeros_like(amax)) * red
        if not bm or not bool(over.any()):
            break
        red = torch.where(over, red * 2, red)
    return out


def exact(case, seed):
    """Values exist where no noise is drawn: the floating-point tile, and constant-step devices with
    implicit pulses. The device parameters of the elements are inputs and are read from the tile."""
    if case["kind"] == "fp":
        s = prepare(case, seed)
        x, d, w = s["x"].double(), s["d"].double(), s["w"].double()
        return x @ w, d @ w.t(), w - 0.01 * (x.t() @ d)
    if case["kind"] != "step" or case["pulse"] != "implicit" or case["bias"] or case["device"] != "constant":
        return None
    s = prepare(case, seed)
    x, d, w = s["x"].double(), s["d"].double(), s["w"].double()
    y, g = _analog_mvm(x, w, True), _analog_mvm(d, w.t().contiguous(), False)
    names = s["tile"].get_hidden_parameter_names()
    hidden = s["tile"].get_hidden_parameters().cuda().double().transpose(1, 2)
    hi, lo, up, down = (hidden[names.index(k)] for k in ("max_bound", "min_bound", "dwmin_up", "dwmin_down"))
    lr, dw_min, bl_max = 0.01, 0.001, 31
    for k in range(case["m"]):
        xm, dm = x[k].abs().max(), d[k].abs().max()
        strength = float(lr * xm * dm / dw_min)
        bl = min(math.ceil(strength), bl_max)
        if bl == 0:
            continue
        unit = math.sqrt(lr / (dw_min * bl))
        ratio = float((xm / (dm * (bl_max / strength if strength > bl_max else 1.0))).sqrt())
        px = (x[k] * (unit / ratio)).clamp(-1.0, 1.0)
        pd = (d[k] * (unit * ratio)).clamp(-1.0, 1.0) * bl
        n = torch.round(px[:, None] * pd[None, :])
        # pulses of one sign on one element: the clip after each is the clip after all
        w = torch.minimum(torch.maximum(w - n * torch.where(n > 0, down, up), lo), hi)
    return y, g, w
