"""The work that users of this framework have it do, as cases to measure.

Every case goes through the public ops of ``rexsc_b200.ops``, with the argument lists that the front end of SC
networks passes: activations between 0 and 1 on a 7-bit grid (about half of them zero, as behind BatchNorm and
Hardtanh), weights N(0, 0.1) on a 7-bit grid, XNOR generators, progressive loading (7, 8, 1).

Families (``"kind"`` of a case):

  conv    one SC conv2d forward, ``conv2d_generic_general_split_acc``: counts of the positive and the negative stream
  net     the SC layers of a whole network, one after the other: per layer the conv forward, its counts as values and
          the OR-n activations of the two guide sums, which is what a forward pass with bit streams calls
  linear  two SC linear layers, ``linear_generic_general_acc``
  fxp     the four fixed-point convs of TinyConv, ``conv2d_saturate_acc``
  train   the point-wise passes of a layer in training: calibrated activation with error injection forward and
          backward, OR-n activation forward and backward
  calib   a calibration step's passes over a layer: conv counts, counts to values, window statistics
"""
import math

import torch

from rexsc_b200 import ops

PROG = (7, 8, 1)
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


# ---- shapes ---------------------------------------------------------------------------------------------------
def _resnet_layers(blocks):
    """(c_in, size, c_out, kernel, stride, pad, repeats) of the SC convs of a BasicBlock ResNet at 224x224."""
    out, cin, h = [], 64, 56
    for stage, (cout, n) in enumerate(zip((64, 128, 256, 512), blocks)):
        if stage == 0:
            out.append((64, 56, 64, 3, 1, 1, 2 * n))
            continue
        out.append((cin, h, cout, 3, 2, 1, 1))
        out.append((cin, h, cout, 1, 2, 0, 1))
        h //= 2
        out.append((cout, h, cout, 3, 1, 1, 2 * n - 1))
        cin = cout
    return out


_VGG = [(3, 32, 64), (64, 32, 64), (64, 16, 128), (128, 16, 128), (128, 8, 256), (256, 8, 256), (256, 8, 256),
        (256, 4, 512), (512, 4, 512), (512, 4, 512), (512, 2, 512), (512, 2, 512), (512, 2, 512)]
NETS = {
    "resnet18": dict(layers=_resnet_layers((2, 2, 2, 2)), or_n=2, L=32, nhwc=True, dtype="f16", guide="f16"),
    "vgg16": dict(layers=[(ci, h, co, 3, 1, 1, 1) for ci, h, co in _VGG], or_n=1, L=32, nhwc=False, dtype="f32",
                  guide="f32"),
}


def _tinyconv(size):
    """(c_in, size, c_out, kernel, pad, input precision) of TinyConv's four fixed-point convs on size x size images."""
    return [(3, size, 32, 5, 2, 5), (32, size // 2, 32, 5, 2, 5), (32, size // 4, 64, 5, 2, 5),
            (64, size // 8, 10, size // 8, 0, 7)]


def _conv(name, n, c, h, w, co, k, stride, pad, own_pad, dtype, nhwc, L, or_n):
    """``own_pad``: the op pads; otherwise the caller has padded before the call, as the front end does."""
    case = dict(kind="conv", n=n, c=c, h=h, w=w, co=co, k=k, stride=stride, pad=pad, own_pad=own_pad, dtype=dtype,
                nhwc=nhwc, L=L, or_n=or_n)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # one layer of a small CIFAR net at a small batch: RGB input, 25-tap filter, NCHW float activations
        _conv("conv5x5_rgb_b32", 32, 3, 32, 32, 32, 5, 1, 2, True, "f32", False, 32, 1),
        # inference of one image, 19 SC convs: what latency and the number of launches decide
        dict(name="resnet18_b1", kind="net", net="resnet18", batch=1),
        # the first stage of SC ResNet-18 at its training batch: 64 channels, the largest maps
        _conv("conv_64_56_b256", 256, 64, 56, 56, 64, 3, 1, 1, False, "f16", True, 32, 2),
        # first conv of a stage: 3x3 with stride 2
        _conv("conv_128_28_s2_b256", 256, 128, 28, 28, 256, 3, 2, 1, False, "f16", True, 32, 2),
        # the last stage: 512 channels on 7x7 maps
        _conv("conv_512_7_b256", 256, 512, 7, 7, 512, 3, 1, 1, False, "f16", True, 32, 2),
        # SC ResNet-34 at batch 192: 64-bit streams, OR-3
        _conv("conv_256_14_L64_b192", 192, 256, 14, 14, 256, 3, 1, 1, False, "f16", True, 64, 3),
        # odd sizes everywhere, NCHW bf16, the op pads
        _conv("conv_ragged_b37", 37, 100, 27, 29, 130, 3, 1, 1, True, "bf16", False, 32, 1),
        # SC VGG-16 on CIFAR images at its training batch, NCHW float: 13 convs and their activations
        dict(name="vgg16_b256", kind="net", net="vgg16", batch=256),
        # the SC classifier: 128-bit streams
        dict(name="linear_512_b256", kind="linear", rows=256, c=512, hidden=512, out=10, L=128, or_n=1, dtype="f32"),
        # fixed-point TinyConv at its training batch
        dict(name="fxp_tinyconv_b256", kind="fxp", n=256, size=32, dtype="f32"),
        # a layer of a calibrated training step: the point-wise passes, both directions, fp16 autocast
        dict(name="train_64_56_b256", kind="train", n=256, c=64, h=56, w=56, dtype="f16", nhwc=True, or_n=2),
        # a calibration step on a second-stage layer, half the training batch
        dict(name="calib_128_28_b128", kind="calib", n=128, c=128, h=28, w=28, co=128, dtype="f16", L=32, or_n=2),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


# most work of a drawn conv: bit operations on the tensor-core range (C >= 32 and at most 9 taps), and outside it
_MOST_WIDE, _MOST_THIN = 1.2e12, 6.0e10


def draw(rng):
    kind = rng.choice(["conv"] * 5 + ["net", "linear", "fxp", "train", "calib"])
    if kind == "conv":
        k = rng.choice([1, 3, 3, 3, 5])
        c = 3 if k == 5 and rng.random() < 0.5 else _log_int(rng, 8, 64) if k == 5 else _log_int(rng, 32, 512)
        stride = rng.choice([1, 1, 2])
        h = _log_int(rng, 4, 56)
        case = _conv(None, _log_int(rng, 1, 256), c, h, max(k, h + rng.randint(-2, 2)), _log_int(rng, 10, 512), k, stride,
                     k // 2, rng.random() < 0.5, rng.choice(["f32", "f16", "bf16"]), rng.random() < 0.6,
                     rng.choice([32, 32, 64, 128]), rng.choice([1, 2, 2, 3]))
        case["h"] = max(case["h"], k)
        most = _MOST_WIDE if c >= 32 and k <= 3 else _MOST_THIN
        while case["n"] > 1 and work(case)["flops"] > most:
            case["n"] = (case["n"] + 1) // 2
        while case["co"] > 10 and work(case)["flops"] > most:
            case["co"] = (case["co"] + 1) // 2
        return case
    if kind == "net":
        net = rng.choice(["resnet18", "vgg16"])
        return dict(kind="net", net=net, batch=_log_int(rng, 1, {"resnet18": 48, "vgg16": 200}[net]))
    if kind == "linear":
        return dict(kind="linear", rows=_log_int(rng, 1, 512), c=_log_int(rng, 40, 1024), hidden=_log_int(rng, 40, 1024),
                    out=rng.choice([10, 100]), L=rng.choice([32, 64, 128]), or_n=rng.choice([1, 2]),
                    dtype=rng.choice(["f32", "f16"]))
    if kind == "fxp":
        return dict(kind="fxp", n=_log_int(rng, 1, 256), size=rng.randint(16, 47), dtype=rng.choice(["f32", "f16"]))
    h = _log_int(rng, 7, 56)
    if kind == "train":
        return dict(kind="train", n=_log_int(rng, 1, 200), c=_log_int(rng, 10, 64), h=h, w=max(3, h + rng.randint(-2, 2)),
                    dtype=rng.choice(["f16", "f16", "f32"]), nhwc=rng.random() < 0.5, or_n=rng.choice([1, 2, 3]))
    return dict(kind="calib", n=_log_int(rng, 1, 64), c=_log_int(rng, 32, 128), h=h, w=h, co=_log_int(rng, 10, 128),
                dtype=rng.choice(["f16", "f32"]), L=rng.choice([32, 64]), or_n=rng.choice([1, 2, 3]))


# ---- inputs ---------------------------------------------------------------------------------------------------
def _activations(g, shape, dtype):
    x = torch.randn(shape, device="cuda", generator=g).mul_(0.45).clamp_(0, 1)
    return x.mul_(128).round_().clamp_(max=127).div_(128).to(dtype)


def _weights(g, shape):
    return torch.randn(shape, device="cuda", generator=g).mul_(0.1 * 128).round_().clamp_(-127, 127).div_(128)


def _sums(g, shape, dtype):
    """Guide sums of one sign: non-negative, mostly around one."""
    return torch.randn(shape, device="cuda", generator=g).mul_(0.8).add_(1.0).abs_().to(dtype)


def _format(t, nhwc):
    return t.contiguous(memory_format=torch.channels_last if nhwc else torch.contiguous_format)


def _out(size, k, stride, pad):
    return (size + 2 * pad - k) // stride + 1


def _conv_inputs(g, n, c, h, w, co, k, pad, own_pad, dtype, nhwc):
    x = _activations(g, (n, c, h, w), dtype)
    if pad and not own_pad:
        x = torch.nn.functional.pad(x, (pad, pad, pad, pad))
    return _format(x, nhwc), _format(_weights(g, (co, c, k, k)), nhwc)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "conv":
        x, w = _conv_inputs(g, case["n"], case["c"], case["h"], case["w"], case["co"], case["k"], case["pad"],
                            case["own_pad"], DTYPES[case["dtype"]], case["nhwc"])
        p = case["pad"] if case["own_pad"] else 0
        return dict(kind=kind, x=x, w=w, L=case["L"], pad=(p, p), stride=(case["stride"],) * 2, bin=case["or_n"] - 1)
    if kind == "net":
        net = NETS[case["net"]]
        calls = []
        for ci, h, co, k, s, p, rep in net["layers"]:
            x, w = _conv_inputs(g, case["batch"], ci, h, h, co, k, p, False, DTYPES[net["dtype"]], net["nhwc"])
            oh = _out(h, k, s, p)
            guide = [_format(_sums(g, (case["batch"], co, oh, oh), DTYPES[net["guide"]]), net["nhwc"]) for _ in range(2)]
            calls += [(x, w, (s, s), guide)] * rep
        return dict(kind=kind, calls=calls, L=net["L"], or_n=net["or_n"], dtype=DTYPES[net["dtype"]])
    if kind == "linear":
        x = _activations(g, (case["rows"], case["c"]), DTYPES[case["dtype"]])
        x2 = _activations(g, (case["rows"], case["hidden"]), DTYPES[case["dtype"]])
        return dict(kind=kind, layers=[(x, _weights(g, (case["hidden"], case["c"]))),
                                       (x2, _weights(g, (case["out"], case["hidden"])))],
                    L=case["L"], bin=case["or_n"] - 1)
    if kind == "fxp":
        layers = []
        for ci, h, co, k, p, prec in _tinyconv(case["size"]):
            x = torch.randn((case["n"], ci, h, h), device="cuda", generator=g).mul_(0.45).clamp_(0, 1)
            x = x.mul_(2 ** prec).round_().clamp_(max=2 ** prec - 1).div_(2 ** prec).to(DTYPES[case["dtype"]])
            layers.append((x, _weights(g, (co, ci, k, k)), prec, p))
        return dict(kind=kind, layers=layers)
    shape = (case["n"], case["c"], case["h"], case["w"])
    if kind == "train":
        dt = DTYPES[case["dtype"]]
        return dict(kind=kind, pos=_format(_sums(g, shape, dt), case["nhwc"]), neg=_format(_sums(g, shape, dt), case["nhwc"]),
                    grad=_format(torch.randn(shape, device="cuda", generator=g), case["nhwc"]), or_n=case["or_n"],
                    bias=torch.tensor([0.002, -0.03, 0.02, -0.01, 0.003, -0.0005], device="cuda"),
                    std=torch.tensor([0.01, 0.06, -0.03, 0.01, -0.002, 0.0002], device="cuda"))
    x, w = _conv_inputs(g, case["n"], case["c"], case["h"], case["w"], case["co"], 3, 1, False, DTYPES[case["dtype"]], True)
    out = (case["n"], case["co"], case["h"], case["w"])
    # float guides of the two signs: what the OR-n activation returned for the guide convs (between 0 and n)
    guide = [_format(_sums(g, out, torch.float32).clamp_(max=case["or_n"]), True) for _ in range(2)]
    return dict(kind=kind, x=x, w=w, guide=guide, L=case["L"], bin=case["or_n"] - 1, dtype=DTYPES[case["dtype"]])


# ---- one pass -------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "conv":
        return ops.conv2d_generic_general_split_acc(state["x"], state["w"], state["L"], -1, 16, state["pad"], state["stride"],
                                                    PROG, state["bin"], 1, True, False)
    if kind == "net":
        out, n = [], state["or_n"]
        for x, w, stride, guide in state["calls"]:
            pos, neg = ops.conv2d_generic_general_split_acc(x, w, state["L"], -1, 16, (0, 0), stride, PROG, n - 1, 1, True,
                                                            False)
            out += [ops.sc_counts_to_value(pos, neg, state["L"], state["dtype"], split=False, diff=True),
                    ops.or_approx_n_forward_acc(guide[0], n), ops.or_approx_n_forward_acc(guide[1], n)]
        return out
    if kind == "linear":
        out = []
        for x, w in state["layers"]:
            out += ops.linear_generic_general_acc(x, w, PROG, state["L"], -1, state["bin"], 1, False, False)
        return out
    if kind == "fxp":
        return [ops.conv2d_saturate_acc(x, w, 0, prec, 24, (p, p), (1, 1)) for x, w, prec, p in state["layers"]]
    if kind == "train":
        ops.manual_seed(20)  # the same noise for the same inputs
        n, pos, neg, grad = state["or_n"], state["pos"], state["neg"], state["grad"]
        return [ops.or_approx_n_forward_bias_std_both_acc(pos, neg, state["bias"], state["std"], n),
                *ops.or_approx_n_backward_bias_std_both_acc(grad, pos, neg, state["bias"], n),
                ops.or_approx_n_forward_acc(pos, n), ops.or_approx_n_backward_acc(grad, pos, n)]
    pos, neg = ops.conv2d_generic_general_split_acc(state["x"], state["w"], state["L"], -1, 16, (0, 0), (1, 1), PROG,
                                                    state["bin"], 1, True, False)
    values = ops.sc_counts_to_value(pos, neg, state["L"], state["dtype"], split=True, diff=True)
    stats = ops.sc_calib_stats(pos, neg, state["guide"][0], state["guide"][1], state["L"],
                               counts_via_half=state["dtype"] == torch.float16)
    return [pos, neg, *values, stats]


# ---- what a pass cannot do without ----------------------------------------------------------------------------
def _conv_work(n, c, h, w, co, k, stride, pad, stored_pad, act_bytes, L):
    """Activations (with the border that the caller stores) and weights in, two int16 counts out; per useful product
    and time slot one AND and one count: every weight is in one of the two streams."""
    oh, ow = _out(h, k, stride, pad), _out(w, k, stride, pad)
    outs = n * co * oh * ow
    return dict(bytes=n * c * (h + 2 * stored_pad) * (w + 2 * stored_pad) * act_bytes + co * c * k * k * 4 + outs * 4,
                flops=2 * L * outs * c * k * k)


def work(case):
    kind = case["kind"]
    size = 4 if case.get("dtype") == "f32" else 2
    if kind == "conv":
        return _conv_work(case["n"], case["c"], case["h"], case["w"], case["co"], case["k"], case["stride"], case["pad"],
                          0 if case["own_pad"] else case["pad"], size, case["L"])
    if kind == "net":
        net = NETS[case["net"]]
        size, gsize = (4 if net[f] == "f32" else 2 for f in ("dtype", "guide"))
        total = dict(bytes=0, flops=0)
        for ci, h, co, k, s, p, rep in net["layers"]:
            one = _conv_work(case["batch"], ci, h, h, co, k, s, p, p, size, net["L"])
            outs = case["batch"] * co * _out(h, k, s, p) ** 2
            # of the counts only the value has to leave the layer
            total["bytes"] += rep * (one["bytes"] + outs * (size - 4) + 2 * outs * (gsize + 4))
            total["flops"] += rep * (one["flops"] + 2 * outs * 6)
        return total
    if kind == "linear":
        rows, c, hid, out = case["rows"], case["c"], case["hidden"], case["out"]
        return dict(bytes=rows * (c + hid) * size + (hid * c + out * hid) * 4 + rows * (hid + out) * 4,
                    flops=2 * case["L"] * rows * (c * hid + hid * out))
    if kind == "fxp":
        total = dict(bytes=0, flops=0)
        for ci, h, co, k, p, _ in _tinyconv(case["size"]):
            outs = case["n"] * co * _out(h, k, 1, p) ** 2
            total["bytes"] += case["n"] * ci * h * h * size + co * ci * k * k * 4 + outs * 4
            total["flops"] += 2 * outs * ci * k * k
        return total
    elems = case["n"] * case.get("co", case["c"]) * case["h"] * case["w"]
    if kind == "train":
        # pos and neg read once, grad once; calibrated output, its two gradients, activation and its gradient written
        return dict(bytes=elems * (2 * size + 4 + 5 * 4), flops=elems * 150)
    conv = _conv_work(case["n"], case["c"], case["h"], case["w"], case["co"], 3, 1, 1, 1, size, case["L"])
    # two guides in, three value tensors out (the counts are results that the later passes find written)
    return dict(bytes=conv["bytes"] + elems * (2 * 4 + 3 * size), flops=conv["flops"] + elems * 40)


def tolerance(case):
    kind = case["kind"]
    if kind in ("conv", "linear", "fxp"):
        return "exact"
    # Single-precision chains with the hardware's exp.  Against the same formulas in float64: activations off by
    # 1.1e-7 (largest difference 4.1e-7), the train passes by 2.0e-7 (2.0e-6); four times that is allowed.
    if kind == "net":
        return {"rel": 5e-7, "max": 2e-6}
    if kind == "train":
        return {"rel": 8e-7, "max": 8e-6}
    # Window sums of single-precision differences, partial sums per thread in float32, double beyond them: off by
    # 6.1e-9 (1.2e-8) from float64; sums of another split of the elements differ by about as much.
    return {"rel": 1e-7, "max": 1e-6}
