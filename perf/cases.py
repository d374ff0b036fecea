"""Timed cases: the work that a program built on this framework has it do, through the public entry points.

    listed()          the standing cases
    draw(rng)         one more case of the same ranges
    prepare(case, s)  what the program holds before the call: inputs made from seed s, model, weights
    run(state)        one pass, as the program calls it; returns its outputs
    work(case)        bytes and operations that the pass cannot do without
    tolerance(case)   how far another correct implementation may be off

Kinds of a case:
    net         a Bi-Real-18-shaped `Net` (float stem, 16 binary blocks, float classifier) on a batch of images that lie
                in device memory ("device"), in an ordinary numpy array ("host") or in pinned memory ("pinned")
    binconv     the BinConv operator: fp32 activations in, fp32 mismatch counts out
    bconv       a binary convolution on packed bits, counts out
    block       a binary convolution with its affine, its shortcut and the next layer's packed signs
    pack_bgemm  fp32 rows packed along K, then multiplied with packed weights
    fconv       a float convolution
"""
import functools

import torch

from dabnn_b200 import ops
from dabnn_b200.bireal import OUTPUT_BLOB, build_bireal18
from dabnn_b200.dab_format import write_dab
from dabnn_b200.net import Net

WIDTHS = (64, 128, 256, 512)   # channels of the network's four stages


def listed():
    return [
        # one photo from the application's own array to its logits: the reference's only use of a network
        {"name": "net_host_image", "kind": "net", "feed": "host", "batch": 1, "hw": 224, "classes": 1000},
        # a server's small batch, images already decoded on the GPU
        {"name": "net_device_64", "kind": "net", "feed": "device", "batch": 64, "hw": 224, "classes": 1000},
        # offline scoring: the large batch of the throughput benchmark
        {"name": "net_device_1024", "kind": "net", "feed": "device", "batch": 1024, "hw": 224, "classes": 1000},
        # a server fed over PCIe: pinned images in, logits back in pinned memory
        {"name": "net_pinned_256", "kind": "net", "feed": "pinned", "batch": 256, "hw": 224, "classes": 1000},
        # a batch that fills no tile evenly, at another resolution and with a small classifier
        {"name": "net_device_37_160px", "kind": "net", "feed": "device", "batch": 37, "hw": 160, "classes": 100},
        # one layer on one image: the smallest call, and the first of the benchmark's workloads
        {"name": "binconv_image", "kind": "binconv", "n": 1, "h": 56, "w": 56, "cin": 64, "cout": 64, "k": 3, "stride": 1, "pad": 1},
        # a downsampling layer on a batch, from float activations
        {"name": "binconv_64_stride2", "kind": "binconv", "n": 64, "h": 28, "w": 28, "cin": 128, "cout": 256, "k": 3, "stride": 2, "pad": 1},
        # a residual block between two binary layers of a network that keeps its activations packed
        {"name": "block_256", "kind": "block", "n": 256, "h": 28, "w": 28, "cin": 128, "cout": 128, "k": 3, "stride": 1, "pad": 1},
        # a pointwise binary layer: few operations for each output
        {"name": "bconv_1x1_256", "kind": "bconv", "n": 256, "h": 14, "w": 14, "cin": 256, "cout": 512, "k": 1, "stride": 1, "pad": 0},
        # pack + GEMM of one image's im2col rows, M below a tile
        {"name": "pack_bgemm_image", "kind": "pack_bgemm", "m": 49, "n": 512, "bits": 4608},
        # the same of a batch of the first stage's images
        {"name": "pack_bgemm_256", "kind": "pack_bgemm", "m": 802816, "n": 64, "bits": 576},
        # a layer that a mixed network leaves in float
        {"name": "fconv_64", "kind": "fconv", "n": 64, "h": 28, "w": 28, "cin": 128, "cout": 128, "k": 3, "stride": 1, "pad": 1},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _draw_net(rng, feed):
    hw = rng.choice((64, 96, 128, 160, 192, 224, 256))   # the strides of the four stages want multiples of 32
    most = {"host": 16, "pinned": 256, "device": 1024}[feed]
    batch = _log_int(rng, 1, min(2 * most, most * 224 * 224 // (hw * hw)))
    return {"kind": "net", "feed": feed, "batch": batch, "hw": hw, "classes": rng.choice((10, 100, 365, 1000))}


def _draw_conv(rng, kind):
    while True:
        k = rng.choice((1, 3, 3, 3, 5))
        h = _log_int(rng, 7, 80)
        w = max(7, min(80, h + rng.choice((0, 0, 0, -2, -1, 1, 3, 8))))
        if kind == "fconv":
            cin, cout = rng.choice((3, 16, 32, 64, 96, 128, 256, 512)), 16 * rng.randint(1, 16)
        else:
            cin, cout = 64 * rng.choice((1, 1, 2, 2, 3, 4, 6, 8)), 16 * rng.randint(1, 32)
        if kind == "block":   # its signs leave as whole words
            cout = 64 * rng.randint(1, 8)
        case = {"kind": kind, "n": _log_int(rng, 1, 256), "h": h, "w": w, "cin": cin, "cout": cout, "k": k,
                "stride": rng.choice((1, 1, 1, 2)), "pad": k // 2}
        need = work(case)
        if need["bytes"] <= 1.7e9 and need["flops"] <= (6e10 if kind == "fconv" else 8e11):
            return case


def _draw_pack_bgemm(rng):
    while True:
        case = {"kind": "pack_bgemm", "m": _log_int(rng, 40, 802816), "n": rng.choice((16 * rng.randint(1, 32), rng.randint(10, 512))),
                "bits": 64 * _log_int(rng, 4, 72)}
        need = work(case)
        if need["bytes"] <= 2.3e9 and need["flops"] <= 8e11:
            return case


def draw(rng):
    kind = rng.choice(("host", "device", "device", "device", "pinned", "binconv", "binconv", "block", "bconv", "pack_bgemm", "pack_bgemm", "fconv"))
    if kind in ("host", "device", "pinned"):
        return _draw_net(rng, kind)
    return _draw_pack_bgemm(rng) if kind == "pack_bgemm" else _draw_conv(rng, kind)


# ---- what the program holds before the call -------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _model(hw, classes):
    """The model file's bytes (the parameters are the builder's own; only the images come from the seed)."""
    return write_dab(build_bireal18(image_hw=hw, num_classes=classes))


def _rand(shape, gen):
    return torch.rand(shape, device="cuda", generator=gen) * 2 - 1


def _words(shape, gen):
    return torch.randint(-2**63, 2**63 - 1, shape, device="cuda", dtype=torch.int64, generator=gen)


def _filters(cout, k, cin, gen):
    """Packed random signs as the converter lays them out: rows padded to 128 bits unless cin is 64."""
    words = k * k * cin // 64
    w = _words((cout, words), gen)
    if cin != 64 and words % 2:
        w = torch.cat([w, torch.zeros((cout, 1), device="cuda", dtype=torch.int64)], dim=1)
    return w.reshape(-1).contiguous()


def _out_hw(case):
    return tuple((case[d] + 2 * case["pad"] - case["k"]) // case["stride"] + 1 for d in ("h", "w"))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "net":
        net = Net.create()
        net.max_batch = case["batch"]
        net.read_buf(_model(case["hw"], case["classes"]))
        images = torch.randn((case["batch"], case["hw"], case["hw"], 3), device="cuda", generator=gen)
        state = {"case": case, "net": net}
        if case["feed"] == "device":
            state["images"] = images
        elif case["feed"] == "host":
            state["images"] = images.cpu().numpy()
        else:
            state["images"] = torch.empty(images.shape, pin_memory=True).copy_(images)
            state["logits"] = torch.zeros((case["batch"], case["classes"]), pin_memory=True)
        return state
    if case["kind"] == "pack_bgemm":
        m, n, words = case["m"], case["n"], case["bits"] // 64
        return {"case": case, "x": _rand((1, 1, m, case["bits"]), gen), "w": _words((words, n), gen), "c": torch.empty((m, n), device="cuda")}
    n, h, w, cin, cout, k = (case[d] for d in ("n", "h", "w", "cin", "cout", "k"))
    if case["kind"] == "fconv":
        weight = torch.randn((cout, k, k, cin), device="cuda", generator=gen) * (2.0 / (cin * k * k)) ** 0.5
        return {"case": case, "x": torch.randn((n, h, w, cin), device="cuda", generator=gen), "w": weight, "bias": 0.01 * _rand(cout, gen)}
    state = {"case": case, "w": _filters(cout, k, cin, gen)}
    state["x"] = _rand((n, h, w, cin), gen) if case["kind"] == "binconv" else _words((n, h, w, cin // 64), gen)
    if case["kind"] == "block":   # a folded BatchNorm over counts of mean K / 2, and a shortcut of its output's size
        scale = (torch.rand(cout, device="cuda", generator=gen) + 0.5) / (k * k * cin) ** 0.5
        state["a"], state["b"] = -2 * scale, k * k * cin * scale + 0.1 * _rand(cout, gen)
        state["shortcut"] = torch.randn((n, *_out_hw(case), cout), device="cuda", generator=gen)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "net":
        net = state["net"]
        if case["feed"] != "pinned":
            return net.run(state["images"]).get_blob(OUTPUT_BLOB)
        logits = state["logits"]
        net.wait(net.submit(state["images"].data_ptr(), case["batch"], OUTPUT_BLOB, logits.data_ptr(), logits.numel()))
        return logits
    if kind == "pack_bgemm":
        m, n, words = case["m"], case["n"], case["bits"] // 64
        bits = ops.pack_mat(state["x"])
        return ops.bgemm(n, m, words, state["w"], n, bits, words, state["c"].zero_(), n)   # bgemm adds to c
    k, pad, stride = case["k"], case["pad"], case["stride"]
    if kind == "fconv":
        return ops.fconv(state["x"], state["w"], state["bias"], pad, pad, stride, stride)
    layer = (state["x"], state["w"], case["cout"], k, k, pad, pad, stride, stride)
    if kind == "binconv":
        return ops.binconv_forward(*layer)
    if kind == "bconv":
        return ops.bconv(*layer)
    return ops.bconv_block(*layer, state["a"], state["b"], state["shortcut"], want_f32=True, want_bits=True)


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _net_work(batch, hw, classes):
    macs, params = (hw // 2) ** 2 * 64 * 147, 64 * 147 * 4
    size, cin = hw // 4, WIDTHS[0]
    for stage, cout in enumerate(WIDTHS):
        if stage:
            size //= 2
            macs += size * size * cout * cin              # the downsample branch's float 1x1
            params += cout * cin * 4
        for block in range(4):
            macs += size * size * cout * 9 * cin
            params += cout * 9 * cin // 8 + 2 * cout * 4
            cin = cout
    macs, params = macs + classes * cin, params + classes * (cin + 1) * 4
    return {"bytes": batch * (hw * hw * 3 + classes) * 4 + params, "flops": 2 * macs * batch}


def work(case):
    """Bytes: every input, weight and output once (bits as bits).  Operations: two for each multiply-accumulate, or for
    each xor and count of a pair of bits."""
    if case["kind"] == "net":
        return _net_work(case["batch"], case["hw"], case["classes"])
    if case["kind"] == "pack_bgemm":
        m, n, bits = case["m"], case["n"], case["bits"]
        return {"bytes": m * bits * 4 + n * bits / 8 + m * n * 4, "flops": 2 * m * n * bits}
    cin, cout, taps = case["cin"], case["cout"], case["k"] ** 2
    oh, ow = _out_hw(case)
    inputs, outputs = case["n"] * case["h"] * case["w"] * cin, case["n"] * oh * ow * cout
    read = inputs * 4 if case["kind"] in ("binconv", "fconv") else inputs / 8
    weights = cout * taps * cin * 4 if case["kind"] == "fconv" else cout * taps * cin / 8
    more = outputs * (4 + 1 / 8) if case["kind"] == "block" else 0   # the shortcut and the signs
    return {"bytes": read + weights + outputs * 4 + more, "flops": 2 * outputs * taps * cin}


def tolerance(case):
    if case["kind"] == "net":
        # The float layers agree to about 1e-5, but a residual sum that close to zero can take the other sign, and from
        # there on that image's logits are off by one or two per cent (seen on 4 of 24 images against the CPU checker).
        return {"rel": 0.02, "max": 0.2}
    if case["kind"] == "fconv":
        return {"rel": 1e-5}       # fp32 products and sums in another order
    return "exact"                 # whole counts; the block's affine and shortcut are each rounded once, in one order
