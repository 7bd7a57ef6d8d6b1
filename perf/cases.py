"""The work this library is asked to do, as calls of its public entry points.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes the
inputs, weights and handles of one, ``run`` is one pass through the library, ``work`` the bytes and
operations the pass cannot do without and ``exact`` the same result from plain torch in 64 bits.
All arithmetic is integer, so every implementation returns the same bytes.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

api = load_package().api

DEV = "cuda"


# ---- the cases ----------------------------------------------------------------------------------

def listed():
    return [
        # one camera frame through MobileNetV1: the latency a single request sees
        dict(name="mobilenet_b1", op="net", batch=1, bits=32, host=False),
        # a serving batch of whatever had arrived, the 64-bit batch-norm tree
        dict(name="mobilenet_b37_bn64", op="net", batch=37, bits=64, host=False),
        # the throughput configuration: MobileNetV1 over 1024 images that lie in HBM
        dict(name="mobilenet_b1024", op="net", batch=1024, bits=32, host=False),
        # images and logits in pinned host memory, one blocking call per batch
        dict(name="mobilenet_host_b64", op="net", batch=64, bits=32, host=True),
        # the single convolution layer of the first configuration, one image
        dict(name="conv_32x32x32_b1", op="conv", batch=1, H=32, W=32, cin=32, cout=64, k=3, s=1,
             bits=32, mode="bn", bias=False),
        # a convolution over channel counts that are no multiple of a vector, with bias, no batch norm
        dict(name="conv_48x48x20_b32", op="conv", batch=32, H=48, W=48, cin=20, cout=40, k=3, s=1,
             bits=32, mode="mult", bias=True),
        # a residual block: two 3x3 convolutions and the add of the shortcut
        dict(name="residual_28x28x128_b32", op="block", batch=32, H=28, W=28, c=128, bits=32),
        # the pointwise configuration
        dict(name="pointwise_56x56x128_b64", op="pointwise", batch=64, H=56, W=56, cin=128, cout=256,
             bits=32, mode="bn", bias=False),
        # the depthwise configuration: the reference's CHW input, stride 2, 64-bit batch norm
        dict(name="depthwise_chw_112x112x64_b64", op="depthwise", batch=64, H=112, W=112, c=64, k=3,
             s=2, hwc=False, bits=64, mode="bn", bias=False),
        # a 5x5 depthwise layer on HWC input, as mobile networks with wider kernels have it
        dict(name="depthwise_hwc_28x28x120_5x5_b32", op="depthwise", batch=32, H=28, W=28, c=120, k=5,
             s=1, hwc=True, bits=32, mode="bn", bias=True),
        # the fully connected configuration
        dict(name="linear_4096_b256", op="linear", batch=256, K=4096, N=4096, raw=False, bits=32,
             mode="mult", bias=True),
        # the overlapping max pooling that follows a first layer
        dict(name="maxpool_112x112x64_b32", op="pool", batch=32, H=112, W=112, c=64, k=3, s=2, pad=1,
             avg=False, bits=32),
    ]


MOST_MACS = 4e9          # of a drawn layer: small beside the largest listed case
MOST_BYTES = 4e8


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.499)))))))


def _channels(rng, lo, hi):
    """Half of them whole vectors, the rest as they come."""
    c = _log(rng, lo, hi)
    return max(16, (c + 8) // 16 * 16) if rng.random() < 0.5 else c


def draw(rng):
    op = rng.choice(["net", "net", "conv", "conv", "pointwise", "pointwise", "depthwise", "depthwise",
                     "linear", "pool", "block"])
    bits = rng.choice([32, 64])
    mode = rng.choice(["bn", "bn", "mult", "none"])
    bias = rng.random() < 0.5
    if op == "net":
        host = rng.random() < 0.25
        return dict(op=op, batch=_log(rng, 1, 256 if host else 1024), bits=bits, host=host)
    if op == "linear":
        return dict(op=op, batch=_log(rng, 1, 512), K=_channels(rng, 64, 4096), N=_channels(rng, 10, 4096),
                    raw=rng.random() < 0.5, bits=bits, mode=mode, bias=bias)
    batch = _log(rng, 1, 64)
    H = _log(rng, 7, 112)
    W = H if rng.random() < 0.7 else _log(rng, 7, 112)
    if op == "conv":
        c = dict(op=op, batch=batch, H=H, W=W, cin=_channels(rng, 3, 256), cout=_channels(rng, 8, 256),
                 k=rng.choice([3, 3, 5]), s=rng.choice([1, 1, 2]), bits=bits, mode=mode, bias=bias)
    elif op == "pointwise":
        c = dict(op=op, batch=batch, H=H, W=W, cin=_channels(rng, 16, 1024), cout=_channels(rng, 16, 1024),
                 bits=bits, mode=mode, bias=bias)
    elif op == "depthwise":
        c = dict(op=op, batch=batch, H=H, W=W, c=_channels(rng, 16, 512), k=rng.choice([3, 3, 5]),
                 s=rng.choice([1, 2]), hwc=rng.random() < 0.6, bits=bits, mode=mode, bias=bias)
    elif op == "pool":
        k, s, pad = rng.choice([(3, 2, 1), (2, 2, 0), (3, 2, 0), (7, 7, 0)])
        c = dict(op=op, batch=batch, H=H, W=W, c=_channels(rng, 16, 512), k=k, s=s, pad=pad,
                 avg=pad == 0 and rng.random() < 0.5, bits=bits)
    else:
        c = dict(op=op, batch=batch, H=H, W=W, c=_channels(rng, 16, 256), bits=bits)
    while c["batch"] > 1 and (work(c)["flops"] > 2 * MOST_MACS or work(c)["bytes"] > MOST_BYTES):
        c["batch"] = max(1, c["batch"] // 2)
    return c


# ---- inputs ---------------------------------------------------------------------------------------

def _out(n, k, s, pad):
    return (n + 2 * pad - k) // s + 1


class _Maker:
    """Tensors on the GPU, made from the seed alone."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed) * 7919 + 17)

    def ints(self, lo, hi, shape, dtype):
        return torch.randint(lo, hi + 1, tuple(shape), generator=self.g, device=DEV, dtype=dtype)

    def x(self, *shape):
        return self.ints(0, 255, shape, torch.uint8)

    def w(self, *shape):
        return self.ints(-16, 16, shape, torch.int8)

    def requant(self, n, terms, bits, mode, bias):
        """Batch-norm parameters, bias and a shift that spreads the results over 0..255."""
        dt = torch.int32 if bits == 32 else torch.int64
        half = math.ceil(math.log2(terms) / 2)
        return dict(
            k=self.ints(1, 64, (n,), dt) if mode == "bn" else None,
            lam=self.ints(-32768, 32767, (n,), dt) if mode == "bn" else None,
            bias=self.ints(-128, 127, (n,), torch.int8) if bias else None,
            mult=3 if mode == "mult" else 1,
            shift=half + dict(bn=8, mult=5, none=3)[mode],
            relu=0 if mode == "none" else 1, bn=1 if mode == "bn" else 0, mode=mode)


# (output channels of the pointwise layer, stride of the depthwise layer) of the 13 pairs
PAIRS = ((64, 1), (128, 2), (128, 1), (256, 2), (256, 1), (512, 2), (512, 1), (512, 1), (512, 1), (512, 1),
         (512, 1), (1024, 2), (1024, 1))


def _mobilenet(seed, bits):
    """MobileNetV1-1.0 at 224x224x3: the layers with random weights, as plain dicts of arrays."""
    rng = np.random.default_rng(int(seed) + 4)
    dt = np.int32 if bits == 32 else np.int64
    layers = []

    def add(op, H, cin, cout, stride, terms, wshape, bn=True):
        Ho = 1 if op == "avgpool" else (H - 1) // stride + 1
        p = dict(op=op, H=H, W=H, Cin=cin, Cout=cout, stride=stride, Ho=Ho, Wo=Ho)
        if wshape:
            p["w"] = rng.integers(-16, 16, size=wshape).astype(np.int8)
        if bn:
            p["k"] = rng.integers(1, 65, size=cout).astype(dt)
            p["lam"] = rng.integers(-32768, 32768, size=cout).astype(dt)
            p["out_shift"] = math.ceil(math.log2(terms)) + 1
        layers.append(p)
        return Ho

    H, c = add("conv", 224, 3, 32, 2, 27, (32, 3, 3, 3)), 32
    for cout, s in PAIRS:
        H = add("depthwise", H, c, c, s, 9, (c, 3, 3))
        add("pointwise", H, c, cout, 1, c, (cout, c))
        c = cout
    add("avgpool", H, c, c, H, 0, None, bn=False)
    add("linear32", 1, c, 1000, 1, c, (1000, c), bn=False)
    return layers


def _inputs(case, seed):
    m = _Maker(seed)
    op, B = case["op"], case["batch"]
    if op == "net":
        return dict(params=_mobilenet(seed, case["bits"]), x=m.x(B, 224, 224, 3))
    if op == "linear":
        i = dict(x=m.x(B, case["K"]), w=m.w(case["N"], case["K"]))
        i.update(m.requant(case["N"], case["K"], case["bits"], case["mode"], case["bias"]))
        i["bias32"] = m.ints(-2 ** 20, 2 ** 20, (case["N"],), torch.int32) if case["bias"] else None
        return i
    H, W = case["H"], case["W"]
    if op == "conv":
        k = case["k"]
        i = dict(x=m.x(B, H, W, case["cin"]), w=m.w(case["cout"], k, k, case["cin"]))
        i.update(m.requant(case["cout"], k * k * case["cin"], case["bits"], case["mode"], case["bias"]))
        return i
    if op == "pointwise":
        i = dict(x=m.x(B, H, W, case["cin"]), w=m.w(case["cout"], case["cin"]))
        i.update(m.requant(case["cout"], case["cin"], case["bits"], case["mode"], case["bias"]))
        return i
    if op == "depthwise":
        c, k = case["c"], case["k"]
        i = dict(x=m.x(B, H, W, c) if case["hwc"] else m.x(B, c, H, W), w=m.w(c, k, k))
        i.update(m.requant(c, k * k, case["bits"], case["mode"], case["bias"]))
        return i
    if op == "pool":
        return dict(x=m.x(B, H, W, case["c"]))
    c = case["c"]
    layers = []
    for _ in range(2):
        layer = dict(w=m.w(c, 3, 3, c))
        layer.update(m.requant(c, 9 * c, case["bits"], "bn", False))
        layers.append(layer)
    return dict(x=m.x(B, H, W, c), layers=layers, m1=37, m2=91, shift=7)


def prepare(case, seed):
    torch.cuda.set_device(0)
    api.set_device(0)
    s = dict(case=case)
    s.update(_inputs(case, seed))
    op, B = case["op"], case["batch"]

    def buffer(*shape, dtype=torch.uint8):
        return torch.empty(shape, dtype=dtype, device=DEV)

    if op == "net":
        s["net"] = api.build_mobilenet_v1(s.pop("params"), bits=case["bits"], max_batch=B)
        s["out"] = buffer(B, 1000, dtype=torch.int32)
        if case["host"]:
            s["x"] = s["x"].cpu().pin_memory()
            s["out"] = torch.empty((B, 1000), dtype=torch.int32, pin_memory=True)
    elif op == "linear":
        s["out"] = buffer(B, case["N"], dtype=torch.int32 if case["raw"] else torch.uint8)
    elif op == "block":
        shape = s["x"].shape
        s["mid"], s["conv"], s["out"] = buffer(*shape), buffer(*shape), buffer(*shape)
    else:
        s["out"] = buffer(*_out_shape(case))
    return s


def _out_shape(case):
    B, H, W, op = case["batch"], case["H"], case["W"], case["op"]
    if op == "pointwise":
        return (B, H, W, case["cout"])
    k, st = case["k"], case["s"]
    pad = case["pad"] if op == "pool" else k // 2
    return (B, _out(H, k, st, pad), _out(W, k, st, pad), case["cout"] if op == "conv" else case["c"])


# ---- one pass -------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    op, B, bits = case["op"], case["batch"], case["bits"]
    if op == "net":
        s["net"].run(s["x"], s["out"], B)
        return s["out"]
    api.set_batch(B)
    if op == "linear":
        K, N = case["K"], case["N"]
        if case["raw"]:
            api.pulp_nn_linear_out_32(bits, s["x"], s["bias32"], s["out"], s["w"], K, N)
        else:
            api.pulp_nn_linear(bits, s["x"], s["bias"], s["out"], s["w"], s["k"], s["lam"], s["mult"], s["shift"],
                               K, N, s["relu"], s["bn"])
        return s["out"]
    H, W = case["H"], case["W"]
    if op == "block":
        c, x = case["c"], s["x"]
        for layer, src, dst in zip(s["layers"], (x, s["mid"]), (s["mid"], s["conv"])):
            api.pulp_nn_conv_Ho_parallel(bits, src, None, None, dst, layer["w"], layer["k"], layer["lam"],
                                         layer["mult"], layer["shift"], W, H, c, W, H, c, 3, 3, 1, 1, 1, 1, 1, 1,
                                         layer["relu"], layer["bn"])
        api.pulp_nn_add(bits, x, s["conv"], s["out"], s["m1"], s["m2"], s["shift"], H, W, c)
        return {"mid": s["mid"], "conv": s["conv"], "out": s["out"]}
    out = s["out"]
    Ho, Wo = out.shape[1], out.shape[2]
    if op == "pool":
        k, st, p = case["k"], case["s"], case["pad"]
        if case["avg"]:
            api.pulp_nn_avgpool(bits, s["x"], out, 0, 0, 0, W, H, case["c"], Wo, Ho, k, k, p, p, p, p, st, st, 0)
        else:
            api.pulp_nn_maxpool(bits, s["x"], out, W, H, case["c"], Wo, Ho, k, k, p, p, p, p, st, st)
    elif op == "conv":
        k, st, p = case["k"], case["s"], case["k"] // 2
        api.pulp_nn_conv_Ho_parallel(bits, s["x"], None, s["bias"], out, s["w"], s["k"], s["lam"], s["mult"],
                                     s["shift"], W, H, case["cin"], Wo, Ho, case["cout"], k, k, p, p, p, p, st, st,
                                     s["relu"], s["bn"])
    elif op == "pointwise":
        api.pulp_nn_pointwise_HoWo_parallel(bits, s["x"], None, s["bias"], out, s["w"], s["k"], s["lam"], s["mult"],
                                            s["shift"], W, H, case["cin"], W, H, case["cout"], 1, 1, 0, 0, 0, 0, 1, 1,
                                            s["relu"], s["bn"])
    else:
        k, st, p, c = case["k"], case["s"], case["k"] // 2, case["c"]
        fn = api.pulpnn_depthwise_hwc if case["hwc"] else api.pulp_nn_depthwise_generic
        fn(bits, s["x"], None, s["bias"], out, s["w"], None, s["k"], s["lam"], s["mult"], s["shift"], W, H, c, Wo, Ho,
           c, k, k, p, p, p, p, st, st, s["relu"], s["bn"])
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------

def work(case):
    op, B = case["op"], case["batch"]
    if op == "net":
        # images in, logits out, the weights once; no activation has to leave the chip
        bn, H, c = case["bits"] // 8, 112, 32
        macs, params = H * H * 32 * 27, 32 * 27 + 2 * 32 * bn
        for cout, st in PAIRS:
            H //= st
            macs += H * H * c * (9 + cout)
            params += 9 * c + c * cout + 2 * (c + cout) * bn
            c = cout
        macs += c * 1000
        params += c * 1000
        return {"bytes": B * (224 * 224 * 3 + 4000) + params, "flops": 2 * B * macs}
    bn = 2 * case["bits"] // 8 if case.get("mode", "bn") == "bn" else 0
    if op == "linear":
        K, N = case["K"], case["N"]
        return {"bytes": B * K + N * K + B * N * (4 if case["raw"] else 1) + (0 if case["raw"] else bn * N),
                "flops": 2 * B * K * N}
    H, W = case["H"], case["W"]
    if op == "block":
        c, a = case["c"], B * H * W * case["c"]
        return {"bytes": 4 * a + 2 * (9 * c * c + bn * c), "flops": 2 * 2 * a * 9 * c + 4 * a}
    out = math.prod(_out_shape(case))
    if op == "conv":
        K = case["k"] ** 2 * case["cin"]
        return {"bytes": B * H * W * case["cin"] + out + case["cout"] * (K + bn), "flops": 2 * out * K}
    if op == "pointwise":
        K = case["cin"]
        return {"bytes": B * H * W * K + out + case["cout"] * (K + bn), "flops": 2 * out * K}
    c, taps = case["c"], case["k"] ** 2
    if op == "pool":
        return {"bytes": B * H * W * c + out, "flops": out * taps}
    return {"bytes": B * H * W * c + out + c * (taps + bn), "flops": 2 * out * taps}


def tolerance(case):
    return "exact"


# ---- the same in plain torch, 64 bits ----------------------------------------------------------------

def _finish(acc, q):
    """Sums in int64 (channel last) to bytes, by the requantisation rules of the reference."""
    if q.get("bias") is not None:
        acc = acc + q["bias"].long()
    if q["mode"] == "bn":
        t = (acc * q["k"].long() + q["lam"].long()) >> q["shift"]
    elif q["mode"] == "mult":
        t = (acc * q["mult"]) >> q["shift"]
        t = ((t + 32768) & 65535) - 32768
    else:
        t = acc >> q["shift"]
    return t.clamp(0, 255).to(torch.uint8)


def _conv64(x, w, q, st, pad):
    """x [B,H,W,C] bytes, w [N,ky,kx,C]: one matrix product in float64 (exact here) per tap."""
    B, H, W, C = x.shape
    N, ky, kx, _ = w.shape
    Ho, Wo = (H + 2 * pad - ky) // st + 1, (W + 2 * pad - kx) // st + 1
    outs = []
    step = max(1, int(3e7 // (H * W * C + Ho * Wo * max(N, C))))
    for b in range(0, B, step):
        xp = torch.nn.functional.pad(x[b:b + step].double(), (0, 0, pad, pad, pad, pad))
        acc = 0
        for fy in range(ky):
            for fx in range(kx):
                v = xp[:, fy:fy + (Ho - 1) * st + 1:st, fx:fx + (Wo - 1) * st + 1:st, :]
                acc = acc + v @ w[:, fy, fx, :].double().t()
        outs.append(_finish(acc.long(), q))
    return torch.cat(outs)


def _depthwise64(x, w, q, st, pad):
    """x [B,H,W,C], w [C,ky,kx]."""
    B, H, W, C = x.shape
    _, ky, kx = w.shape
    Ho, Wo = (H + 2 * pad - ky) // st + 1, (W + 2 * pad - kx) // st + 1
    outs = []
    step = max(1, int(3e7 // (H * W * C)))
    for b in range(0, B, step):
        xp = torch.nn.functional.pad(x[b:b + step].long(), (0, 0, pad, pad, pad, pad))
        acc = 0
        for fy in range(ky):
            for fx in range(kx):
                acc = acc + xp[:, fy:fy + (Ho - 1) * st + 1:st, fx:fx + (Wo - 1) * st + 1:st, :] * w[:, fy, fx].long()
        outs.append(_finish(acc, q))
    return torch.cat(outs)


def exact(case, seed):
    i = _inputs(case, seed)
    op = case["op"]
    if op == "net":
        logits = []
        put = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
        for b in range(0, case["batch"], 64):
            x = i["x"][b:b + 64]
            for p in i["params"]:
                q = dict(mode="bn", shift=p.get("out_shift"), k=put(p["k"]), lam=put(p["lam"])) if "k" in p else None
                if p["op"] == "conv":
                    x = _conv64(x, put(p["w"]), q, 2, 1)
                elif p["op"] == "depthwise":
                    x = _depthwise64(x, put(p["w"]), q, p["stride"], 1)
                elif p["op"] == "pointwise":
                    x = _conv64(x, put(p["w"])[:, None, None, :], q, 1, 0)
                elif p["op"] == "avgpool":
                    x = x.long().sum((1, 2)) // (p["H"] * p["W"])
                else:
                    logits.append((x.double() @ put(p["w"]).double().t()).long())
        out = torch.cat(logits)
        return out.cpu() if case["host"] else out
    if op == "linear":
        acc = (i["x"].double() @ i["w"].double().t()).long()
        if case["raw"]:
            return acc + i["bias32"].long() if case["bias"] else acc
        return _finish(acc, i)
    if op == "block":
        mid = _conv64(i["x"], i["layers"][0]["w"], i["layers"][0], 1, 1)
        conv = _conv64(mid, i["layers"][1]["w"], i["layers"][1], 1, 1)
        t = (i["x"].long() * i["m1"] + conv.long() * i["m2"]) >> i["shift"]
        return {"mid": mid, "conv": conv, "out": t.clamp(0, 255).to(torch.uint8)}
    if op == "conv":
        return _conv64(i["x"], i["w"], i, case["s"], case["k"] // 2)
    if op == "pointwise":
        return _conv64(i["x"], i["w"][:, None, None, :], i, 1, 0)
    if op == "depthwise":
        x = i["x"] if case["hwc"] else i["x"].permute(0, 2, 3, 1)
        return _depthwise64(x, i["w"], i, case["s"], case["k"] // 2)
    k, st, p = case["k"], case["s"], case["pad"]
    _, Ho, Wo, _ = _out_shape(case)
    xp = torch.nn.functional.pad(i["x"].long(), (0, 0, p, p, p, p))
    acc = None
    for fy in range(k):
        for fx in range(k):
            v = xp[:, fy:fy + (Ho - 1) * st + 1:st, fx:fx + (Wo - 1) * st + 1:st, :]
            acc = v if acc is None else acc + v if case["avg"] else torch.maximum(acc, v)
    return acc // (k * k) if case["avg"] else acc
