"""Workloads that a user of this framework runs, for timing and for comparing results.

Every case goes through the public entry points (Context's operators, graph.DeviceRunner) with the operands resident on
the device, as a host that evaluates TOSA graphs keeps them.  The listed cases are the benchmark configurations (one
small int8 convolution, the batched MATMULs, a ResNet-50 layer, the inverted-residual block, the ResNet-50-shaped graph
at three batch sizes) and four that stand for what those leave out: channel counts that are not whole 32-byte runs, fp32
convolution, fp16 MATMUL of odd sizes, int8 depthwise convolution.  draw() spreads over the ranges around them.
"""
import math

import numpy as np
import torch

import reference_model_b200 as tb
from reference_model_b200 import graph as G


def listed():
    return [
        # the smallest call: one 1x1 convolution + RESCALE on a 32x32 map, where launch and host time are everything
        dict(name="conv_i8_small", kind="conv_i8", n=1, h=32, w=32, ic=8, oc=16, k=1, stride=1),
        # the 3x3 layer of a ResNet's first stage at batch 32, with RESCALE and CLAMP
        dict(name="conv_i8_3x3", kind="conv_i8", n=32, h=56, w=56, ic=64, oc=64, k=3, stride=1),
        # channel counts of small mobile networks (24, 40, ...: no whole 32-byte runs) on an odd map
        dict(name="conv_i8_ragged", kind="conv_i8", n=16, h=57, w=57, ic=24, oc=40, k=3, stride=1),
        # fp32 graphs: the 3x3 layer in full precision (no TF32)
        dict(name="conv_f32_3x3", kind="conv_f32", n=8, h=56, w=56, ic=64, oc=64, k=3, stride=1),
        # int8 depthwise layer of a mobile network + RESCALE and CLAMP
        dict(name="depthwise_i8", kind="depthwise_i8", n=32, h=56, w=56, c=144, k=3, stride=1),
        # the batched int8 MATMUL of the benchmark, both zero points set
        dict(name="matmul_i8", kind="matmul_i8", n=64, h=1024, c=4096, w=1024),
        # the same product in fp32
        dict(name="matmul_f32", kind="matmul_f32", n=64, h=1024, c=4096, w=1024),
        # attention-shaped fp16 product: many small batches, odd width
        dict(name="matmul_f16_odd", kind="matmul_f16", n=96, h=197, c=64, w=197, dtype="fp16", out="fp16"),
        # fp16 inverted-residual block: 1x1 expand, 3x3 depthwise stride 2, 1x1 project
        dict(name="block_f16", kind="block", n=64, hw=112, ic=32, mid=192, oc=64, stride=2, dtype="fp16"),
        # the ResNet-50-shaped int8 graph: one image (latency), a server's batch, a throughput batch
        dict(name="resnet_b1", kind="resnet", batch=1, image=224),
        dict(name="resnet_b32", kind="resnet", batch=32, image=224),
        dict(name="resnet_b256", kind="resnet", batch=256, image=224),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _channels(rng, lo, hi):
    """Mostly multiples of eight, sometimes any count."""
    c = _log(rng, lo, hi)
    return c if rng.random() < 0.25 else max(8, (c + 4) // 8 * 8)


def _conv_size(rng, hi, k, stride):
    h = _log(rng, 7, hi)
    return h + 1 if stride == 2 and k == 1 and h % 2 == 0 else h


def draw(rng):
    while True:
        kind = rng.choice(["conv_i8", "conv_i8", "conv_f32", "depthwise_i8", "matmul_i8", "matmul_f32", "matmul_f16", "block",
                           "resnet", "resnet"])
        if kind in ("conv_i8", "conv_f32"):
            k, stride = rng.choice([1, 1, 3, 3, 3, 5]), rng.choice([1, 1, 1, 2])
            c = dict(kind=kind, n=_log(rng, 1, 32), h=_conv_size(rng, 112, k, stride), w=_conv_size(rng, 112, k, stride),
                     ic=_channels(rng, 8, 512), oc=_channels(rng, 8, 512), k=k, stride=stride)
            if work(c)["flops"] > (20e9 if kind == "conv_i8" else 10e9):
                continue
        elif kind == "depthwise_i8":
            stride = rng.choice([1, 1, 2])
            c = dict(kind=kind, n=_log(rng, 1, 64), h=_conv_size(rng, 112, 3, stride), w=_conv_size(rng, 112, 3, stride),
                     c=_channels(rng, 16, 960), k=rng.choice([3, 3, 5]), stride=stride)
            if work(c)["bytes"] > 2e8:
                continue
        elif kind in ("matmul_i8", "matmul_f32", "matmul_f16"):
            c = dict(kind=kind, n=_log(rng, 1, 96), h=_log(rng, 1, 1024), c=_log(rng, 16, 4096), w=_log(rng, 16, 1024))
            if kind == "matmul_f16":
                c.update(dtype=rng.choice(["fp16", "bf16"]))
                c.update(out=rng.choice([c["dtype"], "fp32"]))
            if work(c)["flops"] > 4e10:
                continue
        elif kind == "block":
            # (input channels, output channels, stride, largest map) of the block's places in a network
            ic, oc, stride, hi = rng.choice([(16, 24, 2, 112), (24, 32, 2, 56), (32, 64, 2, 112), (32, 32, 1, 28), (64, 96, 1, 28)])
            hw = _log(rng, 7, hi)
            c = dict(kind=kind, n=_log(rng, 1, 64), hw=hw + hw % 2, ic=ic, mid=6 * ic, oc=oc, stride=stride,
                     dtype=rng.choice(["fp16", "bf16"]))
        else:
            c = dict(kind=kind, batch=_log(rng, 1, 256), image=32 * rng.randint(3, 8))
            if c["batch"] * c["image"] ** 2 > 256 * 224 ** 2 or c["image"] == 224 and c["batch"] in (1, 32, 256):
                continue
        return c


# ------------------------------------------------------------------------------------------------ shapes and work
def _pads(size, k, stride):
    """Padding that keeps the map's size (halves it at stride 2) and meets the exact-division rule."""
    lo = k // 2
    hi = lo if stride == 1 or (size - 1 + 2 * lo - (k - 1)) % stride == 0 else lo - 1
    return lo, hi, (size - 1 + lo + hi - (k - 1)) // stride + 1


def _resnet_convs(image):
    """(input size, input channels, output channels, kernel, output size) of the graph's convolutions."""
    s = image // 2
    yield image, 3, 64, 7, s
    s, c = s // 2, 64
    for stage, (mid, blocks) in enumerate(((64, 3), (128, 4), (256, 6), (512, 3))):
        for blk in range(blocks):
            o = s // 2 if stage > 0 and blk == 0 else s
            yield s, c, mid, 1, s
            yield s, mid, mid, 3, o
            yield o, mid, 4 * mid, 1, o
            if blk == 0:
                yield s, c, 4 * mid, 1, o
            s, c = o, 4 * mid


_SIZE = {"fp16": 2, "bf16": 2, "fp32": 4}


def work(case):
    """Inputs read once, outputs written once; two operations per multiply-add."""
    k = case["kind"]
    if k in ("conv_i8", "conv_f32"):
        n, h, w, ic, oc, ks = (case[x] for x in ("n", "h", "w", "ic", "oc", "k"))
        oh, ow = _pads(h, ks, case["stride"])[2], _pads(w, ks, case["stride"])[2]
        e = 1 if k == "conv_i8" else 4
        extra = oc * (4 + 4 + 1) if k == "conv_i8" else oc * 4
        return {"bytes": e * (n * h * w * ic + oc * ks * ks * ic + n * oh * ow * oc) + extra,
                "flops": 2.0 * n * oh * ow * oc * ks * ks * ic}
    if k == "depthwise_i8":
        n, h, w, c, ks = (case[x] for x in ("n", "h", "w", "c", "k"))
        oh, ow = _pads(h, ks, case["stride"])[2], _pads(w, ks, case["stride"])[2]
        return {"bytes": n * h * w * c + ks * ks * c + n * oh * ow * c + 9 * c, "flops": 2.0 * n * oh * ow * c * ks * ks}
    if k.startswith("matmul"):
        n, h, c, w = (case[x] for x in ("n", "h", "c", "w"))
        ei, eo = {"matmul_i8": (1, 4), "matmul_f32": (4, 4)}.get(k) or (2, _SIZE[case["out"]])
        return {"bytes": ei * n * (h * c + c * w) + eo * n * h * w, "flops": 2.0 * n * h * c * w}
    if k == "block":
        n, hw, ic, mid, oc = (case[x] for x in ("n", "hw", "ic", "mid", "oc"))
        oh = _pads(hw, 3, case["stride"])[2]
        return {"bytes": 2 * (n * hw * hw * ic + n * oh * oh * oc + mid * ic + 9 * mid + oc * mid + 2 * mid + oc),
                "flops": 2.0 * n * (hw * hw * ic * mid + oh * oh * mid * (9 + oc))}
    b, image = case["batch"], case["image"]
    macs = sum(oc * ks * ks * ic * o * o for _, ic, oc, ks, o in _resnet_convs(image)) + 2048 * 1000
    params = sum(oc * (ks * ks * ic + 9) for _, ic, oc, ks, _ in _resnet_convs(image)) + 2048 * 1000
    return {"bytes": b * image * image * 3 + params + b * 4000, "flops": 2.0 * b * macs}


def tolerance(case):
    """Integers are exact.  fp32 sums in another order; fp16 / bf16 results rounded once (fp32 accumulation), the block's
    three times, where a difference in the last bit of an intermediate is carried on."""
    k = case["kind"]
    if k in ("conv_f32", "matmul_f32"):
        return {"rel": 1e-5}
    if k == "matmul_f16":
        return {"rel": {"fp16": 1e-3, "bf16": 8e-3, "fp32": 1e-5}[case["out"]]}
    if k == "block":
        return {"rel": 2e-3 if case["dtype"] == "fp16" else 1e-2}
    return "exact"


# ------------------------------------------------------------------------------------------------ preparing and running
_CONTEXT = []


def _context():
    """One context per process and device, as a host keeps it."""
    if not _CONTEXT:
        _CONTEXT.append(tb.Context(0))
    return _CONTEXT[0]


_DTYPES = {torch.int8: tb.DType.INT8, torch.int32: tb.DType.INT32, torch.float32: tb.DType.FP32,
           torch.float16: tb.DType.FP16, torch.bfloat16: tb.DType.BF16}
_TORCH = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


class _State:
    """Operands over torch memory (or a graph runner), and one call that evaluates them."""

    def __init__(self):
        self.ctx, self.handles, self.runner = _context(), [], None

    def wrap(self, t):
        h = self.ctx.wrap(_DTYPES[t.dtype], tuple(t.shape), t.data_ptr(), t)
        self.handles.append(h)
        return h

    def __del__(self):
        try:
            if self.runner is not None:
                if self.runner.captured is not None:
                    self.ctx.graph_destroy(self.runner.captured)
                views = [t for t in self.runner.t.values() if t._keepalive is not None]
                for t in views + [t for t in self.runner.t.values() if t._keepalive is None]:
                    t.free()
            for h in self.handles:
                h.free()
        except Exception:    # the interpreter is going down
            pass


def _rescale(s, gen, channels):
    """Per-channel RESCALE int32 -> int8 with multipliers in [2^30, 2^31) and shifts in [30, 40]."""
    mult = torch.randint(1 << 30, (1 << 31) - 1, (channels,), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    shift = torch.randint(30, 41, (channels,), generator=gen, device="cuda", dtype=torch.int64).to(torch.int8)
    return tb.RescaleAttr(s.wrap(mult), s.wrap(shift), 0, -128, True, "DOUBLE_ROUND", per_channel=True)


def _int8(gen, lo, *shape):
    return torch.randint(lo, 128, shape, generator=gen, device="cuda", dtype=torch.int8)


def _bias32(gen, n):
    return torch.randint(-65536, 65537, (n,), generator=gen, device="cuda", dtype=torch.int32)


def _randn(gen, dtype, scale, *shape):
    return (torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * scale).to(dtype)


def prepare(case, seed):
    s = _State()
    ctx, kind = s.ctx, case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("conv_i8", "conv_f32", "depthwise_i8"):
        n, h, w, k, st = (case[x] for x in ("n", "h", "w", "k", "stride"))
        pt, pb, oh = _pads(h, k, st)
        pl, pr, ow = _pads(w, k, st)
        pad, stride, one = [pt, pb, pl, pr], [st, st], [1, 1]
        if kind == "conv_f32":
            ic, oc = case["ic"], case["oc"]
            x, b = s.wrap(_randn(gen, torch.float32, 1.0, n, h, w, ic)), s.wrap(_randn(gen, torch.float32, 0.1, oc))
            wt = s.wrap(_randn(gen, torch.float32, 1.0 / math.sqrt(k * k * ic), oc, k, k, ic))
            out = torch.empty((n, oh, ow, oc), dtype=torch.float32, device="cuda")
            to, relu = s.wrap(out), tb.Epilogue(None, (0.0, 6.0))
            s.call = lambda: (ctx.conv2d(x, wt, b, to, pad, stride, one, 0, 0, relu), out)[1]
        elif kind == "conv_i8":
            ic, oc = case["ic"], case["oc"]
            x, wt, b = s.wrap(_int8(gen, -128, n, h, w, ic)), s.wrap(_int8(gen, -127, oc, k, k, ic)), s.wrap(_bias32(gen, oc))
            out = torch.empty((n, oh, ow, oc), dtype=torch.int8, device="cuda")
            to, epi = s.wrap(out), tb.Epilogue(_rescale(s, gen, oc), (-128, 127))
            s.call = lambda: (ctx.conv2d(x, wt, b, to, pad, stride, one, -128, 0, epi), out)[1]
        else:
            c = case["c"]
            x, wt, b = s.wrap(_int8(gen, -128, n, h, w, c)), s.wrap(_int8(gen, -127, k, k, c, 1)), s.wrap(_bias32(gen, c))
            out = torch.empty((n, oh, ow, c), dtype=torch.int8, device="cuda")
            to, epi = s.wrap(out), tb.Epilogue(_rescale(s, gen, c), (-128, 127))
            s.call = lambda: (ctx.depthwise_conv2d(x, wt, b, to, pad, stride, one, -128, 0, epi), out)[1]
    elif kind.startswith("matmul"):
        n, h, c, w = (case[x] for x in ("n", "h", "c", "w"))
        a_zp, b_zp = 0, 0
        if kind == "matmul_i8":
            a, b, odt, a_zp, b_zp = _int8(gen, -128, n, h, c), _int8(gen, -128, n, c, w), torch.int32, 3, -2
        else:
            dt = torch.float32 if kind == "matmul_f32" else _TORCH[case["dtype"]]
            a, b, odt = _randn(gen, dt, 1.0, n, h, c), _randn(gen, dt, 1.0, n, c, w), _TORCH[case.get("out", "fp32")]
        out = torch.empty((n, h, w), dtype=odt, device="cuda")
        ta, tbm, to = s.wrap(a), s.wrap(b), s.wrap(out)
        s.call = lambda: (ctx.matmul(ta, tbm, to, a_zp, b_zp), out)[1]
    elif kind == "block":
        n, hw, ic, mid, oc, st = (case[x] for x in ("n", "hw", "ic", "mid", "oc", "stride"))
        dt = _TORCH[case["dtype"]]
        p0, p1, oh = _pads(hw, 3, st)
        pad, stride = [p0, p1, p0, p1], [st, st]
        x = s.wrap(_randn(gen, dt, 1.0, n, hw, hw, ic))
        w1, b1 = s.wrap(_randn(gen, dt, ic ** -0.5, mid, 1, 1, ic)), s.wrap(_randn(gen, dt, 0.1, mid))
        wd, bd = s.wrap(_randn(gen, dt, 1.0 / 3, 3, 3, mid, 1)), s.wrap(_randn(gen, dt, 0.1, mid))
        w2, b2 = s.wrap(_randn(gen, dt, mid ** -0.5, oc, 1, 1, mid)), s.wrap(_randn(gen, dt, 0.1, oc))
        # the tensor between the first two operators, for shapes that do not run as one kernel
        expanded = s.wrap(torch.empty((n, hw, hw, mid), dtype=dt, device="cuda"))
        t2 = s.wrap(torch.empty((n, oh, oh, mid), dtype=dt, device="cuda"))
        out = torch.empty((n, oh, oh, oc), dtype=dt, device="cuda")
        to, relu6 = s.wrap(out), tb.Epilogue(None, (0.0, 6.0))

        def call():
            ctx.conv2d_depthwise(x, w1, b1, wd, bd, t2, pad, stride, relu6, relu6, expanded)
            ctx.conv2d(t2, w2, b2, to, [0, 0, 0, 0], [1, 1], [1, 1])
            return out

        s.call = call
    else:
        g = G.resnet50_int8(case["batch"], seed=seed, image=case["image"])
        logits = torch.empty((1, case["batch"], 1000), dtype=torch.int32, device="cuda")
        s.runner = G.DeviceRunner(ctx, g, external={g.outputs[0]: s.wrap(logits)})
        s.runner.set_input(G.synthetic_images(case["batch"], seed, case["image"]))
        s.runner.capture()
        s.call = lambda: (s.runner.run(), logits)[1]
    torch.cuda.synchronize()
    return s


def run(state):
    return state.call()
