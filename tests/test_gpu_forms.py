"""Which form of the int8 CONV2D + RESCALE kernels a shape takes (tb200_last_form), each bit for bit against the oracle, with and
without a residual join behind it; and that every kernel gives up its waits and recovers."""
import numpy as np
import pytest

import reference_model_b200 as tb
from oracle import oracle as orc
from tests import util
from tests.test_gpu_conv_chan import LINEAR, _conv, _join, _operands

pytestmark = pytest.mark.gpu

I8 = tb.DType.INT8
OUT = (1700000001, 41, -128)


@pytest.fixture(scope="module")
def ctx():
    c = tb.Context(0)
    yield c
    c.close()


class _Layer:
    def __init__(self, ctx, n, h, w, ic, oc, k, stride=1, pad=None, zp=-128, join=False):
        kh, kw = k if isinstance(k, tuple) else (k, k)
        pad = pad or [kh // 2] * 2 + [kw // 2] * 2
        r, x, wt, b, mult, shift = _operands(n * h + oc, n, h, w, ic, oc, kh, kw)
        q = _conv(x, wt, b, mult, shift, pad, [stride] * 2, [1, 1], zp, "DOUBLE_ROUND", -128, 127)
        ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift)]
        to = ctx.empty(I8, q.shape)
        epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
        if join:
            other = r.integers(-128, 128, size=q.shape).astype(np.int8)
            st, q = _join(q.astype(np.int8), other, LINEAR, OUT, "DOUBLE_ROUND", -128, 127)
            assert st == tb.Status.OK
            cs = [ctx.from_numpy(other)]
            cs += [ctx.from_numpy(np.array([v], dt)) for m, s, _ in LINEAR + (OUT,) for v, dt in ((m, np.int32), (s, np.int8))]
            legs = [tb.RescaleAttr(cs[2 * i + 1], cs[2 * i + 2], LINEAR[i][2], 0) for i in range(2)]
            back = tb.RescaleAttr(cs[5], cs[6], 0, OUT[2], rounding="DOUBLE_ROUND")
            self.run = lambda: ctx.conv2d_add(ts[0], ts[1], ts[2], to, pad, [stride] * 2, [1, 1], zp, 0, epi, legs[0], cs[0], legs[1], back)
            ts = ts + cs
        else:
            self.run = lambda: ctx.conv2d(ts[0], ts[1], ts[2], to, pad, [stride] * 2, [1, 1], zp, 0, epi)
        self.ctx, self.exp, self.to, self.all = ctx, q, to, ts + [to]

    def check(self):
        self.to.upload(np.full(self.exp.shape, 55, np.int8))
        self.run()
        st, out = self.to.download()
        assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), self.exp)

    def free(self):
        for t in self.all:
            t.free()


FORMS = [
    # n, h, w, ic, oc, kernel, join, form
    ((30, 64, 64, 32, 128, 1), False, "conv_chan 192 pixels, 2 slots"),
    ((9, 14, 14, 256, 288, 3), False, "conv_chan 64 pixels, 2 slots"),
    ((32, 56, 56, 64, 256, 1), False, "conv_chan 256 pixels, 2 slots"),
    ((16, 28, 28, 128, 128, 3), False, "conv_chan 128 pixels, 2 slots"),
    ((11, 38, 40, 96, 64, 3), False, "conv_chan 64 pixels, 2 slots, 2 side by side"),
    ((7, 38, 40, 96, 64, 3), False, "lean"),                                    # too few pixels for a window of two
    ((16, 61, 59, 32, 64, 3, 2), False, "conv_chan 64 pixels, 1 slots, 2 side by side"),
    ((17, 30, 30, 32, 64, (5, 3), 1, [2, 2, 1, 1], 0), False, "conv_chan 64 pixels, 2 slots, 2 side by side"),    # no classes
    ((18, 23, 22, 32, 64, 1), False, "conv_chan 64 pixels, 2 slots, 2 side by side"),
    ((1, 28, 28, 128, 128, 3), False, "conv_split 32 pixels, K over 4"),
    ((1, 7, 7, 2048, 512, 1), False, "conv_split 32 pixels, K over 8"),
    ((1, 5, 13, 64, 160, 1), False, "lean"),
    ((16, 30, 30, 64, 160, 3), False, "lean halo"),
    ((1, 97, 87, 32, 64, 1), False, "lean"),
    # channel blocks that are not three quarters full: long products over many pixels
    ((9, 42, 43, 512, 64, 3), False, "conv_chan 192 pixels, 1 slots"),
    ((2, 30, 30, 512, 64, 3, 1, [0, 0, 0, 0]), False, "lean"),
    ((11, 15, 15, 160, 32, 5), False, "lean"),
    # a few channels of a window loaded again for every channel block; many channels of a 1x1 convolution to 64
    ((21, 18, 50, 32, 256, 5), False, "lean"),
    ((8, 33, 50, 320, 64, 1), False, "lean"),
    # joins: the other operand loaded a tile ahead or, with two slots, behind the store of the tile before
    ((30, 64, 64, 32, 128, 1), True, "conv_chan 128 pixels, 3 slots"),
    ((31, 14, 14, 256, 1024, 1), True, "conv_chan 192 pixels, 3 slots"),
    ((8, 28, 28, 128, 256, 3), True, "conv_chan 128 pixels, 2 slots"),
    ((16, 28, 28, 128, 256, 3), True, "conv_chan 192 pixels, 2 slots"),
    ((17, 27, 29, 64, 96, 5), True, "conv_chan 128 pixels, 2 slots"),          # a last tile that is not full
    ((6, 48, 50, 64, 64, 3), True, "conv_chan 64 pixels, 3 slots, 2 side by side"),
    ((1, 6, 6, 32, 128, 1), True, "conv_split 32 pixels, K over 1"),
    ((8, 14, 14, 128, 128, 3), True, "conv_split 32 pixels, K over 2"),
    ((1, 28, 26, 96, 96, 3), True, "conv_split 32 pixels, K over 4"),
    ((8, 14, 14, 128, 128, 5), True, "conv_split 64 pixels, K over 4"),
    ((4, 14, 13, 256, 256, 3), True, "conv_split 64 pixels, K over 4"),
]


@pytest.mark.parametrize("shape,join,form", FORMS)
def test_form(ctx, shape, join, form):
    layer = _Layer(ctx, *shape, join=join)
    for _ in range(2):
        layer.check()
        layer.run()
        assert ctx.last_form() == form and ctx.last_kernel() == "tc_conv_lean_i8" + ("_join" if join else "")
    assert ctx.sync() == tb.Status.OK
    layer.free()


@pytest.mark.parametrize("shape,pad,form", [
    ((1, 224, 224, 3, 64, 7, 2), [3, 2, 3, 2], "conv_chan 64 pixels, 2 slots, 2 side by side"),
    ((5, 131, 128, 3, 32, 3, 2), [1, 1, 1, 0], "conv_chan 64 pixels, 2 slots, 4 side by side"),
    ((2, 128, 129, 3, 64, 7, 2), [3, 2, 3, 3], "lean, a copy per parity"),
])
def test_form_of_few_channels(ctx, shape, pad, form):
    layer = _Layer(ctx, *shape, pad=pad)
    layer.check()
    layer.run()
    assert ctx.last_form() == form
    layer.free()


@pytest.mark.parametrize("shape,join,form", [
    ((16, 30, 30, 64, 160, 3), False, "lean halo"),
    ((16, 30, 31, 64, 160, 1), False, "lean"),
    ((8, 28, 28, 128, 256, 3), False, "conv_chan 128 pixels, 2 slots"),
    ((31, 14, 14, 256, 1024, 1), True, "conv_chan 192 pixels, 3 slots"),
    ((8, 28, 28, 128, 256, 3), True, "conv_chan 128 pixels, 2 slots"),
    ((8, 14, 14, 128, 128, 5), True, "conv_split 64 pixels, K over 4"),
])
def test_gives_up_and_recovers(ctx, shape, join, form):
    """A wait limit far below the latency of a load from memory: the call reports TB200_INTERNAL and the next one is exact."""
    layer = _Layer(ctx, *shape, join=join)
    layer.check()
    ctx.set_wait_limit(100)
    try:
        layer.run()
        assert ctx.last_form() == form
        assert ctx.sync(check=False) == tb.Status.INTERNAL
    finally:
        ctx.set_wait_limit(4000000000)
    layer.check()
    layer.free()


def test_form_of_a_view(ctx):
    """A slice (pitch of its parent) through the tap loads of two pixels side by side."""
    _, x, wt, b, mult, shift = _operands(67, 3, 73, 72, 64, 64, 3, 3)
    ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift)]
    cut = ts[0].slice([0, 1, 2, 0], [3, 71, 68, 64])
    exp = _conv(x[:, 1:72, 2:70], wt, b, mult, shift, [1] * 4, [1, 1], [1, 1], -128, "DOUBLE_ROUND", -128, 127)
    to  = ctx.empty(I8, exp.shape)
    epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
    for _ in range(2):
        ctx.conv2d(cut, ts[1], ts[2], to, [1] * 4, [1, 1], [1, 1], -128, 0, epi)
        assert ctx.last_form().endswith("2 side by side"), ctx.last_form()
        st, out = to.download()
        assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
    cut.free()
    for t in ts + [to]:
        t.free()
