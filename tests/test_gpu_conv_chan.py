"""int8 CONV2D + RESCALE with channels on the accumulator's rows (conv_chan.cu): remainders of pixels, channels and tiles, the
two-pixel form of layers with at most 64 channels, and the residual join behind it, bit for bit against the oracle."""
import numpy as np
import pytest

import reference_model_b200 as tb
from oracle import oracle as orc
from tests import util

pytestmark = pytest.mark.gpu

I8 = tb.DType.INT8


@pytest.fixture(scope="module")
def ctx():
    c = tb.Context(0)
    yield c
    c.close()


def _operands(seed, n, h, w, ic, oc, kh, kw):
    r = util.rng(seed)
    x, wt, b = util.conv_int8_case(r, n, h, w, ic, oc, kh, kw)
    mult, shift = util.rescale_params(r, oc)
    return r, x, wt, b, mult, np.maximum(shift, 33 if kh * kw * ic > 512 else 30).astype(np.int8)


def _conv(x, wt, b, mult, shift, pad, stride, dil, zp, rounding, lo, hi):
    acc = orc.conv2d(x, wt, b, pad, stride, dil, zp, 0, nthreads=orc.num_procs())
    est, q = orc.rescale(acc, mult, shift, True, True, rounding, 0, -3, 32, 8)
    assert est == orc.VALID
    return np.clip(q, lo, hi)


CASES = [
    # n, h, w, ic, oc, (kh, kw), pad, stride, dilation, zero point
    (1, 1, 1, 32, 128, (1, 1), [0, 0, 0, 0], [1, 1], [1, 1], 5),            # one pixel
    (1, 5, 13, 64, 160, (1, 1), [0, 0, 0, 0], [1, 1], [1, 1], -128),        # 65 pixels, a block of 32 channels
    (30, 64, 64, 32, 128, (1, 1), [0, 0, 0, 0], [1, 1], [1, 1], 3),         # several tiles per CTA
    (18, 23, 22, 32, 64, (1, 1), [0, 0, 0, 0], [1, 1], [1, 1], -128),       # two pixels per row
    (2, 67, 63, 32, 64, (1, 1), [0, 0, 0, 0], [1, 1], [1, 1], -128),        # ... odd width
    (1, 97, 87, 32, 64, (1, 1), [0, 0, 0, 0], [1, 1], [1, 1], -128),        # odd number of pixels
    (7, 38, 40, 96, 64, (3, 3), [1, 1, 1, 1], [1, 1], [1, 1], -128),        # two pixels per row, window, classes
    (9, 61, 59, 32, 64, (3, 3), [1, 1, 1, 1], [2, 2], [1, 1], 7),           # ... stride 2
    (11, 30, 30, 32, 64, (5, 3), [0, 2, 1, 1], [1, 1], [1, 1], 0),           # ... no classes, uneven padding
    (1, 11, 11, 64, 96, (3, 3), [2, 2, 2, 2], [1, 1], [2, 2], -7),          # dilation
    (2, 17, 9, 128, 256, (1, 1), [0, 0, 0, 0], [2, 2], [1, 1], 1),          # strided 1x1
    (2, 17, 19, 32, 192, (3, 3), [1, 1, 1, 1], [2, 1], [1, 1], -128),       # a stride per axis
    (5, 7, 7, 512, 512, (3, 3), [1, 1, 1, 1], [1, 1], [1, 1], -128),        # long K
    (9, 14, 14, 256, 288, (3, 3), [1, 1, 1, 1], [1, 1], [1, 1], 100),
    # few tiles: K split over clusters
    (1, 28, 28, 128, 128, (3, 3), [1, 1, 1, 1], [1, 1], [1, 1], -128),      # nine chunks over four CTAs, the last without any
    (1, 7, 7, 2048, 512, (1, 1), [0, 0, 0, 0], [1, 1], [1, 1], 11),         # over eight
    (1, 10, 20, 96, 32, (3, 3), [1, 1, 1, 1], [1, 1], [1, 1], -128),        # 27 short chunks, a quarter of a channel block
    (1, 12, 11, 64, 384, (5, 5), [2, 2, 2, 2], [1, 1], [1, 1], -128),
    (2, 13, 17, 256, 192, (3, 3), [1, 1, 1, 1], [2, 2], [1, 1], 64),
    (1, 31, 19, 384, 32, (3, 3), [1, 1, 1, 1], [1, 1], [1, 1], -1),
]


@pytest.mark.parametrize("rounding", ["SINGLE_ROUND", "DOUBLE_ROUND"])
@pytest.mark.parametrize("case", CASES)
def test_against_oracle(ctx, case, rounding):
    n, h, w, ic, oc, (kh, kw), pad, stride, dil, zp = case
    _, x, wt, b, mult, shift = _operands(n * h + oc, n, h, w, ic, oc, kh, kw)
    lo, hi = (-128, 127) if rounding == "DOUBLE_ROUND" else (-90, 101)
    exp = _conv(x, wt, b, mult, shift, pad, stride, dil, zp, rounding, lo, hi)
    ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift)]
    to = ctx.empty(I8, exp.shape)
    epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, rounding, per_channel=True), (lo, hi))
    for _ in range(2):
        to.upload(np.full(exp.shape, 55, np.int8))
        ctx.conv2d(ts[0], ts[1], ts[2], to, pad, stride, dil, zp, 0, epi)
        assert ctx.last_kernel() == "tc_conv_lean_i8"
        st, out = to.download()
        assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
    for t in ts + [to]:
        t.free()


def test_view_as_input(ctx):
    """A slice (pitch of its parent) through the tap loads, with and without a second pixel per row."""
    for oc, k in ((64, 3), (128, 1)):
        _, x, wt, b, mult, shift = _operands(3 + oc, 2, 73, 72, 64, oc, k, k)
        pad = [k // 2] * 4
        ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift)]
        cut = ts[0].slice([0, 1, 2, 0], [2, 71, 68, 64])
        exp = _conv(x[:, 1:72, 2:70], wt, b, mult, shift, pad, [1, 1], [1, 1], -128, "DOUBLE_ROUND", -128, 127)
        to  = ctx.empty(I8, exp.shape)
        epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
        for _ in range(2):
            ctx.conv2d(cut, ts[1], ts[2], to, pad, [1, 1], [1, 1], -128, 0, epi)
            st, out = to.download()
            assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
        cut.free()
        for t in ts + [to]:
            t.free()


# ------------------------------------------------------------------------------------------------ residual join
def _join(q, other, legs, out, rounding, lo, hi):
    (ma, sa, za), (mb, sb, zb), (mo, so, zo) = legs[0], legs[1], out
    e1, a = orc.rescale(q, [ma], [sa], False, True, "SINGLE_ROUND", za, 0, 8, 32)
    e2, b = orc.rescale(other, [mb], [sb], False, True, "SINGLE_ROUND", zb, 0, 8, 32)
    e3, s = orc.add(a, b)
    e4, y = orc.rescale(s, [mo], [so], False, True, rounding, 0, zo, 32, 8)
    st = tb.Status.OK if e1 == e2 == e3 == e4 == orc.VALID else tb.Status.UNPREDICTABLE
    return st, np.clip(y, lo, hi)


LINEAR = ((1 << 30, 21, -3), (1 << 29, 21, 4))
JOINS = [
    # legs, output (multiplier, shift, zero point), rounding, clip, kernel
    (LINEAR, (1700000001, 40, -128), "DOUBLE_ROUND", (-128, 127), "join"),
    (LINEAR, (1300000001, 39, 9), "SINGLE_ROUND", (-100, 90), "join"),
    (((1 << 30, 30, 0), (1 << 30, 29, 0)), (1500000001, 32, 0), "DOUBLE_ROUND", (-128, 127), "join"),
    (((1 << 30, 30, 0), (1 << 30, 28, 3)), (1500000001, 31, 0), "DOUBLE_ROUND", (-128, 127), "join"),
    (((1 << 30, 30, 0), (1 << 30, 30, 0)), (1 << 30, 31, 0), "SINGLE_ROUND", (-128, 127), "join"),       # many ties
    (((1518500250, 21, -3), (1 << 29, 21, 4)), (1700000001, 41, -128), "DOUBLE_ROUND", (-128, 127), "apart"),
    (((1 << 30, 11, -3), (1 << 30, 11, 4)), (1700000001, 50, 0), "DOUBLE_ROUND", (-128, 127), "apart"),  # beyond 16 bits
]


@pytest.mark.parametrize("shape", [(1, 6, 6, 32, 128, 1), (30, 64, 64, 32, 128, 1), (5, 48, 50, 64, 64, 3), (3, 9, 9, 64, 96, 3), (40, 7, 7, 512, 512, 1),
                                   (1, 7, 7, 512, 512, 3), (1, 14, 14, 256, 320, 1), (1, 28, 26, 96, 96, 3), (31, 14, 14, 256, 1024, 1)])
@pytest.mark.parametrize("join", JOINS)
def test_join_against_oracle(ctx, shape, join):
    n, h, w, ic, oc, k = shape
    legs, outp, rounding, (lo, hi), kind = join
    r, x, wt, b, mult, shift = _operands(n + oc, n, h, w, ic, oc, k, k)
    pad = [k // 2] * 4
    q = _conv(x, wt, b, mult, shift, pad, [1, 1], [1, 1], -128, "DOUBLE_ROUND", -128, 127)
    other = r.integers(-128, 128, size=q.shape).astype(np.int8)
    est, exp = _join(q.astype(np.int8), other, legs, outp, rounding, lo, hi)
    assert est == tb.Status.OK
    ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift, other)]
    cs = [ctx.from_numpy(np.array([v], dt)) for m, s, _ in legs + (outp,) for v, dt in ((m, np.int32), (s, np.int8))]
    at = [tb.RescaleAttr(cs[2 * i], cs[2 * i + 1], legs[i][2], 0) for i in range(2)]
    ao = tb.RescaleAttr(cs[4], cs[5], 0, outp[2], rounding=rounding)
    to  = ctx.empty(I8, exp.shape)
    epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
    for _ in range(2):
        ctx.conv2d_add(ts[0], ts[1], ts[2], to, pad, [1, 1], [1, 1], -128, 0, epi, at[0], ts[5], at[1], ao, (lo, hi))
        assert (ctx.last_kernel() == "tc_conv_lean_i8_join") == (kind == "join"), ctx.last_kernel()
        st, out = to.download()
        assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
    for t in ts + cs + [to]:
        t.free()


def test_join_follows_constants_under_a_captured_graph(ctx):
    """Constants uploaded under a captured graph: legs that are no multiples any more (the kernel's general form), legs
    whose REQUIRE fails for some operand, and back."""
    n, h, w, ic, oc = 2, 9, 7, 32, 96    # a last tile and a last channel block that are not full
    r, x, wt, b, mult, shift = _operands(77, n, h, w, ic, oc, 1, 1)
    q = _conv(x, wt, b, mult, shift, [0] * 4, [1, 1], [1, 1], -128, "DOUBLE_ROUND", -128, 127)
    other = r.integers(-128, 128, size=q.shape).astype(np.int8)
    ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift, other)]
    outp = (1700000001, 41, -128)
    cs = [ctx.from_numpy(np.array([v], dt)) for m, s, _ in LINEAR + (outp,) for v, dt in ((m, np.int32), (s, np.int8))]
    at = [tb.RescaleAttr(cs[2 * i], cs[2 * i + 1], LINEAR[i][2], 0) for i in range(2)]
    ao = tb.RescaleAttr(cs[4], cs[5], 0, -128, rounding="DOUBLE_ROUND")
    to  = ctx.empty(I8, q.shape)
    epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
    run = lambda: ctx.conv2d_add(ts[0], ts[1], ts[2], to, [0] * 4, [1, 1], [1, 1], -128, 0, epi, at[0], ts[5], at[1], ao)
    run()
    assert ctx.sync() == tb.Status.OK and ctx.last_kernel() == "tc_conv_lean_i8_join"
    ctx.capture_begin()
    run()
    g = ctx.capture_end()
    for m, s in ((1518500250, 21), (1 << 20, 8), (1 << 30, 21)):
        cs[0].upload(np.array([m], np.int32))
        cs[1].upload(np.array([s], np.int8))
        est, exp = _join(q.astype(np.int8), other, ((m, s, -3), LINEAR[1]), outp, "DOUBLE_ROUND", -128, 127)
        ctx.graph_launch(g)
        st, out = to.download(check=False)
        assert st == est, (m, s)
        if est == tb.Status.OK:
            assert np.array_equal(out.astype(np.int32), exp)
    ctx.graph_destroy(g)
    # the output may not overlap the other operand
    assert ctx.conv2d_add(ts[0], ts[1], ts[2], to, [0] * 4, [1, 1], [1, 1], -128, 0, epi, at[0], to, at[1], ao, check=False) == tb.Status.ERROR
    for t in ts + cs + [to]:
        t.free()


def test_split_form_gives_up_and_recovers(ctx):
    """A wait limit far below the latency of a load from memory: every CTA of the clusters leaves, the call reports
    TB200_INTERNAL and the next one is exact."""
    _, x, wt, b, mult, shift = _operands(5, 1, 7, 7, 512, 512, 3, 3)
    exp = _conv(x, wt, b, mult, shift, [1] * 4, [1, 1], [1, 1], -128, "DOUBLE_ROUND", -128, 127)
    ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift)]
    to = ctx.empty(I8, exp.shape)
    epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
    run = lambda: ctx.conv2d(ts[0], ts[1], ts[2], to, [1] * 4, [1, 1], [1, 1], -128, 0, epi)
    run()
    assert ctx.sync() == tb.Status.OK
    ctx.set_wait_limit(100)
    try:
        run()
        assert ctx.sync(check=False) == tb.Status.INTERNAL
    finally:
        ctx.set_wait_limit(4000000000)
    run()
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
    for t in ts + [to]:
        t.free()


# ------------------------------------------------------------------------------------------------ constants under a captured graph
REPLACED = [
    # n, h, w, ic, oc, (kh, kw), pad, stride, zero point, join behind it
    (30, 64, 64, 32, 128, (1, 1), [0, 0, 0, 0], [1, 1], 3, False),
    (9, 14, 14, 256, 288, (3, 3), [1, 1, 1, 1], [1, 1], 100, False),      # border classes
    (11, 38, 40, 96, 64, (3, 3), [1, 1, 1, 1], [1, 1], -128, False),      # two pixels side by side
    (1, 28, 28, 128, 128, (3, 3), [1, 1, 1, 1], [1, 1], -128, False),     # K split over clusters
    (5, 7, 7, 512, 512, (3, 3), [1, 1, 1, 1], [1, 1], -128, False),
    (16, 30, 30, 64, 160, (3, 3), [1, 1, 1, 1], [1, 1], -128, False),     # a pixel per thread
    (16, 30, 31, 64, 160, (1, 1), [0, 0, 0, 0], [1, 1], 5, False),
    (1, 224, 224, 3, 64, (7, 7), [3, 2, 3, 2], [2, 2], -128, False),      # few channels, pixels side by side
    (2, 128, 129, 3, 64, (7, 7), [3, 2, 3, 3], [2, 2], 9, False),         # ... an odd number of columns
    (30, 64, 64, 32, 128, (1, 1), [0, 0, 0, 0], [1, 1], 3, True),
    (31, 14, 14, 256, 1024, (1, 1), [0, 0, 0, 0], [1, 1], -128, True),
    (6, 31, 30, 96, 96, (3, 3), [1, 1, 1, 1], [1, 1], -128, True),
    (1, 14, 14, 256, 320, (1, 1), [0, 0, 0, 0], [1, 1], -128, True),
]


@pytest.mark.parametrize("rounding", ["SINGLE_ROUND", "DOUBLE_ROUND"])
@pytest.mark.parametrize("case", REPLACED)
def test_records_follow_constants_under_a_captured_graph(ctx, case, rounding):
    """Multipliers and shifts uploaded under a captured graph: usable records, ones that are not (the RESCALE accepts every value
    there is, but not every value its K could make), a REQUIRE that fails, and back."""
    n, h, w, ic, oc, (kh, kw), pad, stride, zp, join = case
    r, x, wt, b, mult, shift = _operands(n * h + oc, n, h, w, ic, oc, kh, kw)
    acc = orc.conv2d(x, wt, b, pad, stride, [1, 1], zp, 0, nthreads=orc.num_procs())
    bits = int(np.abs(acc).max()).bit_length()
    # |acc| < 2^bits, so shift bits + 1 is accepted; the record of a K that reaches 2^(bits + 1) is not usable
    assert kh * kw * ic * 255 * 128 >= 1 << (bits + 1)
    good = (mult, shift)
    tight, low = ((np.full(oc, 1 << 20, np.int32), np.full(oc, bits + d, np.int8)) for d in (1, -1))
    ts = [ctx.from_numpy(v) for v in (x, wt, b, mult, shift)]
    other = r.integers(-128, 128, size=acc.shape).astype(np.int8)
    outp, lo, hi = (1700000001, 41, -128), -100, 90
    cs = [ctx.from_numpy(other)]
    cs += [ctx.from_numpy(np.array([v], dt)) for m, s, _ in LINEAR + (outp,) for v, dt in ((m, np.int32), (s, np.int8))]
    legs = [tb.RescaleAttr(cs[2 * i + 1], cs[2 * i + 2], LINEAR[i][2], 0) for i in range(2)]
    back = tb.RescaleAttr(cs[5], cs[6], 0, outp[2], rounding="DOUBLE_ROUND")
    to  = ctx.empty(I8, acc.shape)
    epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, rounding, per_channel=True), (lo, hi))
    if join:
        run = lambda: ctx.conv2d_add(ts[0], ts[1], ts[2], to, pad, stride, [1, 1], zp, 0, epi, legs[0], cs[0], legs[1], back)
    else:
        run = lambda: ctx.conv2d(ts[0], ts[1], ts[2], to, pad, stride, [1, 1], zp, 0, epi)
    run()
    assert ctx.sync() == tb.Status.OK and ctx.last_kernel() == "tc_conv_lean_i8" + ("_join" if join else "")
    ctx.capture_begin()
    run()
    g = ctx.capture_end()
    for params in (good, tight, low, good):
        ts[3].upload(params[0]), ts[4].upload(params[1])
        to.upload(np.full(acc.shape, 55, np.int8))
        ctx.graph_launch(g)
        st, out = to.download(check=False)
        est, q = orc.rescale(acc, *params, True, True, rounding, 0, -3, 32, 8)
        assert (est == orc.VALID) == (params is not low)
        if params is low:
            assert st == tb.Status.UNPREDICTABLE
            continue
        exp = np.clip(q, lo, hi)
        if join:
            est, exp = _join(exp.astype(np.int8), other, LINEAR, outp, "DOUBLE_ROUND", -128, 127)
        assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
    ctx.graph_destroy(g)
    for t in ts + cs + [to]:
        t.free()
