"""int8 DEPTHWISE_CONV2D + RESCALE on the sliding kernel, bit for bit against the CPU oracle: both windows and strides, odd
channel counts, odd rows and row ends, padding wider than needed, a narrow CLAMP, SINGLE_ROUND, one scale for all channels,
constants replaced by an upload, and operands whose records are not usable (the general kernels take over)."""
import numpy as np
import pytest

import reference_model_b200 as tb
from oracle import oracle as orc
from tests import util

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = tb.Context(0)
    yield c
    c.close()


# N, IH, IW, C, K, stride, pad, in_zp, rounding, per channel, clamp
CASES = [(2, 31, 33, 16, 3, 1, [1, 1, 1, 1], -128, "DOUBLE_ROUND", True, (-128, 127)),
         (3, 30, 28, 69, 3, 1, [1, 1, 1, 1], 5, "DOUBLE_ROUND", True, (-100, 90)),
         (5, 29, 35, 42, 3, 2, [1, 1, 1, 1], -128, "SINGLE_ROUND", True, (-128, 127)),
         (4, 24, 28, 144, 3, 2, [1, 0, 1, 0], 0, "DOUBLE_ROUND", False, (0, 127)),
         (1, 18, 19, 65, 5, 1, [2, 2, 2, 2], -7, "DOUBLE_ROUND", True, (-128, 127)),
         (2, 27, 41, 80, 5, 2, [2, 2, 2, 2], 127, "SINGLE_ROUND", True, (-128, 127)),
         (40, 1, 2, 960, 3, 1, [1, 1, 1, 1], -128, "DOUBLE_ROUND", True, (-128, 127)),
         (3, 20, 16, 24, 3, 1, [2, 2, 2, 2], 11, "DOUBLE_ROUND", True, (-128, 127)),
         (2, 60, 61, 3, 5, 1, [2, 2, 2, 2], 3, "DOUBLE_ROUND", True, (-128, 127))]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_depthwise_slide(ctx, case):
    N, IH, IW, C, K, s, pad, izp, rounding, per_ch, clamp = CASES[case]
    r = util.rng(1900 + case)
    OH, OW = orc.conv_out_hw(IH, IW, K, K, pad, [s, s], [1, 1])
    N = max(N, -(-(1 << 20) // (OH * OW * C * K * K)))    # 2^20 multiply-adds: below, other kernels run
    x = r.integers(-128, 128, size=(N, IH, IW, C), dtype=np.int8)
    w = r.integers(-128, 128, size=(K, K, C, 1), dtype=np.int8)
    b = r.integers(-65536, 65536, size=C).astype(np.int32)
    mult, shift = util.rescale_params(r, C if per_ch else 1)
    tx, tw, tbias, tm, ts = (ctx.from_numpy(v) for v in (x, w, b, mult, shift))
    epi = tb.Epilogue(tb.RescaleAttr(tm, ts, 0, -5, True, rounding, per_channel=per_ch), clamp)

    def expect():
        acc = orc.depthwise_conv2d(x, w, b, pad, [s, s], [1, 1], izp, 0, nthreads=8)
        est, exp = orc.rescale(acc, mult, shift, per_ch, True, rounding, 0, -5, 32, 8)
        assert est == orc.VALID
        return np.clip(exp, *clamp)

    exp = expect()
    to = ctx.empty(tb.DType.INT8, exp.shape)
    ctx.depthwise_conv2d(tx, tw, tbias, to, pad, [s, s], [1, 1], izp, 0, epi)
    assert ctx.last_kernel() == "depthwise_slide_i8", (ctx.last_kernel(), exp.size)
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out, exp), "%d of %d differ" % ((out != exp).sum(), exp.size)
    if case == 0:
        w = r.integers(-128, 128, size=w.shape, dtype=np.int8)
        tw.upload(w)
        ctx.depthwise_conv2d(tx, tw, tbias, to, pad, [s, s], [1, 1], izp, 0, epi)
        assert np.array_equal(to.download()[1], expect())
        # a shift whose accepted range the accumulators could leave: no usable record, the general kernel checks every value
        ts.upload(np.full_like(shift, 12))
        ctx.depthwise_conv2d(tx, tw, tbias, to, pad, [s, s], [1, 1], izp, 0, epi)
        assert ctx.last_kernel() == "depthwise3x3_i8x16"
        assert ctx.sync(check=False) == tb.Status.UNPREDICTABLE
    for t in (tx, tw, tbias, tm, ts, to):
        t.free()


@pytest.mark.parametrize("C,K,stride", [(24, 3, 1), (21, 5, 2), (33, 3, 2)])
def test_general_arithmetic_and_captured_graph(ctx, C, K, stride):
    """Constants whose records are not usable from the first call on (the kernel's general arithmetic), and constants replaced
    under a captured graph: usable, not usable, usable, out of the accepted range."""
    r = util.rng(1950 + C)
    p = K // 2
    pad, IH, IW = [p, p, p, p], 31, 33
    OH, OW = orc.conv_out_hw(IH, IW, K, K, pad, [stride] * 2, [1, 1])
    N = -(-(1 << 20) // (OH * OW * C * K * K))
    x = r.integers(-128, 128, size=(N, IH, IW, C), dtype=np.int8)
    w = r.integers(-128, 128, size=(K, K, C, 1), dtype=np.int8)
    b = r.integers(-1000, 1000, size=C).astype(np.int32)
    acc = orc.depthwise_conv2d(x, w, b, pad, [stride] * 2, [1, 1], 9, 0, nthreads=8)
    bits = int(np.abs(acc).max()).bit_length()
    assert (1 << (bits - 1)) < K * K * 255 * 128 and np.abs(acc).max() >= 1 << (bits - 2)
    good = util.rescale_params(r, C)
    tight, low = ((np.full(C, 1 << 20, np.int32), np.full(C, bits + d, np.int8)) for d in (1, -1))
    tx, tw, tbias, tm, ts = (ctx.from_numpy(v) for v in (x, w, b, *tight))
    to = ctx.empty(tb.DType.INT8, acc.shape)
    epi = tb.Epilogue(tb.RescaleAttr(tm, ts, 0, -5, True, "DOUBLE_ROUND", per_channel=True), (-128, 100))
    call = lambda: ctx.depthwise_conv2d(tx, tw, tbias, to, pad, [stride] * 2, [1, 1], 9, 0, epi)

    def check(params):
        st, out = to.download(check=False)
        est, exp = orc.rescale(acc, *params, True, True, "DOUBLE_ROUND", 0, -5, 32, 8)
        assert est == orc.VALID and st == tb.Status.OK and np.array_equal(out, np.clip(exp, -128, 100))

    call()
    assert ctx.last_kernel() == "depthwise_slide_i8"
    check(tight)
    tm.upload(good[0]), ts.upload(good[1])
    call()
    check(good)
    ctx.capture_begin()
    call()
    graph = ctx.capture_end()
    for params in (good, tight, good):
        tm.upload(params[0]), ts.upload(params[1])
        ctx.graph_launch(graph)
        check(params)
    tm.upload(low[0]), ts.upload(low[1])
    ctx.graph_launch(graph)
    assert ctx.sync(check=False) == tb.Status.UNPREDICTABLE
    ctx.graph_destroy(graph)
    for t in (tx, tw, tbias, tm, ts, to):
        t.free()


def test_weights_that_an_operator_writes(ctx):
    """Such weights are read where they are: no packing before every call, and never a packed copy that has gone stale."""
    r = util.rng(1990)
    N, C, K = 3, 24, 3
    x = r.integers(-128, 128, size=(N, 57, 57, C), dtype=np.int8)
    w32 = r.integers(-100, 100, size=(K, K, C, 1)).astype(np.int32)
    mult, shift = util.rescale_params(r, C)
    tx, tw32, tw, tbias, tm, ts = (ctx.from_numpy(v) for v in (x, w32, w32.astype(np.int8), np.zeros(C, np.int32), mult, shift))
    one, two = ctx.from_numpy(np.full(1, 1 << 30, np.int32)), ctx.from_numpy(np.full(1, 30, np.int8))
    to = ctx.empty(tb.DType.INT8, x.shape)
    epi = tb.Epilogue(tb.RescaleAttr(tm, ts, 0, 0, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
    for rep in range(3):
        if rep:
            w32 = r.integers(-100, 100, size=w32.shape).astype(np.int32)
            tw32.upload(w32)
            ctx.rescale(tw32, tb.RescaleAttr(one, two, 0, 0, True, "SINGLE_ROUND"), tw)
        launches = ctx.launch_count()
        ctx.depthwise_conv2d(tx, tw, tbias, to, [1] * 4, [1, 1], [1, 1], 0, 0, epi)
        assert rep == 0 or ctx.launch_count() == launches + 1
        acc = orc.depthwise_conv2d(x, w32.astype(np.int8), np.zeros(C, np.int32), [1] * 4, [1, 1], [1, 1], 0, 0, nthreads=8)
        est, exp = orc.rescale(acc, mult, shift, True, True, "DOUBLE_ROUND", 0, 0, 32, 8)
        st, out = to.download()
        assert est == orc.VALID and st == tb.Status.OK and np.array_equal(out, exp)
    for t in (tx, tw32, tw, tbias, tm, ts, one, two, to):
        t.free()
