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
