"""fp32 MATMUL and CONV2D at the edges of the tiled FFMA kernel: row / column / K remainders of every tile size, K split
over a cluster, unaligned rows, window shapes, strides, dilation, a view, infinite weights under padding; against the
fp64 oracle under the DOT_PRODUCT rule.  And on the tensor cores (three bf16 parts per operand): remainders, accuracy,
operands that parts cannot carry, waits that give up."""
import numpy as np
import pytest

import reference_model_b200 as tb
from oracle import oracle as orc
from tests import util
from tests.test_gpu_parity import _dot_check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = tb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (3, 17, 15, 33), (2, 129, 33, 129), (1, 64, 2048, 64), (1, 1, 4096, 1000),
                                   (5, 15, 21, 487), (2, 257, 100, 260), (150, 130, 17, 132), (1, 33, 511, 65)])
def test_matmul_f32_edges(ctx, shape):
    N, H, C, W = shape
    r = util.rng(900 + H + C)
    a, b = r.standard_normal((N, H, C)).astype(np.float32), r.standard_normal((N, C, W)).astype(np.float32)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (N, H, W))
    ctx.matmul(ta, tbb, to)
    assert ctx.last_kernel() == "sgemm_f32"
    st, out = to.download()
    ok, info = _dot_check(out, a.astype(np.float64), b.astype(np.float64), orc.matmul, C, "fp32")
    assert st == tb.Status.OK and ok, info
    for t in (ta, tbb, to):
        t.free()


# N, IH, IW, IC, OC, KH, KW, stride, dilation, pad, bias length
CONV = [(1, 5, 5, 1, 1, 1, 1, [1, 1], [1, 1], [0, 0, 0, 0], 1), (2, 13, 9, 5, 7, 3, 3, [1, 1], [1, 1], [1, 1, 1, 1], 7),
        (3, 17, 20, 16, 65, 3, 2, [2, 1], [1, 2], [1, 1, 2, 0], 65), (1, 9, 9, 130, 129, 1, 1, [2, 2], [1, 1], [0, 0, 0, 0], 129),
        (4, 30, 31, 3, 64, 5, 5, [1, 1], [1, 1], [2, 2, 2, 2], 64), (1, 4, 4, 512, 33, 3, 3, [1, 1], [1, 1], [1, 1, 1, 1], 33),
        (8, 28, 28, 40, 128, 3, 3, [1, 1], [1, 1], [1, 1, 1, 1], 128),
        (1, 5, 5, 21, 1, 1, 1, [1, 1], [1, 1], [0, 0, 0, 0], 1)]


@pytest.mark.parametrize("case", range(len(CONV)))
def test_conv_f32_edges(ctx, case):
    N, IH, IW, IC, OC, KH, KW, stride, dil, pad, nb = CONV[case]
    r = util.rng(950 + case)
    x, w = r.standard_normal((N, IH, IW, IC)).astype(np.float32), r.standard_normal((OC, KH, KW, IC)).astype(np.float32)
    b = r.standard_normal(nb).astype(np.float32)
    OH, OW = orc.conv_out_hw(IH, IW, KH, KW, pad, stride, dil)
    ref = orc.conv2d(x, w, b, pad, stride, dil, mode="f64")
    bnd = orc.conv2d(x, w, b, pad, stride, dil, mode="f64", bounds=True)
    ksb = orc.dot_product_ksb(KH * KW * IC + 1, "fp32", "fp32")
    tx, tw, tbias, to = ctx.from_numpy(x), ctx.from_numpy(w), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (N, OH, OW, OC))
    for cache in (ctx.CACHE_ON, ctx.CACHE_OFF):    # without the cache a padded layer runs the untiled kernel
        ctx.const_cache_control(cache)
        ctx.conv2d(tx, tw, tbias, to, pad, stride, dil)
        tiled = KH * KW * IC > 20 and (cache or not any(pad))    # (shallow sums run one thread per output)
        assert ctx.last_kernel() == ("conv_f32" if tiled else "conv2d_direct")
        st, out = to.download()
        ok, info = orc.verify_dot_product(out, ref, bnd, ksb, out="fp32")
        assert st == tb.Status.OK and ok, (cache, info)
    ctx.const_cache_control(ctx.CACHE_ON)
    ctx.conv2d(tx, tw, tbias, to, pad, stride, dil, epilogue=tb.Epilogue(None, (-0.5, 1.0)))
    st, clamped = to.download()
    assert np.array_equal(clamped, np.clip(out, -0.5, 1.0)) or orc.verify_dot_product(
        clamped, np.clip(ref, -0.5, 1.0), bnd, ksb, out="fp32")[0]
    for t in (tx, tw, tbias, to):
        t.free()


def test_conv_f32_view_and_infinite_weight(ctx):
    r = util.rng(970)
    x, w = r.standard_normal((2, 9, 9, 8)).astype(np.float32), r.standard_normal((5, 3, 3, 8)).astype(np.float32)
    b = r.standard_normal(5).astype(np.float32)
    tx, tw, tbias, to = ctx.from_numpy(x), ctx.from_numpy(w), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (2, 7, 7, 5))
    view = tx.slice([0, 1, 2, 0], [2, 7, 7, 8])
    ctx.conv2d(view, tw, tbias, to, [1, 1, 1, 1], [1, 1], [1, 1])
    assert ctx.last_kernel() == "conv_f32"
    xv = np.ascontiguousarray(x[:, 1:8, 2:9])
    args = ([1, 1, 1, 1], [1, 1], [1, 1])
    ok, info = orc.verify_dot_product(to.download()[1], orc.conv2d(xv, w, b, *args, mode="f64"),
                                      orc.conv2d(xv, w, b, *args, mode="f64", bounds=True), orc.dot_product_ksb(73, "fp32", "fp32"))
    assert ok, info
    # new weights through an upload, one of them infinite: skipped taps stay skipped (the corner has no NaN)
    w[0, 0, 0, 0] = np.inf
    tw.upload(w)
    ctx.conv2d(view, tw, tbias, to, *args)
    assert ctx.last_kernel() == "conv2d_direct"
    out = to.download()[1]
    assert not np.isnan(out).any() and np.isinf(out[:, 1:, 1:, 0]).all() and np.isfinite(out[:, 0, :, 0]).all()


# Products deep and large enough for the tensor-core kernel (three bf16 parts per operand): whole tiles, row / column / K
# remainders, rows of any alignment, the smallest depth it takes.
SPLIT = [(148, 128, 256, 128), (70, 255, 319, 256), (40, 250, 258, 383), (37, 256, 1000, 250), (3, 1000, 515, 777)]


@pytest.mark.parametrize("shape", SPLIT)
def test_matmul_f32_split(ctx, shape):
    N, H, C, W = shape
    r = util.rng(990 + H + C)
    a, b = r.standard_normal((N, H, C)).astype(np.float32), r.standard_normal((N, C, W)).astype(np.float32)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (N, H, W))
    ctx.matmul(ta, tbb, to)
    st, out = to.download()
    ref = a.astype(np.float64) @ b.astype(np.float64)
    # 24-bit operands, six partial products, a cut-off sum per 64 K elements: far below 2^-22 of the sum of magnitudes
    assert st == tb.Status.OK and np.all(np.abs(out - ref) <= 2.0 ** -22 * (np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)))
    assert np.linalg.norm(out - ref) <= 3e-7 * np.linalg.norm(ref)
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("what", ["one_term", "cut", "round", "normal", "positive"])
def test_matmul_f32_split_accuracy(ctx, what):
    """Against the kernel that rounds every multiply-add, and where the parts lose most: operands whose lower bits are all ones
    (parts that were cut off would leave out 2^-21 of every product) and those for which rounded parts leave out most, 2^-24."""
    N, H, C, W = 40, 256, 320, 256
    r = util.rng(78)
    if what in ("cut", "round"):
        v = np.array([0x3F80FFFF if what == "cut" else 0x3F807FC0], np.uint32).view(np.float32)[0]
        a, b = np.full((N, H, C), v, np.float32), np.full((N, C, W), v, np.float32)
    elif what == "one_term":
        a, b = np.zeros((N, H, C), np.float32), r.uniform(1, 2, (N, C, W)).astype(np.float32)
        a[:, np.arange(H), (np.arange(H) * 7) % C] = r.uniform(1, 2, (N, H))
    else:
        draw = r.standard_normal if what == "normal" else lambda s: r.uniform(0.5, 1.0, s)
        a, b = draw((N, H, C)).astype(np.float32), draw((N, C, W)).astype(np.float32)
    ref, err = a.astype(np.float64) @ b.astype(np.float64), []
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (N, H, W))
    for policy in (0, 1):
        old = ctx.set_kernel_policy(policy)
        ctx.matmul(ta, tbb, to)
        ctx.set_kernel_policy(old)
        st, out = to.download()
        assert st == tb.Status.OK
        err.append((np.linalg.norm(out - ref) / np.linalg.norm(ref), np.abs(out / ref - 1).max()))
    print(what, err)
    if what in ("cut", "round"):
        # left out 2^-24; the stage's sum rounded, 2^-24; the sums of one to five stages rounded, a fifth more of 2^-24 each
        assert err[0][1] <= 5 * 2.0 ** -24
    elif what == "one_term":
        # left out 2^-24, rounded once, and what the small products' sum loses
        assert err[0][1] <= 1.02 * 2.0 ** -23 and err[0][0] <= 1.05 * err[1][0]
    else:
        assert err[0][0] <= err[1][0]
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("what", ["rows", "columns", "products", "subnormal", "zeros"])
def test_matmul_f32_split_mixed_magnitudes(ctx, what):
    """Lines whose large elements meet zeros, so that the small ones, whose lower parts or products leave the normal range, make
    the sums."""
    N, H, C, W = 40, 256, 256, 256
    r = util.rng(79)
    a, b = (r.uniform(1, 2, s) * r.choice([-1.0, 1.0], s[-1]) for s in ((N, H, C), (N, C, W)))
    if what == "rows":
        a, b = a * 2.0 ** -120, b * 2.0 ** 60
    elif what == "columns":
        a, b = a * 2.0 ** 60, b * 2.0 ** -120
    elif what == "products":
        a, b = a * 2.0 ** -62, b * 2.0 ** -60
    elif what == "subnormal":
        a, b = a * 2.0 ** -140, b * 2.0 ** 100
    else:    # disjoint: exact zeros beside tiny values
        a[:, :, ::2] *= 2.0 ** -130
        b[:, ::2], a[:, 5], b[:, :, 7] = 0.0, 0.0, 0.0
        a[:, 9, 1::2] = 0.0
    a, b = a.astype(np.float32), b.astype(np.float32)
    if what != "zeros":
        a[:, :, 0], b[:, 0] = 1.0, 0.0
        a[:, :, 1], b[:, 1] = 0.0, 1.0
    ref = a.astype(np.float64) @ b.astype(np.float64)
    bound = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (N, H, W))
    ctx.matmul(ta, tbb, to)
    st, out = to.download()
    assert st == tb.Status.OK and np.all(np.abs(out - ref) <= C * 2.0 ** -24 * bound + C * 2.0 ** -149)
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("what", ["special", "tiny_lines", "tiny", "overflow"])
def test_matmul_f32_split_range(ctx, what):
    """Operands whose parts leave bf16's or the normal range: same classes and the same accuracy as multiply-adds."""
    N, H, C, W = 40, 256, 320, 256
    r = util.rng(77)
    a, b = r.standard_normal((N, H, C)).astype(np.float32), r.standard_normal((N, C, W)).astype(np.float32)
    if what == "special":
        a[0, 3, 5], a[1, 7, 9], b[2, 10, 11], b[3, 5, 6], a[3, :100] = np.inf, np.nan, -np.inf, np.inf, 0.0
        b[4, 0, 0], a[4, :, 0] = 1e38, 2.0
    elif what == "tiny_lines":
        a[:, 17] *= 2.0 ** -118
        b[:, :, 3] *= 2.0 ** -120
        b[:, :, 9] *= 2.0 ** 50
    elif what == "tiny":
        a *= np.float32(2.0 ** -55)
        b *= np.float32(2.0 ** -60)
    else:
        a *= np.float32(2.0 ** 100)
        b[:, :, ::2] *= np.float32(2.0 ** 60)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (N, H, W))
    ctx.matmul(ta, tbb, to)
    st, out = to.download()
    with np.errstate(all="ignore"):
        ref   = a.astype(np.float64) @ b.astype(np.float64)
        ref32 = ref.astype(np.float32)
        bound = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
        assert st == tb.Status.OK and np.array_equal(np.isnan(out), np.isnan(ref32))
        sure = np.abs(bound) < 2.0 ** 127    # no partial sum can overflow: finite, within K roundings and the subnormal step
        assert np.all(np.abs(out[sure] - ref[sure]) <= C * 2.0 ** -24 * bound[sure] + C * 2.0 ** -149)
        assert what != "overflow" or np.isinf(out[:, :, ::2]).all()    # every product is out of range: the first one's sign stays
        inf = np.isinf(ref)
        assert np.array_equal(out[inf], ref32[inf])
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("case", [(32, 28, 28, 64, 128, 3, [1, 1], [1, 1, 1, 1]), (32, 29, 27, 33, 127, 3, [1, 1], [1, 1, 1, 1]),
                                  (32, 57, 57, 256, 260, 1, [2, 2], [0, 0, 0, 0])])
def test_conv_f32_split(ctx, case):
    N, IH, IW, IC, OC, K, stride, pad = case
    r = util.rng(1010 + IC)
    x, w = r.standard_normal((N, IH, IW, IC)).astype(np.float32), r.standard_normal((OC, K, K, IC)).astype(np.float32)
    b = r.standard_normal(OC).astype(np.float32)
    OH, OW = orc.conv_out_hw(IH, IW, K, K, pad, stride, [1, 1])
    tx, tw, tbias, to = ctx.from_numpy(x), ctx.from_numpy(w), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (N, OH, OW, OC))
    ctx.conv2d(tx, tw, tbias, to, pad, stride, [1, 1], epilogue=tb.Epilogue(None, (-20.0, 30.0)))
    assert ctx.last_kernel() == "conv_f32"
    st, out = to.download()
    xp = np.pad(x.astype(np.float64), ((0, 0), (pad[0], pad[1]), (pad[2], pad[3]), (0, 0)))
    ref, bound = np.zeros((N, OH, OW, OC)) + b, np.zeros((N, OH, OW, OC)) + np.abs(b)
    for ky in range(K):
        for kx in range(K):
            win = xp[:, ky:ky + (OH - 1) * stride[0] + 1:stride[0], kx:kx + (OW - 1) * stride[1] + 1:stride[1]]
            wt = w[:, ky, kx].astype(np.float64).T
            ref, bound = ref + win @ wt, bound + np.abs(win) @ np.abs(wt)
    assert st == tb.Status.OK and np.all(np.abs(out - np.clip(ref, -20.0, 30.0)) <= 2.0 ** -22 * bound)
    for t in (tx, tw, tbias, to):
        t.free()


def test_split_results_computed_again_in_time(ctx):
    """Products whose every result is computed again (too small to split, or a NaN per row): no slower than a few times the
    multiply-adds, and never a time-out, however short the limit of a wait for the pipeline (K = 8192 takes milliseconds)."""
    N, H, C, W = 20, 200, 8192, 260
    r = util.rng(81)
    a, b = (r.standard_normal(s).astype(np.float32) for s in ((N, H, C), (N, C, W)))
    small_a, small_b = a * np.float32(2.0 ** -70), b * np.float32(2.0 ** -60)
    nans = a.copy()
    nans[:, ::32, 4000] = np.nan
    tensors = {k: ctx.from_numpy(v) for k, v in dict(a=a, b=b, small_a=small_a, small_b=small_b, nans=nans).items()}
    to = ctx.empty(tb.DType.FP32, (N, H, W))
    ref = a.astype(np.float64) @ b.astype(np.float64)
    mag = np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    try:
        ctx.set_wait_limit(200000)    # about 0.1 ms; a stage takes some microseconds
        for x, y, scale in (("a", "b", 1.0), ("small_a", "small_b", 2.0 ** -130), ("nans", "b", 1.0)):
            ctx.matmul(tensors[x], tensors[y], to)
            st, out = to.download(check=False)
            assert st == tb.Status.OK, x
            if x == "nans":
                assert np.isnan(out[:, ::32]).all()
                keep = np.ones(H, bool)
                keep[::32] = False
                assert np.all(np.abs(out[:, keep] - ref[:, keep]) <= 2.0 ** -21 * mag[:, keep])
            else:
                assert np.all(np.abs(out - scale * ref) <= C * 2.0 ** -24 * scale * mag + C * 2.0 ** -149)
    finally:
        ctx.set_wait_limit(4000000000)
    for t in list(tensors.values()) + [to]:
        t.free()


@pytest.mark.parametrize("conv", [False, True])
def test_split_bounded_waits_give_up(ctx, conv):
    """A wait limit below the time of any stage: the kernel reports it (the multiply-add kernel has no waits and could not), ends,
    and the same call is right afterwards."""
    r = util.rng(82)
    if conv:
        x, w = r.integers(-3, 4, (32, 28, 28, 64)).astype(np.float32), r.integers(-3, 4, (128, 3, 3, 64)).astype(np.float32)
        xp = np.pad(x, ((0, 0), (1, 1), (1, 1), (0, 0)))
        exp = sum(xp[:, ky:ky + 28, kx:kx + 28] @ w[:, ky, kx].T for ky in range(3) for kx in range(3))
        tensors = [ctx.from_numpy(v) for v in (x, w, np.zeros(128, np.float32))] + [ctx.empty(tb.DType.FP32, exp.shape)]
        call = lambda: ctx.conv2d(*tensors, [1, 1, 1, 1], [1, 1], [1, 1])
    else:
        a, b = (r.integers(-3, 4, s).astype(np.float32) for s in ((40, 256, 320), (40, 320, 256)))
        exp = a @ b
        tensors = [ctx.from_numpy(v) for v in (a, b)] + [ctx.empty(tb.DType.FP32, exp.shape)]
        call = lambda: ctx.matmul(*tensors)
    call()
    ctx.sync()
    ctx.set_wait_limit(1)
    try:
        call()
        assert ctx.sync(check=False) == tb.Status.INTERNAL
    finally:
        ctx.set_wait_limit(4000000000)
    call()
    st, out = tensors[-1].download()
    assert st == tb.Status.OK and np.array_equal(out, exp)
    for t in tensors:
        t.free()


@pytest.mark.parametrize("dil,stride,pad,IC,c0", [(1, [1, 1], [1, 1, 1, 1], 64, 4), (2, [1, 1], [2, 2, 2, 2], 64, 4), (2, [1, 2], [2, 2, 0, 2], 63, 0),
                                                 (1, [1, 1], [0, 0, 0, 0], 61, 4)])
def test_conv_f32_split_views(ctx, dil, stride, pad, IC, c0):
    """A zero-copy view as the input of a layer that runs on the tensor cores, dilation, strides, an infinity and a NaN in it."""
    r = util.rng(1050 + IC)
    full, w = r.standard_normal((36, 31, 33, 68)).astype(np.float32), r.standard_normal((128, 3, 3, IC)).astype(np.float32)
    full[5, 7, 8:10, 9], full[6, 20, 20:22, 20] = np.inf, np.nan
    b = r.standard_normal(128).astype(np.float32)
    x = full[2:, 1:30, 3:32, c0:c0 + IC]
    OH, OW = orc.conv_out_hw(29, 29, 3, 3, pad, stride, [dil, dil])
    tfull, tw, tbias, to = ctx.from_numpy(full), ctx.from_numpy(w), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, (34, OH, OW, 128))
    view = tfull.slice([2, 1, 3, c0], [34, 29, 29, IC])
    call = lambda: ctx.conv2d(view, tw, tbias, to, pad, stride, [dil, dil])
    call()
    assert ctx.last_kernel() == "conv_f32"
    st, out = to.download()
    xp = np.pad(x.astype(np.float64), ((0, 0), (pad[0], pad[1]), (pad[2], pad[3]), (0, 0)))
    ref, bound = np.zeros(out.shape) + b, np.zeros(out.shape) + np.abs(b)
    with np.errstate(all="ignore"):
        for ky in range(3):
            for kx in range(3):
                win = xp[:, ky * dil:ky * dil + (OH - 1) * stride[0] + 1:stride[0], kx * dil:kx * dil + (OW - 1) * stride[1] + 1:stride[1]]
                wt = w[:, ky, kx].astype(np.float64).T
                ref, bound = ref + win @ wt, bound + np.abs(win) @ np.abs(wt)
        assert st == tb.Status.OK and np.array_equal(np.isnan(out), np.isnan(ref)) and np.array_equal(out[np.isinf(ref)], ref[np.isinf(ref)])
        # blocks that hold such results are summed with multiply-adds in K order: K roundings
        near = np.abs(out - ref) <= 9 * IC * 2.0 ** -24 * bound
        assert np.isnan(out).any() and np.isinf(out).any() and near[np.isfinite(ref)].all()
    # that it ran there: the multiply-add kernel has no waits to give up
    ctx.set_wait_limit(1)
    try:
        call()
        assert ctx.sync(check=False) == tb.Status.INTERNAL
    finally:
        ctx.set_wait_limit(4000000000)
    view.free()
    for t in (tfull, tw, tbias, to):
        t.free()


@pytest.mark.parametrize("case", [(2, 9, 11, 8, 5), (2, 9, 11, 7, 6), (1, 20, 20, 300, 40), (32, 28, 28, 64, 128), (32, 28, 27, 33, 127)])
def test_conv_f32_nonfinite_weights_under_padding(ctx, case):
    """Infinite and NaN weights of a padded layer, from the first call on (no verdict is known to the host yet) and through an
    upload under a captured graph: they reach only the pixels whose windows hold them.  The last two run on the tensor
    cores, the third splits K over a cluster."""
    N, IH, IW, IC, OC = case
    r = util.rng(1030 + IC)
    x, w = r.standard_normal((N, IH, IW, IC)).astype(np.float32), r.standard_normal((OC, 3, 3, IC)).astype(np.float32)
    b = r.standard_normal(OC).astype(np.float32)
    finite = w.copy()
    w[0, 0, 0, 1], w[2, 2, 1, 0], w[OC - 1, 1, 2, IC - 1] = np.inf, np.nan, -np.inf
    x[0, 4, 5, 2] = np.inf
    args = ([1] * 4, [1, 1], [1, 1])
    ref, bnd = (orc.conv2d(x, w, b, *args, mode="f64", bounds=f, nthreads=8) for f in (False, True))
    ksb = orc.dot_product_ksb(9 * IC + 1, "fp32", "fp32")
    tx, tbias, to = ctx.from_numpy(x), ctx.from_numpy(b), ctx.empty(tb.DType.FP32, ref.shape)

    def check():
        st, out = to.download()
        assert st == tb.Status.OK
        assert np.array_equal(np.isnan(out), np.isnan(ref)) and np.array_equal(np.isinf(out), np.isinf(ref))
        fin = np.isfinite(ref)
        assert fin[..., [0, 2, OC - 1]].any()
        ok, info = orc.verify_dot_product(out[fin], ref[fin], bnd[fin], ksb, out="fp32")
        assert ok, info

    tw = ctx.from_numpy(w)
    ctx.conv2d(tx, tw, tbias, to, *args)
    assert ctx.last_kernel() == "conv_f32"
    check()
    tw2 = ctx.from_numpy(finite)
    ctx.conv2d(tx, tw2, tbias, to, *args)
    ctx.capture_begin()
    ctx.conv2d(tx, tw2, tbias, to, *args)
    graph = ctx.capture_end()
    tw2.upload(w)
    ctx.graph_launch(graph)
    check()
    ctx.graph_destroy(graph)
    for t in (tx, tw, tw2, tbias, to):
        t.free()


def test_split_more_tiles_than_slots(ctx):
    """More tiles per CTA (129 on 148 SMs) than there are words for blocks to be computed again: tiles that share a word."""
    torch = pytest.importorskip("torch")
    N, late = 148 * 129, 5 + 148 * 128
    gen = torch.Generator(device="cuda").manual_seed(83)
    a, b = (torch.randn(N, *s, generator=gen, device="cuda") for s in ((128, 256), (256, 128)))
    a[5, 3, 7], a[late, 70, 0], a[late + 1, 9] = float("nan"), float("inf"), 1e-30
    b[late + 1] *= 1e-8
    out = torch.empty((N, 128, 128), device="cuda")
    torch.cuda.synchronize()
    ta, tbb, to = (ctx.wrap(tb.DType.FP32, tuple(v.shape), v.data_ptr(), v) for v in (a, b, out))
    ctx.matmul(ta, tbb, to)
    ctx.sync()
    for n in (0, 5, 6, late - 148, late, late + 1, N - 1):
        x, y = a[n].double(), b[n].double()
        ref, bound, got = x @ y, x.abs() @ y.abs(), out[n].double()
        fin = torch.isfinite(ref)
        assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
        assert bool(((got - ref).abs() <= 256 * 2.0 ** -24 * bound + 256 * 2.0 ** -149)[fin].all())
        assert bool(fin.all()) == (n not in (5, late))
    for t in (ta, tbb, to):
        t.free()
