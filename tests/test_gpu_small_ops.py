"""MATMUL with up to four rows (matmul_rows.cu) and AVG_POOL2D whose windows are shared between threads, at the sizes where they
can go wrong, against the oracle."""
import numpy as np
import pytest

import reference_model_b200 as tb
from oracle import oracle as orc
from tests import util

pytestmark = pytest.mark.gpu

F16, BF16, F32 = tb.DType.FP16, tb.DType.BF16, tb.DType.FP32


@pytest.fixture(scope="module")
def ctx():
    c = tb.Context(0)
    yield c
    c.close()


# N, H, C, W: one cluster of eight, K of a rank that ends early, last columns of a block, several batches, no cluster
SHAPES = [(1, 1, 2048, 1000), (3, 2, 260, 4), (2, 4, 1028, 132), (70, 3, 256, 260), (1, 1, 4096, 1024), (1, 4, 300, 516), (5, 1, 2052, 128)]


@pytest.mark.parametrize("zp", [(0, 0), (-128, 127), (3, 0), (0, -2)])
@pytest.mark.parametrize("shape", SHAPES)
def test_matmul_rows_i8(ctx, shape, zp):
    N, H, C, W = shape
    r = util.rng(3000 + W + H)
    a, b = r.integers(-128, 128, size=(N, H, C)).astype(np.int8), r.integers(-128, 128, size=(N, C, W)).astype(np.int8)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.INT32, (N, H, W))
    ctx.matmul(ta, tbb, to, *zp)
    assert ctx.last_kernel() == "matmul_rows_i8"
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out, orc.matmul(a, b, *zp, nthreads=8))
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("name", ["fp16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_matmul_rows_float(ctx, name, shape):
    N, H, C, W = shape
    r = util.rng(3100 + W + H)
    a, b = (orc.fptrunc(r.standard_normal(s).astype(np.float32), name) for s in ((N, H, C), (N, C, W)))
    dt = F16 if name == "fp16" else BF16
    up = lambda v: ctx.from_numpy(v.astype(np.float16)) if dt == F16 else ctx.from_numpy(util.to_bf16_bits(v), BF16)
    ta, tbb = up(a), up(b)
    ref, bnd = orc.matmul(a, b, mode="f64"), orc.matmul(np.abs(a), np.abs(b), mode="f64")
    for odt, oname in ((dt, name), (F32, "fp32")):
        to = ctx.empty(odt, (N, H, W))
        ctx.matmul(ta, tbb, to)
        assert ctx.last_kernel() == "matmul_rows_f16"
        st, out = to.download()
        out = util.from_bf16_bits(out) if odt == BF16 else out.astype(np.float32)
        ok, info = orc.verify_dot_product(out, ref, bnd, orc.dot_product_ksb(C, "fp32", oname), out=oname)
        assert st == tb.Status.OK and ok, info
        to.free()
    ta.free(), tbb.free()


def test_matmul_rows_keeps_infinities_apart(ctx):
    """An infinite element or a NaN meets only what the product pairs it with, also where K ends inside a block's share."""
    a, b = np.ones((1, 2, 260), np.float16), np.ones((1, 260, 8), np.float16)
    a[0, 1, 259], b[0, 100, 3], b[0, 7, 5] = np.inf, -np.inf, np.nan
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(F32, (1, 2, 8))
    ctx.matmul(ta, tbb, to)
    assert ctx.last_kernel() == "matmul_rows_f16"
    st, out = to.download()
    with np.errstate(invalid="ignore"):
        exp = a[0].astype(np.float32) @ b[0].astype(np.float32)
    assert np.array_equal(out[0], exp, equal_nan=True)
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("case", [((1, 7, 7, 2048), [7, 7], [0] * 4, [1, 1]), ((3, 9, 8, 36), [5, 4], [2, 2, 1, 1], [2, 1]),
                                  ((2, 20, 17, 4), [16, 9], [3, 3, 4, 4], [2, 2]), ((1, 33, 33, 8), [33, 33], [0] * 4, [1, 1])])
def test_avg_pool_shared_windows(ctx, case):
    shape, kernel, pad, stride = case
    x = util.rng(3200 + shape[3]).integers(-128, 128, size=shape).astype(np.int8)
    st, exp = orc.avg_pool2d(x, kernel, pad, stride, -7, 11)
    assert st == orc.VALID
    tx, to = ctx.from_numpy(x), ctx.empty(tb.DType.INT8, exp.shape)
    ctx.avg_pool2d(tx, to, kernel, pad, stride, -7, 11)
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
    tx.free(), to.free()


@pytest.mark.parametrize("case", [
    # N, H, W, IC, OC, KH, KW, stride, pad, in_zp, shift
    (1, 224, 224, 3, 64, 7, 7, 2, (3, 2, 3, 2), -128, 33),      # two pixels of a row side by side
    (3, 113, 116, 3, 64, 3, 3, 2, (0, 0, 0, 1), 5, 33),         # windows up to the last byte of a row
    (5, 131, 132, 3, 32, 3, 3, 2, (1, 1, 1, 0), -128, 33),      # four
    (2, 77, 72, 4, 32, 5, 5, 1, (2, 2, 2, 2), 0, 33),
    (1, 96, 100, 1, 32, 3, 2, 1, (1, 1, 1, 0), 17, 33),
    (3, 90, 512, 2, 64, 2, 12, 4, (0, 0, 4, 4), -128, 33),
    (2, 128, 129, 3, 64, 7, 7, 2, (3, 2, 3, 3), 9, 33),         # an odd number of columns: another form
    (1, 224, 224, 3, 64, 7, 7, 2, (3, 2, 3, 2), -128, 20),      # records that are not usable: another form
])
def test_few_channels_side_by_side(ctx, case):
    N, H, W, IC, OC, KH, KW, s, pad, izp, sh = case
    r = util.rng(3100 + W + OC + sh)
    x, w, b = util.conv_int8_case(r, N, H, W, IC, OC, KH, KW, bias_range=1 << 12)
    mult, shift = util.rescale_params(r, OC)
    shift = np.maximum(shift, 33).astype(np.int8) if sh >= 33 else np.full(OC, sh, np.int8)
    if sh < 33:
        mult = (mult >> 12).astype(np.int32)
    acc = orc.conv2d(x, w, b, list(pad), [s, s], [1, 1], izp, 0, nthreads=orc.num_procs())
    est, q = orc.rescale(acc, mult, shift, True, True, "SINGLE_ROUND", 0, -3, 32, 8)
    exp = np.clip(q, -120, 119)
    ts = [ctx.from_numpy(v) for v in (x, w, b, mult, shift)]
    to = ctx.empty(tb.DType.INT8, exp.shape)
    epi = tb.Epilogue(tb.RescaleAttr(ts[3], ts[4], 0, -3, True, "SINGLE_ROUND", per_channel=True), (-120, 119))
    for _ in range(2):
        to.upload(np.full(exp.shape, 55, np.int8))
        ctx.conv2d(ts[0], ts[1], ts[2], to, list(pad), [s, s], [1, 1], izp, 0, epi)
        st, out = to.download()
        assert (st == tb.Status.OK) == (est == orc.VALID)
        assert est != orc.VALID or np.array_equal(out.astype(np.int32), exp)
    for t in ts + [to]:
        t.free()


@pytest.mark.parametrize("H", [1, 4])
@pytest.mark.parametrize("name", ["fp16", "bf16"])
def test_matmul_rows_long_sums(ctx, name, H):
    """K = 4000 in one block per column (as many batches as fill the SMs).  Sums of 16 products, 31 of those per warp, eight
    warps: with unit roundoff u the rounding errors' root mean square is u / sqrt(3) * sqrt((248 * 136 + 8 * 496 * 16 + 36 *
    500) / 4000) = 1.85e-7 of the result's, less for mantissas above one; a running sum over 500 gives 5.5e-7 by the same rule,
    sums of 64 by the tensor core 1.8e-7."""
    N, C, W = 160, 4000, 100
    r = util.rng(3400 + H)
    a, b = (orc.fptrunc(r.standard_normal(s).astype(np.float32), name) for s in ((N, H, C), (N, C, W)))
    up = lambda v: ctx.from_numpy(v.astype(np.float16)) if name == "fp16" else ctx.from_numpy(util.to_bf16_bits(v), BF16)
    ta, tbb, to = up(a), up(b), ctx.empty(F32, (N, H, W))
    ctx.matmul(ta, tbb, to)
    assert ctx.last_kernel() == "matmul_rows_f16"
    st, out = to.download()
    ref = np.matmul(a.astype(np.float64), b.astype(np.float64))
    err = np.sqrt(np.mean((out - ref) ** 2) / np.mean(ref ** 2))
    assert st == tb.Status.OK and err < 1.85e-7, err
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("captured", [False, True])
def test_matmul_rows_read_what_the_launch_before_wrote(ctx, captured):
    """A chain of products with permutations, each launch overlapping the tail of the one whose result it reads (as B in the
    last one): exact for every input."""
    r, C, steps = util.rng(3500), 512, 24
    ps = [r.permutation(C) for _ in range(4)]
    ms = []
    for p in ps:
        m = np.zeros((1, C, C), np.float16)
        m[0, p, np.arange(C)] = 1.0
        ms.append(ctx.from_numpy(m))
    xs, last = [ctx.empty(F16, (1, 4, C)) for _ in range(2)], ctx.empty(F32, (1, 1, 4))
    one = ctx.from_numpy(np.ones((1, 1, C), np.float16))

    def chain():
        for i in range(steps):
            ctx.matmul(xs[i % 2], ms[i % 4], xs[1 - i % 2])
            assert ctx.last_kernel() == "matmul_rows_f16"
        ctx.matmul(one, column, last)

    column = xs[steps % 2].reshape([1, C, 4])
    chain()
    if captured:
        ctx.capture_begin()
        chain()
        g = ctx.capture_end()
    for k in range(8):
        x = r.integers(-8, 8, size=(1, 4, C)).astype(np.float16)
        xs[0].upload(x)
        ctx.graph_launch(g) if captured else chain()
        exp = x
        for i in range(steps):
            exp = exp[:, :, ps[i % 4]]
        assert np.array_equal(xs[steps % 2].download()[1], exp)
        assert np.array_equal(last.download()[1][0, 0], exp.reshape(C, 4).astype(np.float32).sum(0))
    if captured:
        ctx.graph_destroy(g)
    column.free()
    for t in ms + xs + [one, last]:
        t.free()


@pytest.mark.parametrize("shape", [(1, 1, 8196, 132), (2, 2, 4100, 12), (1, 3, 1540, 260), (1, 4, 2052, 64), (300, 4, 256, 128)])
def test_matmul_rows_sums_of_a(ctx, shape):
    """B's zero point alone: the sums of A's rows, shared out among warps, with words behind the ones that are asked for first."""
    N, H, C, W = shape
    r = util.rng(3600 + C)
    a, b = r.integers(-128, 128, size=(N, H, C)).astype(np.int8), r.integers(-128, 128, size=(N, C, W)).astype(np.int8)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.INT32, (N, H, W))
    ctx.matmul(ta, tbb, to, 0, 77)
    assert ctx.last_kernel() == "matmul_rows_i8"
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out, orc.matmul(a, b, 0, 77, nthreads=8))
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("shape,kernel,stride,form", [
    ((63, 26, 26, 84), [4, 4], [2, 2], "avg_pool2d"),                       # 190 512 words of outputs
    ((37, 9, 9, 164), [5, 5], [2, 2], "avg_pool2d, taps shared"),           # 13 653
    ((40, 7, 7, 2048), [7, 7], [1, 1], "avg_pool2d, taps shared"),          # a classifier's pool
    ((80, 7, 7, 2048), [7, 7], [1, 1], "avg_pool2d"),
])
def test_avg_pool_shares_taps_where_outputs_are_few(ctx, shape, kernel, stride, form):
    x = util.rng(3700 + shape[3]).integers(-128, 128, size=shape).astype(np.int8)
    st, exp = orc.avg_pool2d(x, kernel, [0] * 4, stride, -7, 11)
    assert st == orc.VALID
    tx, to = ctx.from_numpy(x), ctx.empty(tb.DType.INT8, exp.shape)
    ctx.avg_pool2d(tx, to, kernel, [0] * 4, stride, -7, 11)
    assert ctx.last_form() == form
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out.astype(np.int32), exp)
    tx.free(), to.free()
