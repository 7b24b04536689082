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
