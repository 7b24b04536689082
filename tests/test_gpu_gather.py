"""The gathering tensor-core kernel at the edges of its tiles: runs, rows and columns of every alignment, K shorter than a
chunk and split over a cluster, one row, borders, views, strides, dilation, both zero points, every element type and pair of
fp8 types, outputs that are no whole 16-byte rows, constants that change; integers bit for bit against the oracle, floats
under the DOT_PRODUCT rule and against the kernel that rounds every multiply-add."""
import threading

import numpy as np
import pytest

import reference_model_b200 as tb
from oracle import oracle as orc
from tests import util
from tests.test_gpu_parity import _fp8_codes, oracle_conv_i8, run_conv_fp, run_conv_i8

pytestmark = pytest.mark.gpu
F16, BF16, F32 = tb.DType.FP16, tb.DType.BF16, tb.DType.FP32


@pytest.fixture(scope="module")
def ctx():
    c = tb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 129, 17, 33), (3, 128, 100, 257), (1, 5, 3000, 300), (4, 250, 36, 40), (1, 33, 130, 515),
                                   (1, 1, 65, 1), (2, 129, 81, 33), (4, 250, 100, 40), (40, 129, 60, 33)])
@pytest.mark.parametrize("zp", [(0, 0), (3, 0), (0, -2), (-128, 127)])
def test_matmul_i8(ctx, shape, zp):
    N, H, C, W = shape
    r = util.rng(2000 + H + W)
    a, b = r.integers(-128, 128, size=(N, H, C)).astype(np.int8), r.integers(-128, 128, size=(N, C, W)).astype(np.int8)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.INT32, (N, H, W))
    ctx.matmul(ta, tbb, to, *zp)
    tiny = C <= 64 and N * H * C * W <= 1 << 23    # one thread per output
    assert ctx.last_kernel() == ("matmul_direct" if tiny else "tc_gemm_any_i8_i32")
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out, orc.matmul(a, b, *zp, nthreads=8))
    for t in (ta, tbb, to):
        t.free()


@pytest.mark.parametrize("name", ["fp16", "bf16", "e4m3"])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (3, 130, 26, 31), (2, 197, 64, 197), (1, 7, 2679, 72), (2, 60, 77, 300),
                                   (1, 1, 65, 1), (3, 130, 90, 31), (5, 197, 64, 197)])
def test_matmul_float(ctx, name, shape):
    N, H, C, W = shape
    r = util.rng(2100 + H + W)
    if name == "e4m3":
        ca, cb = _fp8_codes(r, (N, H, C), name), _fp8_codes(r, (N, C, W), name)
        a, b = orc.fp8_to_f32(ca, name), orc.fp8_to_f32(cb, name)
        ta, tbb, outs = ctx.from_numpy(ca, tb.DType.FP8E4M3), ctx.from_numpy(cb, tb.DType.FP8E4M3), ((F16, "fp16"), (F32, "fp32"))
    else:
        a, b = (orc.fptrunc(r.standard_normal(s).astype(np.float32), name) for s in ((N, H, C), (N, C, W)))
        dt = F16 if name == "fp16" else BF16
        ta, tbb = (ctx.from_numpy(v.astype(np.float16)) if dt == F16 else ctx.from_numpy(util.to_bf16_bits(v), BF16) for v in (a, b))
        outs = ((dt, name), (F32, "fp32"))
    ref, bnd = orc.matmul(a, b, mode="f64"), orc.matmul(np.abs(a), np.abs(b), mode="f64")
    for dt, oname in outs:
        to = ctx.empty(dt, (N, H, W))
        ctx.matmul(ta, tbb, to)
        tiny = C <= 64 and N * H * C * W <= 1 << 23
        assert ctx.last_kernel().startswith("matmul_direct" if tiny else "tc_gemm_any"), ctx.last_kernel()
        st, out = to.download()
        out = util.from_bf16_bits(out) if dt == BF16 else out.astype(np.float32)
        ok, info = orc.verify_dot_product(out, ref, bnd, orc.dot_product_ksb(C, "fp32", oname), out=oname)
        assert st == tb.Status.OK and ok, info
        to.free()
    ta.free(), tbb.free()


@pytest.mark.parametrize("name", ["fp16", "bf16", "e4m3", "e5m2"])
@pytest.mark.parametrize("shape", [(8, 200, 65, 203), (8, 200, 81, 200), (8, 130, 100, 99), (2, 130, 300, 33), (1, 257, 1003, 203), (4, 100, 1160, 61), (2, 60, 4001, 300), (1, 33, 6007, 40)])
def test_matmul_fp32_output_sums(ctx, name, shape):
    """fp32 results of operands of one sign, where a running sum that is cut off at every step drifts: no further from the
    64-bit product than the kernel that rounds every multiply-add."""
    N, H, C, W = shape
    r = util.rng(2600 + C)
    if name[0] == "e":
        ca, cb = (r.integers(0x28, 0x40, size=s).astype(np.uint8) for s in ((N, H, C), (N, C, W)))
        a, b = orc.fp8_to_f32(ca, name), orc.fp8_to_f32(cb, name)
        dt = tb.DType.FP8E4M3 if name == "e4m3" else tb.DType.FP8E5M2
        ta, tbb = ctx.from_numpy(ca, dt), ctx.from_numpy(cb, dt)
    else:
        a, b = (orc.fptrunc(r.uniform(0.5, 1.0, size=s).astype(np.float32), name) for s in ((N, H, C), (N, C, W)))
        ta, tbb = (ctx.from_numpy(v.astype(np.float16)) if name == "fp16" else ctx.from_numpy(util.to_bf16_bits(v), BF16) for v in (a, b))
    ref, err, to = a.astype(np.float64) @ b.astype(np.float64), [], ctx.empty(F32, (N, H, W))
    for policy in (0, 1):
        old = ctx.set_kernel_policy(policy)
        ctx.matmul(ta, tbb, to)
        assert ctx.last_kernel().startswith("matmul_direct" if policy else "tc_gemm_any"), ctx.last_kernel()
        ctx.set_kernel_policy(old)
        st, out = to.download()
        assert st == tb.Status.OK
        err.append(np.linalg.norm(out - ref) / np.linalg.norm(ref))
    print(name, shape, err)
    assert err[0] <= err[1]
    for t in (ta, tbb, to):
        t.free()


# N, IH, IW, IC, OC, K, stride, pad, in_zp
CONV = [(1, 32, 32, 8, 16, 1, 1, 0, 5), (2, 13, 11, 24, 40, 3, 1, 1, -128), (1, 9, 10, 13, 7, 3, 1, 1, 3), (3, 7, 7, 20, 300, 1, 1, 0, -128),
        (1, 15, 15, 50, 33, 5, 2, 2, 9), (1, 3, 3, 200, 65, 3, 1, 1, -128), (2, 5, 130, 12, 31, 3, 1, 1, 0), (1, 4, 4, 500, 24, 3, 1, 1, 7),
        (9, 32, 32, 8, 16, 1, 1, 0, 5), (4, 7, 7, 20, 300, 1, 1, 0, -128)]


@pytest.mark.parametrize("case", CONV)
def test_conv_i8(ctx, case):
    N, IH, IW, IC, OC, K, s, p, izp = case
    r = util.rng(2200 + IC + OC)
    x, w, b = util.conv_int8_case(r, N, IH, IW, IC, OC, K, K, bias_range=1 << 16)
    args = ([p] * 4, [s, s], [1, 1], izp, 0)
    _, exp = oracle_conv_i8(x, w, b, *args)
    st, out, kernel = run_conv_i8(ctx, x, w, b, *args)
    tiny = K * K * IC <= 64 and exp.size * K * K * IC <= 1 << 20    # one thread per output
    assert kernel == ("conv2d_direct" if tiny else "tc_gemm_any_i8_i32") and st == tb.Status.OK and np.array_equal(out, exp), kernel
    mult, shift = util.rescale_params(r, OC)
    for rounding, clamp in (("DOUBLE_ROUND", (-128, 127)), ("SINGLE_ROUND", (-90, 100))):
        resc = (mult, shift, -3, rounding)
        est, exp = oracle_conv_i8(x, w, b, *args, rescale=resc, clamp=clamp)
        assert est == orc.VALID
        for cache in (True, False):    # with proven records and with the general arithmetic
            st, out, kernel = run_conv_i8(ctx, x, w, b, *args, rescale=resc, clamp=clamp, cache=cache)
            assert kernel == ("conv2d_direct" if tiny else "tc_gemm_any_i8_rescale") and st == tb.Status.OK and np.array_equal(out, exp), (rounding, cache)


def test_conv_i8_constants_replaced(ctx):
    """RESCALE operands replaced by uploads, eagerly and under a captured graph: from provable records to ones that need the
    general arithmetic and its range check, and back."""
    r = util.rng(2280)
    x, w, b = util.conv_int8_case(r, 2, 21, 19, 24, 40, 3, 3, bias_range=1 << 10)
    args = ([1] * 4, [1, 1], [1, 1], 3, 0)
    acc = orc.conv2d(x, w, b, *args, nthreads=8)
    top = int(np.abs(acc).max())
    bits = top.bit_length()              # every accumulator fits these bits, which the worst case of the layer does not
    good, tight, low = (util.rescale_params(r, 40), (np.full(40, 1 << 20, np.int32), np.full(40, bits + 1, np.int8)),
                        (np.full(40, 1 << 20, np.int32), np.full(40, bits - 1, np.int8)))
    assert (1 << bits) < 24 * 9 * 255 * 128 and top >= 1 << (bits - 2)    # (low: some accumulator is out of the accepted range)
    tx, tw, tbias, tm, ts = (ctx.from_numpy(v) for v in (x, w, b, *good))
    to = ctx.empty(tb.DType.INT8, acc.shape)
    epi = tb.Epilogue(tb.RescaleAttr(tm, ts, 0, 7, True, "DOUBLE_ROUND", per_channel=True), (-100, 120))
    call = lambda: ctx.conv2d(tx, tw, tbias, to, *args, epi)

    def check(run):
        for mult, shift in (good, tight, good, low):
            tm.upload(mult), ts.upload(shift)
            run()
            st, out = to.download(check=False)
            est, exp = orc.rescale(acc, mult, shift, True, True, "DOUBLE_ROUND", 0, 7, 32, 8)
            if shift is low[1]:
                assert est != orc.VALID and st == tb.Status.UNPREDICTABLE
            else:
                assert est == orc.VALID and st == tb.Status.OK and np.array_equal(out, np.clip(exp, -100, 120))

    check(call)
    assert ctx.last_kernel() == "tc_gemm_any_i8_rescale"
    tm.upload(good[0]), ts.upload(good[1])
    call()
    ctx.capture_begin()
    call()
    graph = ctx.capture_end()
    check(lambda: ctx.graph_launch(graph))
    ctx.graph_destroy(graph)
    for t in (tx, tw, tbias, tm, ts, to):
        t.free()


@pytest.mark.parametrize("dt,name", [(F16, "fp16"), (BF16, "bf16")])
@pytest.mark.parametrize("case", [(2, 9, 11, 12, 20, 3, 1), (1, 14, 14, 9, 33, 3, 1), (2, 6, 6, 100, 70, 1, 0), (1, 20, 7, 3, 8, 5, 2)])
def test_conv_float(ctx, dt, name, case):
    N, IH, IW, IC, OC, K, p = case
    r = util.rng(2300 + IC)
    x, w, b = (orc.fptrunc(r.standard_normal(s).astype(np.float32), name) for s in ((N, IH, IW, IC), (OC, K, K, IC), (OC,)))
    args = ([p] * 4, [1, 1], [1, 1])
    ref, bnd = (orc.conv2d(x, w, b, *args, mode="f64", bounds=f) for f in (False, True))
    st, out, kernel = run_conv_fp(ctx, x, w, b, *args, dt)
    ok, info = orc.verify_dot_product(out, ref, bnd, orc.dot_product_ksb(K * K * IC + 1, "fp32", name), out=name)
    assert kernel == "tc_gemm_any_f16" and st == tb.Status.OK and ok, (kernel, info)


# parent [N, IH, IW, bytes of channels], view start and size (channels in elements), OC, KH, KW, stride, dilation, pad; what the
# run and the pitches are multiples of: 16 bytes, 8, 4, less
VIEWS = [((2, 13, 15, 64), (0, 1, 2), (2, 11, 12), 16, 48, 20, 3, 2, [1, 1], [2, 1], [2, 2, 1, 0]),
         ((1, 19, 32, 48), (0, 0, 16), (1, 18, 15), 16, 24, 33, 2, 3, [1, 3], [1, 2], [0, 1, 2, 3]),
         ((3, 10, 24, 44), (1, 0, 8), (2, 9, 16), 0, 20, 65, 3, 3, [3, 1], [1, 3], [1, 2, 3, 3]),
         ((2, 12, 32, 46), (0, 2, 16), (2, 9, 16), 0, 22, 30, 2, 5, [2, 1], [1, 3], [1, 0, 5, 4])]


@pytest.mark.parametrize("name", ["i8", "i8 rescale", "fp16", "bf16", "e4m3", "e5m2"])
@pytest.mark.parametrize("case", range(len(VIEWS)))
def test_conv_views(ctx, name, case):
    """A zero-copy view as the input (pitches beyond the run), unequal strides, dilation and padding, every element type."""
    (N0, H0, W0, cb), (n, y, x0), (N, IH, IW), cstart, run, OC, KH, KW, stride, dil, pad = VIEWS[case]
    es = 2 if name in ("fp16", "bf16") else 1
    C0, c0, IC = cb // es, cstart // es, run // es
    r = util.rng(2900 + case)
    oname = "bf16" if name == "bf16" else "fp16"
    up = lambda v: ctx.from_numpy(util.to_bf16_bits(v), BF16) if name == "bf16" else ctx.from_numpy(v.astype(np.float16))
    shapes, izp = ((N0, H0, W0, C0), (OC, KH, KW, IC)), 0
    if name[0] == "i":
        izp = -7
        full, w = (r.integers(-128, 128, sh).astype(np.int8) for sh in shapes)
        b = r.integers(-1000, 1000, OC).astype(np.int32)
        tfull, tw, tbias = (ctx.from_numpy(v) for v in (full, w, b))
    elif name[0] == "e":
        cf, cw = (_fp8_codes(r, sh, name) for sh in shapes)
        full, w, b = orc.fp8_to_f32(cf, name), orc.fp8_to_f32(cw, name), r.standard_normal(OC).astype(np.float16).astype(np.float32)
        dt = tb.DType.FP8E4M3 if name == "e4m3" else tb.DType.FP8E5M2
        tfull, tw, tbias = ctx.from_numpy(cf, dt), ctx.from_numpy(cw, dt), up(b)
    else:
        full, w, b = (orc.fptrunc(r.standard_normal(sh).astype(np.float32), name) for sh in shapes + ((OC,),))
        tfull, tw, tbias = up(full), up(w), up(b)
    view = tfull.slice([n, y, x0, c0], [N, IH, IW, IC])
    x = np.ascontiguousarray(full[n:n + N, y:y + IH, x0:x0 + IW, c0:c0 + IC])
    args, extra, epi = (pad, stride, dil), [], None
    if name[0] == "i":
        exp = orc.conv2d(x, w, b, *args, izp, 0, nthreads=8)
        odt = tb.DType.INT32
        if name == "i8 rescale":
            mult, shift = util.rescale_params(r, OC)
            extra, odt = [ctx.from_numpy(mult), ctx.from_numpy(shift)], tb.DType.INT8
            epi = tb.Epilogue(tb.RescaleAttr(*extra, 0, 3, True, "DOUBLE_ROUND", per_channel=True), (-120, 110))
            exp = np.clip(orc.rescale(exp, mult, shift, True, True, "DOUBLE_ROUND", 0, 3, 32, 8)[1], -120, 110)
    else:
        exp, bnd = (orc.conv2d(x, w, b, *args, mode="f64", bounds=f) for f in (False, True))
        odt = BF16 if name == "bf16" else F16
    to = ctx.empty(odt, exp.shape)
    ctx.conv2d(view, tw, tbias, to, *args, izp, 0, epi)
    assert ctx.last_kernel().startswith("tc_gemm_any"), ctx.last_kernel()
    st, out = to.download()
    assert st == tb.Status.OK
    if name[0] == "i":
        assert np.array_equal(out, exp)
    else:
        out = util.from_bf16_bits(out) if name == "bf16" else out.astype(np.float32)
        ok, info = orc.verify_dot_product(out, exp, bnd, orc.dot_product_ksb(KH * KW * IC + 1, "fp32", oname), out=oname)
        assert ok, info
    view.free()
    for t in [tfull, tw, tbias, to] + extra:
        t.free()


@pytest.mark.parametrize("fa,fb", [("e4m3", "e5m2"), ("e5m2", "e4m3"), ("e5m2", "e5m2")])
@pytest.mark.parametrize("shape", [(3, 130, 90, 31), (2, 60, 177, 300), (1, 7, 2679, 72)])
def test_matmul_fp8_pairs(ctx, fa, fb, shape):
    N, H, C, W = shape
    r = util.rng(2950 + C)
    ca, cb = _fp8_codes(r, (N, H, C), fa), _fp8_codes(r, (N, C, W), fb)
    a, b = orc.fp8_to_f32(ca, fa), orc.fp8_to_f32(cb, fb)
    ref, bnd = orc.matmul(a, b, mode="f64"), orc.matmul(np.abs(a), np.abs(b), mode="f64")
    dts = {"e4m3": tb.DType.FP8E4M3, "e5m2": tb.DType.FP8E5M2}
    ta, tbb = ctx.from_numpy(ca, dts[fa]), ctx.from_numpy(cb, dts[fb])
    for dt, oname in ((F16, "fp16"), (F32, "fp32")):
        to = ctx.empty(dt, (N, H, W))
        ctx.matmul(ta, tbb, to)
        assert ctx.last_kernel() == "tc_gemm_any_f8"
        st, out = to.download()
        ok, info = orc.verify_dot_product(out.astype(np.float32), ref, bnd, orc.dot_product_ksb(C, "fp32", oname), out=oname)
        assert st == tb.Status.OK and ok, info
        to.free()
    ta.free(), tbb.free()


@pytest.mark.parametrize("name", ["fp16", "bf16", "e5m2"])
@pytest.mark.parametrize("case", [(2, 9, 11, 12, 20, 1, 1, 1), (1, 12, 9, 9, 70, 2, 1, 2), (1, 5, 6, 200, 33, 1, 2, 2)])
def test_conv_nonfinite_weights_under_padding(ctx, name, case):
    """A tap outside the image is skipped, whatever its weight: infinities and NaNs reach only the pixels whose windows hold
    them.  (The last case splits K over a cluster.)"""
    N, IH, IW, IC, OC, s, d, p = case
    r = util.rng(2350 + IC)
    shapes = (N, IH, IW, IC), (OC, 3, 3, IC)
    if name == "e5m2":
        cx, cw = (_fp8_codes(r, sh, name) for sh in shapes)
        cw[0, 0, 0, 1], cw[2, 2, 1, 0], cw[OC - 1, 1, 2, IC - 1] = 0x7C, 0x7F, 0xFC    # infinity, NaN, -infinity
        x, w = orc.fp8_to_f32(cx, name), orc.fp8_to_f32(cw, name)
    else:
        x, w = (orc.fptrunc(r.standard_normal(sh).astype(np.float32), name) for sh in shapes)
        w[0, 0, 0, 1], w[2, 2, 1, 0], w[OC - 1, 1, 2, IC - 1] = np.inf, np.nan, -np.inf
    b = orc.fptrunc(r.standard_normal(OC).astype(np.float32), "bf16" if name == "bf16" else "fp16")
    pad = [p, p - 1 if (IH + 2 * p - 1 - 2 * d) % s else p, p, p - 1 if (IW + 2 * p - 1 - 2 * d) % s else p]
    args = (pad, [s, s], [d, d])
    ref, bnd = (orc.conv2d(x, w, b, *args, mode="f64", bounds=f) for f in (False, True))
    if name == "e5m2":
        dt, odt = tb.DType.FP8E5M2, F16
        tx, tw, tbias, to = ctx.from_numpy(cx, dt), ctx.from_numpy(cw, dt), ctx.from_numpy(b.astype(np.float16)), ctx.empty(odt, ref.shape)
        ctx.conv2d(tx, tw, tbias, to, *args)
        kernel = ctx.last_kernel()
        st, out = to.download()
        out = out.astype(np.float32)
        for t in (tx, tw, tbias, to):
            t.free()
    else:
        st, out, kernel = run_conv_fp(ctx, x, w, b, *args, F16 if name == "fp16" else BF16)
    assert kernel.startswith("tc_gemm_any") and st == tb.Status.OK
    assert np.array_equal(np.isnan(out), np.isnan(ref)) and np.array_equal(np.isinf(out), np.isinf(ref))
    assert np.isnan(out).any() and np.isfinite(out[..., [0, 2, OC - 1]]).any()
    fin = np.isfinite(ref)
    oname = "bf16" if name == "bf16" else "fp16"
    ok, info = orc.verify_dot_product(out[fin], ref[fin], bnd[fin], orc.dot_product_ksb(9 * IC + 1, "fp32", oname), out=oname)
    assert ok, info


def test_bounded_waits_give_up(ctx):
    """A wait limit far below the time the first copies take: the kernel reports, frees what it holds, and the same call is
    exact afterwards (a call that finishes in time is fine as well)."""
    r = util.rng(2400)
    a, b = r.integers(-128, 128, size=(4, 300, 1001)).astype(np.int8), r.integers(-128, 128, size=(4, 1001, 300)).astype(np.int8)
    ta, tbb, to = ctx.from_numpy(a), ctx.from_numpy(b), ctx.empty(tb.DType.INT32, (4, 300, 300))
    exp = orc.matmul(a, b, 3, -2, nthreads=8)
    ctx.set_wait_limit(200)
    try:
        ctx.matmul(ta, tbb, to, 3, -2)
        assert ctx.last_kernel() == "tc_gemm_any_i8_i32"
        st = ctx.sync(check=False)
        assert st in (tb.Status.INTERNAL, tb.Status.OK)
    finally:
        ctx.set_wait_limit(4000000000)
    ctx.matmul(ta, tbb, to, 3, -2)
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out, exp)


@pytest.mark.parametrize("kind", ["i8 split", "f16 split", "f16 to f32", "f16 to f32 split", "f16 to f32 unaligned", "f8 to f32"])
def test_every_form_gives_up_and_recovers(ctx, kind):
    """The shortest wait limit on each form of the kernel: clusters that meet after a role gave up, tensor memory given back early,
    chunk sums read back.  It ends and reports (one call of twenty at least does not finish in time), and the same call is right
    afterwards."""
    N, H, C, W = {"i8 split": (1, 5, 3000, 300), "f16 split": (1, 64, 4000, 62), "f16 to f32": (40, 300, 2000, 61), "f16 to f32 split": (1, 64, 4000, 62),
                  "f16 to f32 unaligned": (2, 130, 3001, 63), "f8 to f32": (2, 130, 3001, 63)}[kind]
    r = util.rng(2450 + W)
    to = ctx.empty(tb.DType.INT32 if kind[0] == "i" else F32 if "f32" in kind else F16, (N, H, W))
    zp = (3, -2) if kind[0] == "i" else (0, 0)
    a, b = (r.integers(-3, 4, size=s).astype(np.int8) for s in ((N, H, C), (N, C, W)))    # small whole numbers: exact
    exp = (a.astype(np.float64) - zp[0]) @ (b.astype(np.float64) - zp[1])
    if kind[0] == "i":
        ta, tbb = ctx.from_numpy(a), ctx.from_numpy(b)
    elif kind[:3] == "f16":
        ta, tbb = ctx.from_numpy(a.astype(np.float16)), ctx.from_numpy(b.astype(np.float16))
    else:
        code = np.array([0, 0x38, 0x40, 0x44], np.uint8)    # E4M3 of 0, 1, 2, 3
        ta, tbb = (ctx.from_numpy(code[np.abs(v)] | (v < 0).astype(np.uint8) << 7, tb.DType.FP8E4M3) for v in (a, b))
    ctx.matmul(ta, tbb, to, *zp)
    assert ctx.last_kernel().startswith("tc_gemm_any")
    ctx.sync()
    ctx.set_wait_limit(1)
    try:
        for _ in range(20):
            ctx.matmul(ta, tbb, to, *zp)
            st = ctx.sync(check=False)
            if st == tb.Status.INTERNAL:
                break
    finally:
        ctx.set_wait_limit(4000000000)
    assert st == tb.Status.INTERNAL
    ctx.matmul(ta, tbb, to, *zp)
    st, out = to.download()
    assert st == tb.Status.OK and np.array_equal(out.astype(np.float64), exp)
    for t in (ta, tbb, to):
        t.free()


def test_two_streams_share_the_chip():
    """Products whose K is split over clusters, from two contexts (two streams) and two threads at once.  Their plans leave room
    for both on an SM in shared memory but not in tensor memory (512 and 64 columns and more): CTAs queue for columns, and
    the clusters still all meet."""
    errors = []

    def work(kind, shape, zp):
        try:
            N, H, C, W = shape
            r = util.rng(2500 + C)
            with tb.Context(0) as c:
                if kind == "i8":
                    a, b = r.integers(-128, 128, size=(N, H, C)).astype(np.int8), r.integers(-128, 128, size=(N, C, W)).astype(np.int8)
                    exp, dt = orc.matmul(a, b, *zp, nthreads=8), tb.DType.INT32
                else:    # small whole numbers: sums are exact in any order
                    a, b = (r.integers(-3, 4, size=s).astype(np.float16) for s in ((N, H, C), (N, C, W)))
                    exp, dt = np.matmul(a.astype(np.float32), b.astype(np.float32)).astype(np.float16), F16
                ta, tbb = c.from_numpy(a), c.from_numpy(b)
                outs = [c.empty(dt, exp.shape) for _ in range(4)]
                for i in range(400):
                    c.matmul(ta, tbb, outs[i % 4], *zp)
                assert c.last_kernel().startswith("tc_gemm_any")
                for to in outs:
                    st, out = to.download()
                    assert st == tb.Status.OK and np.array_equal(out, exp)
                for t in [ta, tbb] + outs:
                    t.free()
        except BaseException as e:    # reported by the main thread
            errors.append(e)

    jobs = [("i8", (6, 5, 3000, 300), (3, -2)), ("f16", (24, 64, 4000, 62), (0, 0))]
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("kind,size", [("i8", 30), ("i8", 120), ("f16", 14), ("f16", 90), ("f32", 14), ("f32", 90)])
def test_weights_that_an_operator_writes(ctx, kind, size):
    """Their tables would be built on every call: small layers read the weights where they are, in one launch; larger ones build
    them, and never use ones that have gone stale."""
    r = util.rng(2650 + size)
    IC, OC = 24, 40
    dt = {"i8": tb.DType.INT8, "f16": F16, "f32": F32}[kind]
    np_dt = {"i8": np.int8, "f16": np.float16, "f32": np.float32}[kind]
    x = r.integers(-3, 4, (1, size, size, IC)).astype(np_dt)    # small whole numbers: exact in any type and order
    tw = ctx.from_numpy(np.zeros((OC, 3, 3, IC), np_dt))
    tx, tbias, to = ctx.from_numpy(x), ctx.from_numpy(np.zeros(OC, np.int32 if kind == "i8" else np_dt)), ctx.empty(
        tb.DType.INT32 if kind == "i8" else dt, (1, size, size, OC))
    source = [ctx.empty(dt, tw.shape), ctx.empty(dt, tw.shape)]
    for rep in range(3):
        w = r.integers(-1, 2, tw.shape).astype(np_dt)
        if rep:    # CLAMP copies: its output is the weight tensor
            source[rep - 1].upload(w)
            ctx.clamp(source[rep - 1], tw, -100, 100)
        else:
            tw.upload(w)
        launches = ctx.launch_count()
        ctx.conv2d(tx, tw, tbias, to, [1] * 4, [1, 1], [1, 1])
        if rep:
            large = 9 * IC * OC * size * size > {"i8": 40000000, "f16": 0, "f32": 4000000}[kind]    # (fp16: sums of more than 128)
            assert (ctx.last_kernel() == "conv2d_direct") == (not large) and (large or ctx.launch_count() == launches + 1)
        xp = np.pad(x.astype(np.float64), ((0, 0), (1, 1), (1, 1), (0, 0)))
        exp = sum(xp[:, ky:ky + size, kx:kx + size] @ w[:, ky, kx].astype(np.float64).T for ky in range(3) for kx in range(3))
        st, out = to.download()
        assert st == tb.Status.OK and np.array_equal(out.astype(np.float64), exp)
    for t in [tx, tw, tbias, to] + source:
        t.free()


@pytest.mark.parametrize("kind", ["i8", "i8 rescale", "f16", "f32"])
def test_capture_before_any_eager_call(kind):
    """A convolution whose tables are neither built nor have room while capturing is captured all the same, on a kernel that needs
    none."""
    r = util.rng(2700)
    N, H, IC, OC = 2, 14, 100, 70
    with tb.Context(0) as c:
        if kind[0] == "i":
            x, w, b = util.conv_int8_case(r, N, H, H, IC, OC, 1, 1)
            exp = orc.conv2d(x, w, b, [0] * 4, [1, 1], [1, 1], 5, 0, nthreads=8)
        else:
            x, w, b = (r.integers(-3, 4, s).astype(np.float32) for s in ((N, H, H, IC), (OC, 1, 1, IC), (OC,)))
            exp = x @ w[:, 0, 0].T + b    # small whole numbers: exact
            if kind == "f16":
                x, w, b, exp = (v.astype(np.float16) for v in (x, w, b, exp))
        tensors = [c.from_numpy(v) for v in (x, w, b)]
        epi = None
        if kind == "i8 rescale":
            mult, shift = util.rescale_params(r, OC)
            tensors += [c.from_numpy(mult), c.from_numpy(shift)]
            epi = tb.Epilogue(tb.RescaleAttr(*tensors[3:], 0, 3, True, "DOUBLE_ROUND", per_channel=True), (-128, 127))
            exp = np.clip(orc.rescale(exp, mult, shift, True, True, "DOUBLE_ROUND", 0, 3, 32, 8)[1], -128, 127)
        to = c.empty({"i8": tb.DType.INT32, "i8 rescale": tb.DType.INT8, "f16": F16, "f32": F32}[kind], exp.shape)
        c.capture_begin()
        c.conv2d(*tensors[:3], to, [0] * 4, [1, 1], [1, 1], 5 if kind[0] == "i" else 0, 0, epi)
        graph = c.capture_end()
        c.graph_launch(graph)
        st, out = to.download()
        assert st == tb.Status.OK and np.array_equal(out, exp)
        c.graph_destroy(graph)
        for t in tensors + [to]:
            t.free()


def test_as_many_pixels_as_a_tensor_holds(ctx):
    """2^31 - 8 output pixels: the last tile's rows would not have 32-bit numbers, another kernel takes the call."""
    n = (1 << 31) - 8
    x = np.frombuffer(util.rng(2800).bytes(n), np.int8).reshape(1, 1, n, 1)
    w, b = np.array([77], np.int8).reshape(1, 1, 1, 1), np.array([-1234], np.int32)
    mult, shift = np.array([1 << 30], np.int32), np.array([37], np.int8)
    every = np.arange(256, dtype=np.uint8).view(np.int8)    # the result depends on the byte alone
    lut = orc.rescale(every.astype(np.int32) * 77 - 1234, mult, shift, False, True, "SINGLE_ROUND", 0, 2, 32, 8)[1].astype(np.int8)
    tensors = [ctx.from_numpy(v) for v in (x, w, b, mult, shift)]
    to = ctx.empty(tb.DType.INT8, x.shape)
    ctx.conv2d(*tensors[:3], to, [0] * 4, [1, 1], [1, 1], 0, 0, tb.Epilogue(tb.RescaleAttr(*tensors[3:], 0, 2, True, "SINGLE_ROUND"), None))
    st, out = to.download()
    assert st == tb.Status.OK
    x, out = x.reshape(-1).view(np.uint8), out.reshape(-1)
    for at in range(0, n, 1 << 27):
        assert np.array_equal(out[at:at + (1 << 27)], lut[x[at:at + (1 << 27)]])
    for t in tensors + [to]:
        t.free()
