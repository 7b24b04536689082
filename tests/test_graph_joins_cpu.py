"""The graph runner around residual joins that run inside a convolution (fuse_joins, CONV_JOIN), without a GPU: a context
whose operators are the oracle's, on host arrays."""
import numpy as np
import pytest

import reference_model_b200 as tb
from oracle import graph_eval
from oracle import oracle as orc
from reference_model_b200 import graph as G

I8, I32 = tb.DType.INT8, tb.DType.INT32


class _Tensor:
    def __init__(self, ctx, dtype, shape):
        self.ctx, self.a = ctx, np.full(shape, 77, {I8: np.int8, I32: np.int32}[tb.DType(dtype)])
        self.written = 0

    def upload(self, array):
        self.a[...] = array
        self.ctx.writes += 1
        self.written = self.ctx.writes

    def download(self, check=True):
        return tb.Status.OK, self.a.copy()


class _Context:
    """Results are written into the output's array at once, as a kernel would."""

    def __init__(self):
        self.kinds, self.writes = [], 0

    def empty(self, dtype, shape):
        return _Tensor(self, dtype, shape)

    def from_numpy(self, array, dtype=None):
        t = _Tensor(self, I8 if array.dtype == np.int8 else I32, array.shape)
        t.upload(array)
        return t

    def conv2d(self, x, w, b, out, pad, stride, dil, izp, wzp, epi):
        self.kinds.append("conv2d")
        acc = orc.conv2d(x.a, w.a, b.a, pad, stride, dil, izp, wzp, nthreads=4)
        rs, (lo, hi) = epi
        out.a[...] = np.clip(orc.rescale(acc, rs[0].a, rs[1].a, *rs[2:], 32, 8)[1], lo, hi)

    def residual_add(self, a, ra, b, rb, ro, out, clamp):
        self.kinds.append("residual_add")
        leg = lambda t, r: orc.rescale(t.a, r[0].a, r[1].a, *r[2:], 8, 32)[1]
        s = orc.add(leg(a, ra), leg(b, rb))[1]
        out.a[...] = np.clip(orc.rescale(s, ro[0].a, ro[1].a, *ro[2:], 32, 8)[1], *clamp)

    def conv2d_add(self, x, w, b, out, pad, stride, dil, izp, wzp, epi, leg, other, other_leg, ro, clamp):
        t = _Tensor(self, I8, out.a.shape)
        self.conv2d(x, w, b, t, pad, stride, dil, izp, wzp, epi)
        self.residual_add(t, leg, other, other_leg, ro, out, clamp)
        self.kinds[-2:] = ["conv2d_add"]


@pytest.fixture()
def ctx(monkeypatch):
    monkeypatch.setattr(G.tb, "Epilogue", lambda rescale, clamp: (rescale, clamp))
    monkeypatch.setattr(G.tb, "RescaleAttr", lambda m, s, izp, ozp, scale32, rounding, per_channel, iu, ou: (m, s, per_channel, scale32, rounding, izp, ozp))
    return _Context()


class _Net:
    """A graph of 8-channel 5x5 convolutions and joins, by name."""

    def __init__(self, inputs=("x",)):
        self.g, self.r = G.Graph(), np.random.default_rng(5)
        for name in inputs:
            self.g.inputs.append(self.g.tensor(name, I8, (1, 5, 5, 8)))

    def conv(self, x, y):
        g, r = self.g, self.r
        w, b = g.const(y + "_w", r.integers(-127, 128, (8, 1, 1, 8)).astype(np.int8)), g.const(y + "_b", np.zeros(8, np.int32))
        m, s = g.const(y + "_m", np.array([1 << 30], np.int32)), g.const(y + "_s", np.array([38], np.int8))
        acc, q = g.tensor(y + "_acc", I32, (1, 5, 5, 8)), g.tensor(y + "_q", I8, (1, 5, 5, 8))
        g.add("CONV2D", [x, w, b], [acc], pad=[0] * 4, stride=[1, 1], dilation=[1, 1], input_zp=0, weight_zp=0)
        g.add("RESCALE", [acc, m, s], [q], input_zp=0, output_zp=0, scale32=True, rounding="SINGLE_ROUND", per_channel=False)
        g.add("CLAMP", [q], [g.tensor(y, I8, (1, 5, 5, 8))], min_val=-128, max_val=127)

    def join(self, a, b, y):
        g = self.g
        t = lambda k, dt: g.tensor(y + k, dt, (1, 5, 5, 8))
        c = lambda k, m, s: [g.const(y + k + "m", np.array([m], np.int32)), g.const(y + k + "s", np.array([s], np.int8))]
        rs = dict(input_zp=0, output_zp=0, scale32=True, rounding="SINGLE_ROUND", per_channel=False)
        g.add("RESCALE", [a] + c("a", 1 << 30, 30), [t("_a", I32)], **rs)
        g.add("RESCALE", [b] + c("b", 1 << 30, 30), [t("_b", I32)], **rs)
        g.add("ADD", [y + "_a", y + "_b"], [t("_sum", I32)])
        g.add("RESCALE", [y + "_sum"] + c("o", 1 << 30, 31), [t("_q", I8)], **rs)
        g.add("CLAMP", [y + "_q"], [t("", I8)], min_val=-128, max_val=127)

    def image(self, k=0):
        return np.random.default_rng(100 + k).integers(-128, 128, (1, 5, 5, 8)).astype(np.int8)


def _block(outputs=("y",)):
    """x -> stem -> (a -> b) + stem -> y: the block of a residual network."""
    n = _Net()
    n.conv("x", "stem")
    n.conv("stem", "a")
    n.conv("a", "b")
    n.join("b", "stem", "y")
    n.g.outputs += list(outputs)
    return n


def _ref(n, x):
    return graph_eval.evaluate(n.g, {"x": x}, nthreads=4)[1]


def test_a_buffer_of_the_caller_is_written_by_every_evaluation(ctx):
    n, mine = _block(), ctx.empty(I8, (1, 5, 5, 8))
    run = G.DeviceRunner(ctx, n.g, external={"b": mine})
    for k in range(2):
        run.set_input(n.image(k))
        run.run()
        ref = _ref(n, n.image(k))
        assert np.array_equal(mine.a, ref["b"]) and np.array_equal(run.output()[1], ref["y"])


def test_a_result_inside_a_step_is_that_of_the_last_evaluation(ctx):
    n = _block()
    run = G.DeviceRunner(ctx, n.g)
    assert [k for k, _ in run.steps] == ["CONV_RESCALE_CLAMP"] * 2 + ["CONV_JOIN"]
    run.set_input(n.image(0))
    run.run()
    ref = _ref(n, n.image(0))
    run.set_input(n.image(1))    # the next image is there already
    for name in ("b", "a", "stem", "y"):
        assert np.array_equal(run.output(name)[1], ref[name]), name
        assert np.array_equal(run.t[name].download()[1], ref[name]), name
    run.run()
    ref = _ref(n, n.image(1))
    assert np.array_equal(run.t["b"].download()[1], ref["b"]) and np.array_equal(run.output("b")[1], ref["b"])
    assert "b" not in run.t    # nothing that the next evaluation would leave as it is
    with pytest.raises(KeyError):
        run.t["b_q"]
    # its weights are others now: what it was cannot be made again, and it says so
    run.t["b_w"].upload(np.zeros((8, 1, 1, 8), np.int8))
    with pytest.raises(RuntimeError):
        run.output("b")
    run.run()
    assert np.array_equal(run.output("b")[1], np.zeros((1, 5, 5, 8), np.int8))


@pytest.mark.parametrize("view", [False, True])
def test_a_convolution_of_the_graphs_input_keeps_its_result(ctx, view):
    """... as an evaluation made it, whatever the caller has uploaded since."""
    n = _Net(("x", "z"))
    src = "x"
    if view:
        src = n.g.tensor("v", I8, (1, 5, 5, 8))
        n.g.add("IDENTITY", ["x"], [src])
    n.conv(src, "a")
    n.join("a", "z", "y")
    n.g.outputs.append("y")
    run = G.DeviceRunner(ctx, n.g)
    z = n.image(9)
    run.set_input(n.image(0), "x"), run.set_input(z, "z")
    run.run()
    ref = graph_eval.evaluate(n.g, {"x": n.image(0), "z": z}, nthreads=4)[1]
    run.set_input(n.image(1), "x")
    assert np.array_equal(run.output("a")[1], ref["a"]) and np.array_equal(run.output()[1], ref["y"])


def test_joins_in_place_on_memory_of_the_caller(ctx):
    """The join's result over its other operand, or over what a step between the convolution and the join reads."""
    n = _Net(("x", "z"))
    n.conv("x", "a")
    n.conv("a", "b")
    n.join("b", "z", "y")
    n.g.outputs.append("y")
    buf = ctx.empty(I8, (1, 5, 5, 8))
    ref = graph_eval.evaluate(n.g, {"x": n.image(0), "z": n.image(1)}, nthreads=4)[1]
    run = G.DeviceRunner(ctx, n.g, external={"z": buf, "y": buf})
    assert "CONV_JOIN" not in [k for k, _ in run.steps]    # tb200_conv2d_add refuses an output over the other operand
    run.set_input(n.image(0), "x"), run.set_input(n.image(1), "z")
    run.run()
    assert np.array_equal(buf.a, ref["y"])

    n = _Net(("x", "z"))
    n.conv("x", "a")
    n.conv("a", "b")
    n.conv("z", "late")
    n.join("b", "a", "y")
    n.g.outputs += ["y", "late"]
    ref = graph_eval.evaluate(n.g, {"x": n.image(0), "z": n.image(1)}, nthreads=4)[1]
    run = G.DeviceRunner(ctx, n.g, external={"z": buf, "y": buf})
    run.set_input(n.image(0), "x"), run.set_input(n.image(1), "z")
    run.run()
    assert np.array_equal(run.output("late")[1], ref["late"]) and np.array_equal(buf.a, ref["y"])
    # an output of the caller's that meets none of its other tensors is no obstacle
    run = G.DeviceRunner(ctx, _block().g, external={"y": buf, "x": ctx.empty(I8, (1, 5, 5, 8))})
    assert "CONV_JOIN" in [k for k, _ in run.steps]


def test_bench_counts_the_other_operand_of_a_join_inside_a_convolution():
    import bench
    g = G.resnet50_int8(1, image=96)
    fused, inside = G.fuse_joins(g, G.fuse(g))
    apart = [s for s in G.fuse(g)]
    size = lambda n: int(np.prod(g.meta[n][1]))
    # a join inside saves writing the convolution's result and reading it again, and nothing else
    assert len(inside) == 16
    assert bench.activation_bytes(g, apart) - bench.activation_bytes(g, fused) == 2 * sum(size(n) for n in inside)


def _kinds(n):
    return [k for k, _ in G.fuse_joins(n.g, G.fuse(n.g))[0]]


def _runs_right(ctx, n, inputs=("x",)):
    """Every tensor that the runner can name is that of the oracle."""
    x = {name: n.image(k) for k, name in enumerate(inputs)}
    run = G.DeviceRunner(ctx, n.g)
    for name, a in x.items():
        run.set_input(a, name)
    run.run()
    ref = graph_eval.evaluate(n.g, x, nthreads=4)[1]
    for name in n.g.meta:
        if name in run.t or name in run._inside:
            assert np.array_equal(run.output(name)[1], ref[name]), name


def test_the_later_of_two_convolutions_takes_the_join(ctx):
    n = _Net()
    n.conv("x", "in")
    n.conv("in", "a")
    n.conv("in", "b")
    n.join("a", "b", "y")    # b is there last
    n.g.outputs.append("y")
    steps, inside = G.fuse_joins(n.g, G.fuse(n.g))
    assert [k for k, _ in steps] == ["CONV_RESCALE_CLAMP"] * 2 + ["CONV_JOIN"] and list(inside) == ["b"]
    _runs_right(ctx, n)
    n = _Net()
    n.conv("x", "in")
    n.conv("in", "a")
    n.conv("in", "b")
    n.join("b", "a", "y")    # ... as the first operand
    n.g.outputs.append("y")
    assert list(G.fuse_joins(n.g, G.fuse(n.g))[1]) == ["b"]
    _runs_right(ctx, n)


def test_an_operand_that_is_made_later_is_waited_for(ctx):
    """Only the convolution that is there first has no other reader: it cannot take what is not there yet."""
    n = _Net()
    n.conv("x", "in")
    n.conv("in", "a")
    n.conv("in", "b")
    n.conv("b", "c")         # a second reader of b
    n.join("a", "b", "y")
    n.join("y", "c", "z")    # c is there before y is
    n.g.outputs.append("z")
    kinds = _kinds(n)
    assert kinds.count("RESIDUAL_JOIN") == 2 and "CONV_JOIN" not in kinds
    _runs_right(ctx, n)


@pytest.mark.parametrize("why", ["graph output", "second reader", "same tensor"])
def test_results_that_others_read_stay_outside(ctx, why):
    n = _Net()
    n.conv("x", "in")
    n.conv("in", "a")
    n.join("a", "a" if why == "same tensor" else "in", "y")
    n.g.outputs.append("y")
    if why == "graph output":
        n.g.outputs.append("a")
    elif why == "second reader":
        n.conv("a", "c")
        n.g.outputs.append("c")
    assert "CONV_JOIN" not in _kinds(n)
    _runs_right(ctx, n)


def test_a_chain_of_blocks(ctx):
    """Joins over joins, as a network has them: the result of one is the other operand of the next."""
    n = _Net()
    n.conv("x", "s0")
    for i in range(3):
        n.conv("s%d" % i, "a%d" % i)
        n.conv("a%d" % i, "b%d" % i)
        n.join("b%d" % i, "s%d" % i, "s%d" % (i + 1))
    n.g.outputs.append("s3")
    assert _kinds(n).count("CONV_JOIN") == 3
    _runs_right(ctx, n)


def test_a_runner_goes_with_its_last_reference(ctx):
    """... and its graph's arrays with it, not at the garbage collector's next look."""
    import gc
    import weakref
    gc.disable()
    try:
        n = _block()
        run = G.DeviceRunner(ctx, n.g)
        ref = weakref.ref(run)
        del run
        assert ref() is None
    finally:
        gc.enable()
