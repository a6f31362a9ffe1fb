"""Convolutions over channel counts of any size on the tensor cores, operands as sums of two TF32 numbers: tiles, blocks of
channels and pixels that are not full, strides, several groups of images, against 64 bits and against the CUDA-core kernels."""
import numpy as np
import pytest

from oracle import ops as O

pytestmark = pytest.mark.gpu


def _operands(n, cin, cout, h, w, k, stride, pad, seed=0):
    rng = np.random.default_rng(seed + cin + cout)
    x, wt = rng.standard_normal((n, cin, h, w)).astype(np.float32), (rng.standard_normal((cout, cin, k, k)) / (cin * k * k) ** 0.5).astype(np.float32)
    dy = rng.standard_normal((n, cout, (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1)).astype(np.float32)
    return x, wt, dy


def _run(x, wt, b, dy, stride, pad):
    import gpu_util as g

    s, p = (stride, stride), (pad, pad)
    xt, wtt, bt = g.dev(x, True), g.dev(wt, True), g.dev(b)
    y = g.op("conv2d")(xt, wtt, bt, s, p)
    dx, dw, _ = g.op("conv2d_backward")(g.dev(dy), xt, wtt, None, s, p)
    return [g.host(t) for t in (y, dx, dw)]


@pytest.mark.parametrize("n,cin,cout,h,w,k,stride,pad", [
    (8, 33, 31, 12, 13, 3, 1, 1), (5, 48, 82, 19, 17, 3, 1, 1), (9, 70, 129, 21, 15, 3, 2, 1), (40, 36, 100, 9, 11, 1, 1, 0), (3, 130, 66, 23, 20, 5, 1, 0),
    (33, 41, 161, 10, 10, 3, 3, 0), (20, 37, 35, 16, 16, 1, 2, 0), (2, 64, 70, 41, 39, 3, 1, 2)])
def test_against_64_bits_and_the_other_kernels(n, cin, cout, h, w, k, stride, pad, monkeypatch):
    x, wt, dy = _operands(n, cin, cout, h, w, k, stride, pad)
    b = np.random.default_rng(1).standard_normal(cout).astype(np.float32)
    monkeypatch.setenv("MTB_TC_SPLIT_ALWAYS", "1")
    got = _run(x, wt, b, dy, stride, pad)
    assert all(np.array_equal(u, v) for u, v in zip(got, _run(x, wt, b, dy, stride, pad)))
    monkeypatch.delenv("MTB_TC_SPLIT_ALWAYS")
    monkeypatch.setenv("MTB_DISABLE_TC", "1")
    other = _run(x, wt, b, dy, stride, pad)
    d = [t.astype(np.float64) for t in (x, wt, b, dy)]
    s, p = (stride, stride), (pad, pad)
    exact = lambda x, wt, b, dy: [O.conv2d_forward(x, wt, b, s, p), *O.conv2d_backward(dy, x, wt, False, s, p)[:2]]
    terms = (cin * k * k, cout * k * k, dy[:, 0].size)
    for a, o, want, size, count in zip(got, other, exact(*d), exact(*(np.abs(t) for t in d)), terms):
        # an operand is off by 2^-22 at most, the term left out is 2^-22, a chain truncates 12 times, chains are added in FP32
        assert (np.abs(a - want) <= (18 + count / 32) * 2.0 ** -23 * size).all()
        err = lambda t: np.linalg.norm(t - want) / np.linalg.norm(want)
        assert not np.array_equal(a, o)  # it was these kernels that ran
        assert err(a) <= max(err(o), 2.0e-7)  # 2e-7: what sums of some hundred terms, which these kernels are taken for, have in FP32


def test_several_groups_of_images(monkeypatch):
    x, wt, dy = _operands(70, 33, 40, 64, 64, 3, 1, 1)  # packed, 2 MB an image: three groups
    b = np.zeros(40, np.float32)
    monkeypatch.setenv("MTB_TC_SPLIT_ALWAYS", "1")
    got = _run(x, wt, b, dy, 1, 1)
    monkeypatch.delenv("MTB_TC_SPLIT_ALWAYS")
    monkeypatch.setenv("MTB_DISABLE_TC", "1")
    want, size = _run(x, wt, b, dy, 1, 1), _run(*(np.abs(t) for t in (x, wt, b, dy)), 1, 1)
    for a, o, m, count in zip(got, want, size, (33 * 9, 40 * 9, 70 * 64 * 64)):
        assert not np.array_equal(a, o)
        terms = 18 + count / 32 + count  # both sides' rounding
        assert (np.abs(a - o) <= terms * 2.0 ** -23 * m).all()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.3e38])
def test_values_that_cannot_be_split(value, monkeypatch):
    x, wt, dy = _operands(70, 33, 40, 64, 64, 3, 1, 1)
    x[69, 5, 7, 9] = dy[1, 2, 3, 4] = value  # x in the last group of images, dy in the first
    b = np.zeros(40, np.float32)
    monkeypatch.setenv("MTB_TC_SPLIT_ALWAYS", "1")
    got = _run(x, wt, b, dy, 1, 1)
    monkeypatch.delenv("MTB_TC_SPLIT_ALWAYS")
    monkeypatch.setenv("MTB_DISABLE_TC", "1")
    want = _run(x, wt, b, dy, 1, 1)
    assert np.array_equal(got[0], want[0], equal_nan=True) and np.array_equal(got[1], want[1], equal_nan=True)
    a, o = got[2], want[2]  # the sum over pixels is split otherwise: a partial sum may overflow on one side only
    clean = np.isfinite(a) & np.isfinite(o) & (np.abs(o) < 1e30)
    assert np.array_equal(np.isnan(a), np.isnan(o)) if not np.isfinite(value) else True
    assert np.allclose(a[clean], o[clean], rtol=0, atol=1e-5 * 70 * 64 * 64 ** 0.5) and clean.any()


@pytest.mark.parametrize("x_scale,w_scale", [(1e-37, 1.0), (1.0, 1e-37), (1e-35, 1e10), (0.0, 1.0)])
def test_tiny_operands(x_scale, w_scale, monkeypatch):
    """Where a whole operand is so small that its remainders are no normal numbers, the other kernels do the work."""
    x, wt, dy = _operands(5, 48, 82, 19, 17, 3, 1, 1)
    x, wt, dy = x * np.float32(x_scale), wt * np.float32(w_scale), dy * np.float32(x_scale)
    b = np.zeros(82, np.float32)
    monkeypatch.setenv("MTB_TC_SPLIT_ALWAYS", "1")
    got = _run(x, wt, b, dy, 1, 1)[:2]  # weight gradients of such operands are zero, or do not see the filter
    monkeypatch.delenv("MTB_TC_SPLIT_ALWAYS")
    monkeypatch.setenv("MTB_DISABLE_TC", "1")
    assert all(np.array_equal(a, o) for a, o in zip(got, _run(x, wt, b, dy, 1, 1)))


def test_a_tiny_value_among_others_refuses_nothing(monkeypatch):
    x, wt, dy = _operands(5, 48, 82, 19, 17, 3, 1, 1)
    x[1, 2, 3, 4] = wt[5, 6, 1, 1] = 1e-39
    b = np.zeros(82, np.float32)
    monkeypatch.setenv("MTB_TC_SPLIT_ALWAYS", "1")
    got = _run(x, wt, b, dy, 1, 1)
    monkeypatch.delenv("MTB_TC_SPLIT_ALWAYS")
    monkeypatch.setenv("MTB_DISABLE_TC", "1")
    for a, o in zip(got, _run(x, wt, b, dy, 1, 1)):
        assert not np.array_equal(a, o) and np.linalg.norm(a - o) <= 2e-6 * np.linalg.norm(o)


def test_without_scratch_the_other_kernels_run():
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv

    env = CudaEnv.instance()
    x, wt, _ = _operands(32, 48, 82, 37, 37, 3, 1, 1)
    xt, wtt = g.dev(x), g.dev(wt)
    y, args = g.dev(np.zeros((32, 82, 37, 37), np.float32)), (32, 48, 37, 37, 3, 3, 1, 1, 1, 1, 82)
    env.lib.conv2d_forward_f32(*args, xt, wtt, None, y, 0, None, 0, env.stream())
    want = g.host(g.op("conv2d")(xt, wtt, None, (1, 1), (1, 1)))
    assert np.abs(g.host(y) - want).max() <= 432 * 2.0 ** -23 * np.abs(x).max() * np.abs(wt).sum((1, 2, 3)).max()


def test_price_and_packed_image_decide(monkeypatch):
    """Without being forced: taken where the price says so, and not where one packed image is over the limit."""
    b = np.zeros(82, np.float32)
    x, wt, dy = _operands(32, 48, 82, 37, 37, 3, 1, 1)
    got = _run(x, wt, b, dy, 1, 1)
    monkeypatch.setenv("MTB_DISABLE_TC_SPLIT", "1")
    assert not any(np.array_equal(a, o) for a, o in zip(got, _run(x, wt, b, dy, 1, 1)))
    monkeypatch.delenv("MTB_DISABLE_TC_SPLIT")
    x, wt, dy = _operands(1, 33, 34, 800, 700, 3, 1, 1)  # 287 MB packed
    got = _run(x, wt, b[:34], dy, 1, 1)
    monkeypatch.setenv("MTB_DISABLE_TC_SPLIT", "1")
    assert all(np.array_equal(a, o) for a, o in zip(got, _run(x, wt, b[:34], dy, 1, 1)))


@pytest.mark.parametrize("relu", [True, False])
def test_with_batch_norm_and_residual(relu, monkeypatch):
    """Convolution and BatchNorm with running statistics in one operator have the bits of the two; so have a residual and the ReLU."""
    import gpu_util as g

    x, wt, _ = _operands(8, 48, 82, 37, 37, 3, 1, 1)
    rng = np.random.default_rng(4)
    gamma, beta, mean = (g.dev(rng.standard_normal(82).astype(np.float32)) for _ in range(3))
    var, res = g.dev(rng.uniform(0.5, 1.5, 82).astype(np.float32)), g.dev(rng.standard_normal((8, 82, 37, 37)).astype(np.float32))
    xt, wtt, bt = g.dev(x), g.dev(wt), g.dev(rng.standard_normal(82).astype(np.float32))
    one = g.op("conv2d_batch_norm")(xt, wtt, bt, (1, 1), (1, 1), gamma, beta, mean, var, 1e-5, relu, res if relu else None)
    monkeypatch.setenv("MTB_DISABLE_TC_SPLIT", "1")
    assert not np.array_equal(g.host(one), g.host(g.op("conv2d_batch_norm")(xt, wtt, bt, (1, 1), (1, 1), gamma, beta, mean, var, 1e-5, relu,
                                                                            res if relu else None)))
    monkeypatch.delenv("MTB_DISABLE_TC_SPLIT")
    y = g.op("conv2d")(xt, wtt, bt, (1, 1), (1, 1))
    norm = g.op("batch_norm2d")(y, gamma, beta, 1e-5, False, 0.1, mean, var)[0]
    want = g.host(norm)
    if relu:
        want = np.maximum(want + g.host(res), 0)
    assert np.array_equal(g.host(one), want)


def test_data_gradient_added_to_another(monkeypatch):
    import gpu_util as g

    x, wt, dy = _operands(8, 48, 82, 37, 37, 3, 1, 1)
    add = np.random.default_rng(3).standard_normal(x.shape).astype(np.float32)
    xt, wtt, dyt = g.dev(x, True), g.dev(wt), g.dev(dy)
    run = lambda **more: g.host(g.op("conv2d_backward")(dyt, xt, wtt, None, (1, 1), (1, 1), **more)[0])
    dx = run()
    assert np.array_equal(run(accumulate_dx=g.dev(add)), dx + add)
    monkeypatch.setenv("MTB_DISABLE_TC_SPLIT", "1")
    assert not np.array_equal(dx, run())


def test_captured():
    """Replays of a captured forward and backward pass on refilled inputs have the bits of eager calls."""
    import gpu_util as g
    from mytorch_b200.cuda_graph import StepGraph

    x, wt, dy = _operands(8, 48, 82, 37, 37, 3, 1, 1)
    xt, wtt, dyt = g.dev(x, True), g.dev(wt, True), g.dev(dy)

    def step():
        y = g.op("conv2d")(xt, wtt, None, (1, 1), (1, 1))
        return [y, *g.op("conv2d_backward")(dyt, xt, wtt, None, (1, 1), (1, 1))[:2]]

    graph = StepGraph(step)
    out = graph.capture()
    for scale in (1.0, 0.5, np.inf):
        xt.copy_(g.dev((x * np.float32(scale)).astype(np.float32)))
        graph.replay()
        got = [g.host(t) for t in out]
        assert all(np.array_equal(a, g.host(b), equal_nan=True) for a, b in zip(got, step()))
    graph.destroy()
