"""An operator may add its data gradient in place only to a gradient that belongs to its input alone: an addition hands
one tensor to both operands, and a leaf may hold the gradient of an earlier pass."""
import numpy as np
import pytest

import mytorch_b200 as mt


def _total(x, factor=1.0):
    return (x * factor).sum()


@pytest.fixture
def tape():
    """A strided pick with a weight (y = k x[::2]) whose backward adds in place when it may, and an addition, on the host."""
    from mytorch_b200.autograd import DAGTracker
    from mytorch_b200.ops._common import record

    tr = DAGTracker.instance()
    names = ("t_pick", "t_add", "t_total")
    in_place = []

    def out(a, *inputs):
        t = mt.tensor(a.astype(np.float32))
        t.requires_grad = any(i.requires_grad for i in inputs)
        return t

    def pick(x, k):
        return record("t_pick", [x, k], out(k * x._cpu_array[::2], x))

    def add(a, b):
        return record("t_add", [a, b], out(a._cpu_array + b._cpu_array, a, b))

    def total(*xs):
        return record("t_total", list(xs), out(np.array([sum(x._cpu_array.sum() for x in xs)]), *xs))

    @tr.register_backward_function("t_pick")
    def _(dy, x, k, accumulate_dx=None, accumulate_shared=False):
        mine = np.zeros(x.shape, np.float32)
        mine[::2] = k * dy._cpu_array
        if accumulate_dx is None:
            return [mt.tensor(mine), None]
        in_place.append(not accumulate_shared)
        if accumulate_shared:
            return [mt.tensor(mine + accumulate_dx._cpu_array), None]
        accumulate_dx._cpu_array += mine
        return [accumulate_dx, None]

    @tr.register_backward_function("t_add")
    def _(dy, a, b):
        return [dy, dy]

    @tr.register_backward_function("t_total")
    def _(dy, *xs):
        return [mt.tensor(np.full(x.shape, dy._cpu_array[0], np.float32)) for x in xs]

    tr.fused_accumulate["t_pick"] = 0
    tr.accumulates_in_place.add("t_pick")
    yield pick, add, total, in_place
    for name in names:
        del tr._backward_funcs[name]
    del tr.fused_accumulate["t_pick"]
    tr.accumulates_in_place.discard("t_pick")


def _leaf(values):
    return mt.tensor(np.array(values, np.float32), requires_grad=True)


def test_gradient_of_an_addition_stays_as_it_was(tape):
    pick, add, total, in_place = tape
    x, w = _leaf([1, 2, 3, 4]), _leaf([5, 6, 7, 8])
    y = pick(x, 3.0)
    total(y, add(x, w)).backward()
    assert np.array_equal(x.grad._cpu_array, [4, 1, 4, 1]) and np.array_equal(w.grad._cpu_array, [1, 1, 1, 1])
    assert in_place == [False]


def test_gradient_of_an_earlier_pass_stays_as_it_was(tape):
    pick, add, total, in_place = tape
    x = _leaf([1, 2])
    total(x).backward()
    before = x.grad
    total(pick(x, 2.0)).backward()
    assert np.array_equal(x.grad._cpu_array, [3, 1]) and np.array_equal(before._cpu_array, [1, 1]) and in_place == [False]


def test_gradient_made_for_the_input_alone_is_added_to(tape):
    pick, add, total, in_place = tape
    x = _leaf([1, 2])
    a, b = pick(x, 2.0), pick(x, 5.0)
    total(a, b).backward()
    assert np.array_equal(x.grad._cpu_array, [7, 0]) and in_place == [True]


@pytest.mark.gpu
def test_strided_convolution_beside_an_addition():
    """The 1x1 / stride-2 convolution accumulates in place; its input's gradient so far is also the other operand's."""
    import gpu_util as g
    import mytorch_b200.nn as nn

    rng = np.random.default_rng(2)
    x, w = (g.dev(rng.standard_normal((8, 64, 32, 32)).astype(np.float32), True) for _ in range(2))
    conv = nn.Conv2d(64, 128, 1, 2, bias=False)
    conv.to(g.DEV)
    y = conv(x)
    (_total(y) + _total(x + w)).backward()
    assert np.array_equal(g.host(w.grad), np.ones(w.shape, np.float32))
    column = g.host(conv.weight.detach()).astype(np.float64).sum((0, 2, 3))
    want = np.ones(x.shape)
    want[:, :, ::2, ::2] += column[None, :, None, None]
    assert np.abs(g.host(x.grad) - want).max() < 2e-3  # sums of 128 weights under 1/8, operands in TF32: 128 / 8 * 2^-11 / sqrt(128)
