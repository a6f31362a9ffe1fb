"""BatchNorm + addition + ReLU on tensors that are windows of larger blocks, at any float: the form without a mask takes them."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _window(array, offset):
    """`array` (channels-last in memory) in a window that starts `offset` floats into its block."""
    import mytorch_b200 as mt
    from mytorch_b200.backends.cuda.env import CudaMemory, CudaMemoryView
    from mytorch_b200.tensor import Device, Tensor

    view = CudaMemoryView(CudaMemory(0, 4 * (array.size + 4)), 4 * offset, 4 * array.size, 0)
    view.write(np.ascontiguousarray(array.transpose(0, 2, 3, 1)))
    return Tensor._on_device(array.shape, mt.float32, Device("cuda:0"), view)


@pytest.mark.parametrize("offsets", [(1, 0, 0), (0, 2, 0), (0, 0, 3), (3, 3, 1)], ids="x{0[0]} res{0[1]} dy{0[2]}".format)
def test_windows_at_any_float(offsets):
    import gpu_util as g

    rng = np.random.default_rng(8)
    x, res, dy = rng.standard_normal((3, 3, 8, 5, 7)).astype(np.float32)
    gamma, beta = g.dev(rng.uniform(0.5, 1.5, 8).astype(np.float32), True), g.dev(rng.standard_normal(8).astype(np.float32), True)

    def run(place):
        xt, rt, dyt = (place(a, o) for a, o in zip((x, res, dy), offsets))
        running = g.dev(np.zeros(8, np.float32)), g.dev(np.ones(8, np.float32))
        y, mean, var = g.op("batch_norm2d_add_relu")(xt, rt, gamma, beta, 1e-5, True, 0.1, *running)
        grads = g.op("batch_norm2d_add_relu_backward")(dyt, mean, var, xt, rt, gamma, beta, 1e-5)
        return [g.host(t) for t in (y, mean, var, *running, *grads)]

    for got, want in zip(run(_window), run(lambda a, _: g.dev(a))):
        assert rel_err(got, want) < 1e-5  # 32-bit sums of 105 terms in another order


def test_refused_call_leaves_the_running_statistics():
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv, CudaMemory, NativeError

    env = CudaEnv.instance()
    a = np.random.default_rng(1).standard_normal((2, 8, 4, 4)).astype(np.float32)
    x, res, y = _window(a, 1), g.dev(a), g.dev(a)
    mean, var, rm, rv = (g.dev(np.full(8, v, np.float32)) for v in (0, 0, 3, 4))
    ws, nbytes = env.workspace(env.lib.batch_norm2d_workspace_bytes(2, 8, 4, 4))
    with pytest.raises(NativeError):
        env.lib.batch_norm2d_add_relu_forward_masked_f32(2, 8, 4, 4, x, res, None, None, 1e-5, 1, 0.1, rm, rv, y, mean, var, CudaMemory(0, 64), None, 0,
                                                         ws, nbytes, env.stream())
    assert (g.host(rm) == 3).all() and (g.host(rv) == 4).all()
