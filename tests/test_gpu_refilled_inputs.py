"""A weight gradient belongs to the values it is asked for: an input of few channels, which forward packs into blocks of 32,
may be refilled in place between a forward call and a backward call."""
import gc

import numpy as np
import pytest

from conftest import rel_err
from oracle import ops as O

pytestmark = pytest.mark.gpu
TF32_TOL = 5e-3


@pytest.mark.parametrize("cin,k", [(1, 3), (3, 3), (3, 7), (20, 3)])  # every form of the packing
@pytest.mark.parametrize("refill", ["copy_", "upload_into"])
def test_operator_call_reads_the_input_it_is_given(cin, k, refill):
    import gpu_util as g
    from mytorch_b200.backends.cuda.ops import upload_into

    rng = np.random.default_rng(cin + k)
    first, second = rng.standard_normal((2, 2, cin, 32, 32)).astype(np.float32)
    wt, dy = rng.standard_normal((32, cin, k, k)).astype(np.float32), rng.standard_normal((2, 32, 32, 32)).astype(np.float32)
    x, w, stride, pad = g.dev(first), g.dev(wt, True), (1, 1), (k // 2, k // 2)
    g.op("conv2d")(x, w, None, stride, pad)
    if refill == "copy_":
        x.copy_(g.dev(second))
    else:
        upload_into(x, second)
    _, dw, _ = g.op("conv2d_backward")(g.dev(dy), x, w, None, stride, pad)
    assert rel_err(g.host(dw), O.conv2d_backward(dy, second, wt, False, stride, pad)[1]) < TF32_TOL


def test_tape_keeps_the_packed_input_as_long_as_the_result():
    import gpu_util as g
    import mytorch_b200.nn.functional as F
    from mytorch_b200.backends.cuda.env import CudaEnv

    rng = np.random.default_rng(1)
    x, w = g.dev(rng.standard_normal((4, 3, 64, 64)).astype(np.float32)), g.dev(rng.standard_normal((32, 3, 3, 3)).astype(np.float32), True)
    F.conv2d(x, w, None, 1, 1)
    in_use = CudaEnv.instance().lib.pool_in_use_bytes
    gc.collect()
    before = in_use()
    y = F.conv2d(x, w, None, 1, 1)
    during = in_use()
    del y  # a result that is never differentiated, as in a validation pass with trainable weights
    gc.collect()
    assert during - before >= 2 * 4 * 32 * 64 * 64 * 4 and in_use() == before
    y = F.conv2d(x, w, None, 1, 1)
    y.sum().backward()
    want = O.conv2d_backward(np.ones(y.shape, np.float32), g.host(x), g.host(w.detach()), False, (1, 1), (1, 1))[1]
    assert rel_err(g.host(w.grad), want) < TF32_TOL
