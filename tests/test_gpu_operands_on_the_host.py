"""An operand that lies on the host is refused, also where the operator could do without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_optional_operands_on_the_host_are_refused():
    import gpu_util as g
    import mytorch_b200 as mt

    rng = np.random.default_rng(0)
    arr = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, w = g.dev(arr(2, 8, 6, 6)), g.dev(arr(8, 8, 3, 3))
    on_host, vector = mt.tensor(arr(8)), g.dev(np.ones(8, np.float32))
    conv, norm, fused = g.op("conv2d"), g.op("batch_norm2d"), g.op("conv2d_batch_norm")
    with pytest.raises(TypeError):
        conv(x, w, on_host, (1, 1), (1, 1))
    for training in (True, False):
        with pytest.raises(TypeError):
            norm(x, vector, vector, 1e-5, training, 0.1, on_host, vector)
        with pytest.raises(TypeError):
            norm(x, vector, on_host, 1e-5, training, 0.1, vector, vector)
    with pytest.raises(TypeError):
        fused(x, w, None, (1, 1), (1, 1), vector, on_host, vector, vector, 1e-5, False)
    conv(x, w, vector, (1, 1), (1, 1))
    norm(x, None, None, 1e-5, True, 0.1, None, None)
