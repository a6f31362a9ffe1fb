"""Column sums around the row count where one launch takes over from two, and at the edges of its 8-column blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 7, 8, 10, 128, 132, 2052])
@pytest.mark.parametrize("rows", [1, 31, 33, 64, 1000, 1024, 1025])
def test_column_sums(rows, cols):
    from mytorch_b200.backends.cuda.env import CudaEnv
    from mytorch_b200.tensor import Tensor, tensor

    rng = np.random.default_rng(rows * 4099 + cols)
    a = rng.standard_normal((rows, cols)).astype(np.float32)
    at = tensor(a, device="cuda:0")
    out = Tensor(cpu_array=np.zeros(cols, np.float32), device="cuda:0")
    env = CudaEnv.instance()
    ws, ws_bytes = env.workspace(env.lib.colsum_workspace_bytes(cols))
    env.lib.colsum_f32(at, rows, cols, 0.5, out, ws, ws_bytes, env.stream())
    exact = a.astype(np.float64).sum(0) * 0.5
    bound = (rows + 1) * 2.0 ** -24 * np.abs(a).astype(np.float64).sum(0) * 0.5  # rows - 1 additions and a scaling, each rounded once
    assert (np.abs(out.to("cpu").numpy() - exact) <= bound).all()


@pytest.mark.parametrize("m,n,k", [(32, 8, 32), (33, 10, 516), (64, 32, 4000), (63, 33, 128), (64, 130, 132), (64, 4736, 96), (64, 4737, 96), (65, 40, 128)])
def test_product_of_few_rows(m, n, k):
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv

    env = CudaEnv.instance()
    rng = np.random.default_rng(m + n + k)
    a, b, bias = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (n, k), (n,)))
    c = g.dev(np.full((m, n), 9.0, np.float32))
    env.lib.gemm_f32(m, n, k, g.dev(a), 0, g.dev(b), 1, g.dev(bias), 1, c, env.stream())
    exact = a.astype(np.float64) @ b.T.astype(np.float64) + bias
    # TF32 operands (10 fraction bits, at worst truncated: 2^-10 each) and K additions in FP32
    bound = (2 * 2.0 ** -10 + 2.0 ** -20 + (k + 1) * 2.0 ** -23) * (np.abs(a).astype(np.float64) @ np.abs(b.T) + np.abs(bias))
    assert (np.abs(g.host(c) - np.maximum(exact, 0)) <= bound).all()
