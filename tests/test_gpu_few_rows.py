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
