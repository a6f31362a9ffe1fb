"""The kernel a convolution runs on, and so the bits of its result, follow from the call alone: scratch of just the size that
``conv2d_workspace_bytes`` asks for and scratch that an earlier call has left larger give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LARGE = 128 << 20


@pytest.mark.parametrize("n,cin,h,cout,k,pad,off", [
    (3, 32, 18, 1216, 5, 2, 0), (3, 32, 16, 512, 5, 2, 0), (1, 96, 17, 1152, 7, 3, 0),  # channels of the TF32 kernels, too small for them
    (32, 64, 56, 64, 3, 1, 1),      # the same channels, the tensors one float off 16 bytes
    (8, 48, 37, 82, 3, 1, 0), (8, 48, 37, 82, 3, 1, 1)])  # channel counts of the two-term products
def test_more_scratch_than_asked_for_changes_no_bit(n, cin, h, cout, k, pad, off):
    import gpu_util as g
    from mytorch_b200.backends.cuda.env import CudaEnv, CudaMemory

    rng = np.random.default_rng(cin + cout)
    env = CudaEnv.instance()
    oh = h + 2 * pad - k + 1
    args = (n, cin, h, h, k, k, 1, 1, pad, pad, cout)
    need = env.lib.conv2d_workspace_bytes(*args)
    assert 0 < need < LARGE
    block = CudaMemory(0, LARGE)
    x, wt, dy = (g.dev(np.concatenate([np.zeros(off), rng.standard_normal(size)]).astype(np.float32))
                 for size in (n * h * h * cin, cout * k * k * cin, n * oh * oh * cout))
    xp, wp, dyp = (t._native_array.ptr + 4 * off for t in (x, wt, dy))

    def run(nbytes):
        y, dx, dw = (g.dev(np.zeros(size + off, np.float32)) for size in (n * oh * oh * cout, n * h * h * cin, cout * k * k * cin))
        env.lib.conv2d_forward_f32(*args, xp, wp, None, y._native_array.ptr + 4 * off, 0, block.ptr, nbytes, env.stream())
        env.lib.conv2d_dgrad_f32(*args, dyp, wp, dx._native_array.ptr + 4 * off, block.ptr, nbytes, env.stream())
        env.lib.conv2d_wgrad_f32(*args, xp, dyp, dw._native_array.ptr + 4 * off, block.ptr, nbytes, env.stream())
        return [g.host(t) for t in (y, dx, dw)]

    for got, want, what in zip(run(LARGE), run(need), ("forward", "data gradient", "weight gradient")):
        assert np.array_equal(got, want), what


@pytest.mark.parametrize("n,cin,h,cout,k,pad,which", [
    (40000, 24, 1, 130, 3, 1, 0),   # 9 x 24 terms, of which 24 are not padding
    (20000, 100, 2, 12, 5, 2, 1),   # 25 x 12 and 48
    (1, 1500, 6, 470, 7, 3, 2)])    # sums over 36 pixels
def test_short_sums_stay_in_fp32(n, cin, h, cout, k, pad, which, monkeypatch):
    """Sums of fewer than 96 terms round less in FP32 than the operands of the two-term products do."""
    import gpu_util as g

    rng = np.random.default_rng(which)
    x, wt, dy = (rng.standard_normal(shape).astype(np.float32) for shape in ((n, cin, h, h), (cout, cin, k, k), (n, cout, h, h)))

    def run():
        xt, wtt = g.dev(x, True), g.dev(wt, True)
        if which == 0:
            return g.host(g.op("conv2d")(xt, wtt, None, (1, 1), (pad, pad)))
        return g.host(g.op("conv2d_backward")(g.dev(dy), xt, wtt, None, (1, 1), (pad, pad))[which - 1])

    got = run()
    monkeypatch.setenv("MTB_DISABLE_TC_SPLIT", "1")
    assert np.array_equal(got, run())
