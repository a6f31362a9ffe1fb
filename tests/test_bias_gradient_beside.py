"""The bias gradient on the side stream, beside the other two gradients of the same call: memory, order, switch and values."""
import types

import numpy as np
import pytest

import mytorch_b200 as mt
from conftest import rel_err
from oracle import ops as O


class _Recorder:
    """Stands in for the CUDA state: notes what is allocated and enqueued, on which stream, in order."""

    def __init__(self, overlap=True):
        self.events, self.overlap_weight_gradients = [], overlap
        self.lib = self

    def __getattr__(self, name):  # an entry point
        if name.endswith("_bytes"):
            return lambda *a: 256
        if name.endswith("in_place"):
            return lambda *a: 0
        return lambda *a: self.events.append((name, a[-1]))

    def stream(self):
        return "main"

    def workspace(self, n):
        return 16, n

    def side_workspace(self, n):
        self.events.append(("scratch", "side"))
        return 16, n

    def fork_side(self, kept):
        self.events.append(("fork", tuple(kept)))
        return "side"

    def join_side(self):
        self.events.append(("join", None))


def _backward(monkeypatch, overlap=True, cin=64, **more):
    import mytorch_b200.backends.cuda.ops as ops
    from mytorch_b200.tensor import Device, Tensor

    env, made = _Recorder(overlap), {}
    device = Device("cuda:0")

    def tensor(shape, grad=False):
        t = Tensor._on_device(tuple(shape), mt.float32, device, types.SimpleNamespace(nbytes=4 * int(np.prod(shape)), device_index=0))
        t.requires_grad = grad
        return t

    def new(shape, like, dtype=None):
        made[tuple(shape)] = t = tensor(shape)
        env.events.append(("memory", tuple(shape)))
        return t

    monkeypatch.setattr(ops, "_env", lambda t: env)
    monkeypatch.setattr(ops, "_new", new)
    monkeypatch.setattr(ops, "CudaMemory", lambda index, n: types.SimpleNamespace(nbytes=n, device_index=0))
    x, w, b, dy = tensor((4, cin, 64, 64), True), tensor((96, cin, 3, 3), True), tensor((96,), True), tensor((4, 96, 64, 64))
    monkeypatch.setattr(ops, "_BIAS_BESIDE_BYTES", dy._native_array.nbytes)
    if more.pop("accumulate", False):
        more["accumulate_dx"] = tensor(x.shape)
    out = ops.cuda_conv2d_backward(dy, x, w, b, (1, 1), (1, 1), **more)
    return env.events, out, dy


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("cin", [64, 3])
def test_memory_comes_before_the_fork(monkeypatch, cin, accumulate):
    events, (dx, dw, db), dy = _backward(monkeypatch, cin=cin, accumulate=accumulate)
    names = [e[0] for e in events]
    fork, join, colsum = names.index("fork"), names.index("join"), names.index("colsum_f32")
    assert events[fork][1] == (dy, db) and events[colsum][1] == "side" and fork < colsum < join == len(events) - 1
    assert events.index(("memory", (96,))) < fork and names.index("scratch") < fork


@pytest.mark.parametrize("more", [{"overlap": False}, {"defer_weight_gradient": True}])
def test_compute_stream_when_the_side_stream_is_off_or_taken(monkeypatch, more):
    events, (_, _, db), _ = _backward(monkeypatch, **more)
    assert [e for e in events if e[0] == "colsum_f32"] == [("colsum_f32", "main")] and db.shape == (96,)
    assert ("fork" in [e[0] for e in events]) == ("overlap" not in more)


@pytest.mark.gpu
@pytest.mark.parametrize("n,cin,cout,hw,k", [(2, 64, 64, 16, 3), (3, 48, 82, 13, 3), (2, 3, 64, 32, 3), (2, 3, 64, 32, 7), (1, 20, 7, 9, 1)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_values(monkeypatch, n, cin, cout, hw, k, accumulate):
    import gpu_util as g
    import mytorch_b200.backends.cuda.ops as ops

    rng = np.random.default_rng(cin + cout)
    x, wt = rng.standard_normal((n, cin, hw, hw)).astype(np.float32), rng.standard_normal((cout, cin, k, k)).astype(np.float32)
    dy, add = rng.standard_normal((n, cout, hw, hw)).astype(np.float32), rng.standard_normal(x.shape).astype(np.float32)
    args = g.dev(dy), g.dev(x, True), g.dev(wt, True), g.dev(np.zeros(cout, np.float32), True), (1, 1), (k // 2, k // 2)
    want = O.conv2d_backward(dy, x, wt, True, (1, 1), (k // 2, k // 2))
    extra = {"accumulate_dx": g.dev(add)} if accumulate else {}
    plain = [g.host(t) for t in ops.cuda_conv2d_backward(*args, **extra)]
    monkeypatch.setattr(ops, "_BIAS_BESIDE_BYTES", 0)
    for got, same, ref in zip(ops.cuda_conv2d_backward(*args, **extra), plain, (want[0] + add if accumulate else want[0], *want[1:])):
        assert np.array_equal(g.host(got), same) and rel_err(same, ref) < 5e-3  # TF32 operands
    assert rel_err(plain[2], want[2]) < 1e-5  # 32-bit sums of at most 2048 terms
