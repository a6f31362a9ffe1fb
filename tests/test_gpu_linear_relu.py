"""Linear + ReLU in one launch: the bits of the two operators, forward and backward, on every kernel that stores a dense product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _separate(net, x):
    for layer in net._modules.values():
        x = layer(x)
    return x


@pytest.mark.parametrize("m,fin,fout,bias", [(1, 288, 128, True), (64, 288, 128, True), (1000, 90, 500, True), (1000, 500, 500, False), (40, 64, 3, True),
                                             (33, 36, 70, True), (300, 300, 301, True), (2000, 160, 260, True), (5, 7, 9, True), (64, 9216, 128, True)])
def test_sequential_runs_the_pair_as_one(m, fin, fout, bias):
    import gpu_util as g
    import mytorch_b200 as mt
    import mytorch_b200.nn as nn

    rng = np.random.default_rng(m + fin + fout)
    net = nn.Sequential(nn.Linear(fin, fout, bias=bias), nn.ReLU())
    net.to(g.DEV)
    x = rng.standard_normal((m, fin)).astype(np.float32)
    x[m // 2] = 0  # with a zero bias the products here are exactly zero, and the gradient passes
    if bias:
        net._modules["0"].bias.copy_(g.dev(np.where(np.arange(fout) % 3 == 0, 0, rng.standard_normal(fout)).astype(np.float32)))
    results = []
    for run in (net, lambda t: _separate(net, t)):
        for p in net.parameters():
            p.grad = None
        xt = g.dev(x, True)
        y = run(xt)
        (y * y).sum().backward()
        results.append([g.host(t) for t in (y, xt.grad, *(p.grad for p in net.parameters()))])
    assert all(np.array_equal(a, b) for a, b in zip(*results))
    with mt.no_grad():
        assert np.array_equal(g.host(net(g.dev(x))), results[1][0])


def test_layers_with_another_forward_stay_apart():
    import gpu_util as g
    import mytorch_b200.nn as nn

    class Doubled(nn.Linear):
        def forward(self, x):
            return super().forward(x) * 2.0

    net = nn.Sequential(Doubled(8, 6), nn.ReLU())
    net.to(g.DEV)
    x = g.dev(np.random.default_rng(0).standard_normal((4, 8)).astype(np.float32))
    assert np.array_equal(g.host(net(x)), g.host(_separate(net, x)))
