"""Two host threads on one device share its stream and its scratch: a call that hands something on from one launch to the next in
scratch gets through undisturbed by what the other thread enqueues, and both get the bits that one thread alone gets."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_that_share_scratch():
    import gpu_util as g

    rng = np.random.default_rng(0)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)

    def case(n, cin, cout, h, k):
        x, wt, b, dy = f32(n, cin, h, h), f32(cout, cin, k, k), f32(cout), f32(n, cout, h, h)
        gamma, beta = f32(cout), f32(cout)

        def run():
            s, p = (1, 1), (k // 2, k // 2)
            xt, wtt, bt = g.dev(x, True), g.dev(wt, True), g.dev(b, True)
            y = g.op("conv2d")(xt, wtt, bt, s, p)
            grads = g.op("conv2d_backward")(g.dev(dy), xt, wtt, bt, s, p)
            norm = g.op("batch_norm2d")(y, g.dev(gamma), g.dev(beta), 1e-5, True, 0.1, None, None)
            return [y, *grads, *norm]

        return run

    # two-term products twice (of different sizes), the TF32 kernels, and the CUDA cores
    cases = [case(8, 48, 82, 37, 3), case(16, 70, 50, 30, 3), case(8, 64, 64, 32, 3), case(2, 5, 7, 20, 3)]
    alone = [[g.host(t) for t in run()] for run in cases]
    wrong = []

    def worker(order):
        for _ in range(20):
            results = [(i, cases[i]()) for i in order]
            for i, tensors in results:
                if not all(np.array_equal(g.host(t), want) for t, want in zip(tensors, alone[i])):
                    wrong.append(i)

    threads = [threading.Thread(target=worker, args=(order,)) for order in ((0, 1, 2, 3), (1, 3, 0, 2))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
