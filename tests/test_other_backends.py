"""A backend registered by someone else is called with the arguments its operators are documented with."""
import numpy as np
import pytest

import mytorch_b200 as mt


@pytest.mark.parametrize("name,extra", [("add", (2.0,)), ("sub", (1.0,)), ("mul", ()), ("div", ()), ("pow", ())])
def test_backward_of_binary_operators(monkeypatch, name, extra):
    from mytorch_b200.backends.backend_dispatcher import BackendDispatcher
    from mytorch_b200.ops import broadcast_binary_ops as B

    table, seen = BackendDispatcher.instance()._impls["cpu"], []

    def backward(output_grad, x, y, *rest):
        seen.append(rest)
        return mt.tensor(np.full(3, 5, np.float32)), mt.tensor(np.full(3, 7, np.float32))

    # the result has one element, so that backward may start from it
    monkeypatch.setitem(table, name, lambda x, y, *rest: mt.tensor(np.ones(1, np.float32)))
    monkeypatch.setitem(table, name + "_backward", backward)
    x, constant = mt.tensor(np.ones(3, np.float32), requires_grad=True), mt.tensor(np.ones(3, np.float32))
    getattr(B, name)(x, constant, *extra).backward()
    assert seen == [extra] and x.grad._cpu_array.tolist() == [5, 5, 5] and constant.grad is None
