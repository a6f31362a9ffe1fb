"""Tape-based reverse-mode differentiation.

Observable behaviour follows the reference's ``mytorch/autograd.py``: operators call
``add_node(name, input_args, output_tensors, helper_tensors)`` (``:33-54``); ``backward``
(``:120-179``) accepts only a one-element tensor, seeds its gradient with 1, calls each
operator's registered backward as ``f(*output_grads, *helpers, *input_args)``, zips the returned
list with ``input_args`` and accumulates into every input that requires a gradient (first
contribution assigned, later ones added), then forgets the visited graph — a second
``backward`` through the same graph raises "Make sure you don't backward a tensor twice".
``no_grad()`` (``:181-196``) is re-entrant.

The implementation differs: every node carries a creation sequence number, so the nodes
upstream of the loss sorted by descending sequence are already a valid reverse topological
order — no degree counting, no dictionary keyed by tensors.
"""
from __future__ import annotations

import operator


class _Node:
    __slots__ = ("name", "inputs", "outputs", "helpers", "seq", "keywords")

    def __init__(self, name, inputs, outputs, helpers, seq):
        self.name = name
        self.inputs = inputs
        self.outputs = outputs
        self.helpers = helpers
        self.seq = seq
        self.keywords = None  # more for the backward function, by name: what forward made and backward can use again


_creation = operator.attrgetter("seq")


class DAGTracker:
    _instance = None

    @classmethod
    def instance(cls):
        if cls._instance is None:
            cls._instance = cls()
        return cls._instance

    def __init__(self):
        self._backward_funcs = {}
        self._seq = 0
        self.no_grad = False
        # optional callback(tensor): a leaf tensor has received its last gradient contribution of
        # the running backward pass (used to start gradient all-reduces while backward continues)
        self.leaf_grad_final_hook = None
        # optional callback(): a backend that ran gradient kernels beside the main chain (weight gradients
        # on a second CUDA stream) makes them visible to it; called before a gradient is read or handed
        # out during the pass, and when the pass ends
        self.join_hook = None
        # operators whose backward may be told ``defer_weight_gradient=True``: the returned parameter
        # gradient then becomes valid at the next join_hook() call, not when the backward returns
        self.deferrable = set()
        # operator name -> index of the input whose already accumulated gradient the operator's
        # backward can add itself (keyword ``accumulate_dx``); the tape then stores the returned
        # gradient instead of launching an add
        self.fused_accumulate = {}
        # those of them that may return the handed-in tensor itself, with their share added in place.  They return
        # dx in memory of its own otherwise, and are told ``accumulate_shared=True`` where the gradient so far may
        # also be another tensor's (an addition passes one tensor to both operands) or was there before the pass
        self.accumulates_in_place = set()

    def register_backward_function(self, op_name):
        def decorator(func):
            self._backward_funcs[op_name] = func
            return func

        return decorator

    def add_node(self, name, input_args, output_tensors, helper_tensors=None):
        self._seq += 1
        node = _Node(name, tuple(input_args), tuple(output_tensors), tuple(helper_tensors) if helper_tensors else (), self._seq)
        for t in output_tensors:
            t._grad_node = node

    def _upstream(self, root):
        from mytorch_b200.tensor import Tensor

        seen, stack = {root}, [root]
        while stack:
            for arg in stack.pop().inputs:
                if isinstance(arg, Tensor):
                    node = arg._grad_node
                    if node is not None and node not in seen:
                        seen.add(node)
                        stack.append(node)
        return sorted(seen, key=_creation, reverse=True)

    def backward(self, tensor):
        from mytorch_b200.tensor import MismatchShapesError, Tensor, shape_size

        if tensor._grad_node is None:
            raise RuntimeError("Make sure you don't backward a tensor twice")
        if shape_size(tensor.shape) != 1:
            raise RuntimeError("Backward tensor must be a scalar")
        order = self._upstream(tensor._grad_node)
        seed = Tensor(shape=tensor.shape, dtype=tensor.dtype, device=tensor.device)
        seed.fill_(1)
        tensor.grad = seed

        hook, join = self.leaf_grad_final_hook, self.join_hook
        pending = {}
        if hook is not None:  # how many contributions every leaf will receive
            for node in order:
                for arg in node.inputs:
                    if isinstance(arg, Tensor) and arg.requires_grad and arg._grad_node is None:
                        pending[id(arg)] = pending.get(id(arg), 0) + 1

        funcs, fusable, deferrable, in_place = self._backward_funcs, self.fused_accumulate, self.deferrable, self.accumulates_in_place
        owned = set()  # ids of the tensors whose gradient was made in this pass, for them alone
        for node in order:
            name, inputs = node.name, node.inputs
            fused = None  # the input whose gradient so far is handed to the operator
            slot = -1
            if name in fusable or name in deferrable or node.keywords:
                extra = dict(node.keywords) if node.keywords else {}
                slot = fusable.get(name, -1)
                if slot >= 0:
                    cand = inputs[slot]
                    if isinstance(cand, Tensor) and cand.requires_grad and cand.grad is not None:
                        fused = cand
                        extra["accumulate_dx"] = cand.grad
                        if name in in_place and id(cand) not in owned:
                            extra["accumulate_shared"] = True
                if join is not None and name in deferrable:
                    extra["defer_weight_gradient"] = True
                grads = funcs[name](*[t.grad for t in node.outputs], *node.helpers, *inputs, **extra)
            else:
                grads = funcs[name](*[t.grad for t in node.outputs], *node.helpers, *inputs)
            for k, grad in enumerate(grads):  # operators may return fewer gradients than they have inputs
                if grad is None:
                    continue
                arg = inputs[k]
                if not isinstance(arg, Tensor) or not arg.requires_grad:
                    continue
                if arg.grad is None or (k == slot and arg is fused):
                    arg.grad = grad
                    if k == slot and name in in_place:
                        owned.add(id(arg))
                else:
                    if arg.grad.shape != grad.shape:
                        raise MismatchShapesError([arg.grad.shape, grad.shape])
                    if join is not None and arg._grad_node is None:  # a leaf: its gradient may come from there
                        join()
                    arg.grad = arg.grad + grad
                    owned.add(id(arg))
            if hook is not None:
                for arg in inputs:
                    if isinstance(arg, Tensor) and arg.requires_grad and id(arg) in pending:
                        pending[id(arg)] -= 1
                        if pending[id(arg)] == 0 and arg.grad is not None:
                            hook(arg)  # the gradient may still be in flight on the backend's side stream: the hook orders itself after it

        if join is not None:
            join()

        for node in order:
            for t in node.outputs:
                t._grad_node = None
            node.inputs = node.outputs = node.helpers = ()
            node.keywords = None


class NoGrad:
    _depth = 0

    def __enter__(self):
        NoGrad._depth += 1
        DAGTracker.instance().no_grad = True

    def __exit__(self, exc_type, exc_value, traceback):
        NoGrad._depth -= 1
        if NoGrad._depth == 0:
            DAGTracker.instance().no_grad = False


def no_grad():
    return NoGrad()
