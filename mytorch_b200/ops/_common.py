"""Shared front-end plumbing: look up the backend function, mark the result, record the node."""
from mytorch_b200.autograd import DAGTracker
from mytorch_b200.backends.backend_dispatcher import BackendDispatcher

tracker = DAGTracker.instance()


def dispatch(device, name):
    try:
        return BackendDispatcher._instance._impls[device.type][name]
    except (AttributeError, KeyError):  # not loaded yet, or not there: the registry says which
        return BackendDispatcher.instance().dispatch(device.type, name)


def grad_enabled(*tensors):
    if tracker.no_grad:
        return False
    for t in tensors:
        if t is not None and t.requires_grad:
            return True
    return False


def record(name, inputs, output, helpers=None):
    if output.requires_grad:
        tracker.add_node(name, inputs, [output], helpers)
    return output
