"""The work that users of this package have it do, as cases that can be timed one by one.

Whole models of ``mytorch_b200.examples`` (training steps issued operator by operator and as a
captured graph, inference), an MLP regression written with the tensor operators, and the operators
of the registry that an embedding front-end calls directly (convolution, BatchNorm - ReLU - max-pool).
All storage is float32 (convolutions and matrix products may use TF32 arithmetic), labels are int64.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` builds what a
program holds before the call, ``run`` is one pass, ``work`` the bytes and operations that a pass
cannot do without, ``tolerance`` what two correct implementations may differ by.
"""
import math

import numpy as np
import torch

import mytorch_b200 as mt
import mytorch_b200.nn as nn
import mytorch_b200.nn.functional as F
from mytorch_b200.backends.backend_dispatcher import BackendDispatcher
from mytorch_b200.backends.cuda.env import CudaMemory, CudaMemoryView
from mytorch_b200.cuda_graph import StepGraph
from mytorch_b200.examples.mnist import CNN as MnistCNN
from mytorch_b200.examples.models import ResNet18Cifar, ResNet50, small_cnn
from mytorch_b200.optim import SGD
from mytorch_b200.parallel import GradBucket, torch_view

DEVICE = "cuda:0"


# ------------------------------------------------------------------------------ which cases

def listed():
    return [
        # answering one request: the example's digit classifier on a single image; launches and host time are all there is
        {"name": "mnist_infer_b1", "path": "mnist", "mode": "infer", "batch": 1},
        # the loop of examples/mnist.py: its CNN, batches of 64, plain SGD, operators issued one by one
        {"name": "mnist_train_b64", "path": "mnist", "mode": "train", "batch": 64},
        # the small two-convolution CNN's training step at its configured batch, replayed as a graph
        {"name": "small_cnn_graph_b64", "path": "small_cnn", "mode": "graph", "batch": 64},
        # regression with an MLP whose sizes are no multiples of anything: matrix products, broadcasts, powers, means
        {"name": "mlp_train_b1000", "path": "mlp", "batch": 1000, "fin": 90, "hidden": 500, "fout": 1},
        # evaluating a trained CIFAR ResNet-18 in batches that do not divide evenly
        {"name": "resnet18_infer_b100", "path": "resnet18", "mode": "infer", "batch": 100},
        # training it interactively: every operator issued by the host
        {"name": "resnet18_train_b128", "path": "resnet18", "mode": "train", "batch": 128},
        # one rank's share of a global batch of 512 on 8 GPUs, replayed as a graph
        {"name": "resnet18_graph_b64", "path": "resnet18", "mode": "graph", "batch": 64},
        # the benchmark's training step on one GPU
        {"name": "resnet18_graph_b512", "path": "resnet18", "mode": "graph", "batch": 512},
        # ImageNet-shaped training: the largest step of the configurations
        {"name": "resnet50_train_b128", "path": "resnet50", "mode": "train", "batch": 128, "size": 224},
        # the single-convolution configuration, forward and both gradients
        {"name": "conv64_56x56_n128", "path": "conv", "n": 128, "cin": 64, "cout": 64, "hw": 56, "k": 3, "stride": 1, "pad": 1},
        # a convolution whose channel counts and image fit no tile
        {"name": "conv_ragged_n32", "path": "conv", "n": 32, "cin": 48, "cout": 82, "hw": 37, "k": 3, "stride": 1, "pad": 1},
        # the bandwidth block: BatchNorm (training) - ReLU - 2x2 max-pool, forward and backward
        {"name": "bn_relu_pool_n256", "path": "bn_relu_pool", "n": 256, "c": 128, "hw": 56},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mnist", "small_cnn", "mlp", "resnet18", "resnet18", "resnet50", "conv", "conv", "bn_relu_pool"])
    if kind == "mnist":
        return {"path": "mnist", "mode": rng.choice(["infer", "train"]), "batch": _log_int(rng, 1, 1024)}
    if kind == "small_cnn":
        return {"path": "small_cnn", "mode": rng.choice(["graph", "train"]), "batch": _log_int(rng, 8, 1024)}
    if kind == "mlp":
        return {"path": "mlp", "batch": _log_int(rng, 16, 8192), "fin": _log_int(rng, 8, 2048), "hidden": _log_int(rng, 16, 2048),
                "fout": _log_int(rng, 1, 1000)}
    if kind == "resnet18":
        return {"path": "resnet18", "mode": rng.choice(["infer", "train", "graph"]), "batch": _log_int(rng, 16, 512)}
    if kind == "resnet50":
        return {"path": "resnet50", "mode": "train", "batch": _log_int(rng, 8, 96), "size": rng.choice([160, 192, 224])}
    if kind == "bn_relu_pool":
        return {"path": "bn_relu_pool", "n": _log_int(rng, 4, 256), "c": _log_int(rng, 16, 256), "hw": rng.randint(14, 56)}
    while True:
        case = {"path": "conv", "n": _log_int(rng, 1, 256), "cin": _log_int(rng, 3, 512), "cout": _log_int(rng, 8, 512), "hw": rng.randint(7, 80),
                "k": rng.choice([1, 3, 3, 5]), "stride": rng.choice([1, 1, 2]), "pad": 0}
        if rng.random() < 0.5:  # channel counts that networks use beside arbitrary ones
            case["cin"], case["cout"] = (max(16, c // 32 * 32) for c in (case["cin"], case["cout"]))
        case["pad"] = case["k"] // 2 if rng.random() < 0.8 else 0
        pixels = case["n"] * case["hw"] ** 2
        if work(case)["flops"] <= 6e10 and pixels * max(case["cin"], case["cout"]) <= 1 << 27:
            return case


# ------------------------------------------------------------------------------ what a program holds

def _op(name):
    return BackendDispatcher.instance().dispatch("cuda", name)


def _dev(array, requires_grad=False):
    return mt.tensor(array, device=DEVICE, requires_grad=requires_grad)


def _group(name, t):
    """Tensors of like magnitude are kept together: the convolution / linear weights of a stage, its vectors."""
    return name.split(".")[0] + (".weights" if len(t.shape) > 1 else ".vectors")


def _side_by_side(named):
    """Lays tensors out in one block per group, so that a model of hundreds is handed over whole: {group: PyTorch view of the block}."""
    groups, views = {}, {}
    for name, t in named:
        groups.setdefault(_group(name, t), []).append(t)
    for key, tensors in groups.items():
        places = GradBucket(tensors)
        block = CudaMemory(0, 4 * places.total)
        view = views[key] = torch_view(block, places.total)
        view._block = block  # the view does not own the memory
        view.zero_()
        torch.cuda.synchronize()
        for t, off in zip(tensors, places.offsets):
            window = CudaMemoryView(block, 4 * off, t._native_array.nbytes, 0)
            window.copy_from(t._native_array, window.nbytes)
            t._native_array = window
    return views


class _Views:
    """PyTorch views of tensors of this package, remembered by address (the pool hands the same blocks out again)."""

    def __init__(self):
        self.known, self.held = {}, None

    def __call__(self, tensors):
        self.held = tensors  # the memory stays with these until the next pass
        out = []
        for t in tensors:
            key = (t._native_array.ptr, t.shape)
            v = self.known.get(key)
            if v is None:
                v = self.known[key] = torch_view(t._native_array, math.prod(t.shape))
            out.append(v)
        return out


class _Captured:
    """A captured step that gives its memory back when the program drops it."""

    def __init__(self, step):
        self.graph = StepGraph(step)
        self.result = self.graph.capture()

    def replay(self):
        self.graph.replay()

    def __del__(self):
        self.graph.destroy()


def _trained(net, rng):
    """BatchNorm parameters and running statistics as training leaves them, not as initialisation sets them: residual
    branches, which training starts near zero, still weak."""
    for name, m in net.named_modules():
        if isinstance(m, nn.BatchNorm2d):
            c = m.num_features
            closing = name.endswith("bn3" if isinstance(net, ResNet50) else "bn2")
            for t, a in ((m.weight, rng.uniform(0.1, 0.3, c) if closing else rng.uniform(0.5, 1.5, c)), (m.bias, rng.normal(0, 0.1, c)),
                         (m.running_mean, rng.normal(0, 0.1, c)), (m.running_var, rng.uniform(0.5, 1.5, c))):
                t.copy_(_dev(a.astype(np.float32)))


_MODELS = {"mnist": (MnistCNN, 1, 28, 10), "small_cnn": (small_cnn, 1, 28, 10), "resnet18": (ResNet18Cifar, 3, 32, 10),
           "resnet50": (ResNet50, 3, 224, 1000)}
# the example's rate for the example; the deep networks at the rate of their warm-up
_SGD = {"mnist": {"lr": 0.1}, "small_cnn": {"lr": 0.01, "momentum": 0.9}, "resnet18": {"lr": 0.01, "momentum": 0.9},
        "resnet50": {"lr": 0.01, "momentum": 0.9}}


def _prepare_model(case, seed):
    rng = np.random.default_rng(seed)
    make, channels, size, classes = _MODELS[case["path"]]
    size = case.get("size", size)
    mt.manual_seed(seed)
    net = make()
    net.to(DEVICE)
    x = _dev(rng.standard_normal((case["batch"], channels, size, size), dtype=np.float32))
    state = {"case": case, "net": net, "x": x, "views": _Views()}
    deep = case["path"] in ("resnet18", "resnet50")
    if deep or case["mode"] == "infer":
        _trained(net, rng)
    if case["mode"] == "infer":
        net.eval()
        return state
    named = list(net.named_parameters())
    state.update(target=_dev(rng.integers(0, classes, case["batch"]).astype(np.int64)), opt=SGD(net.parameters(), **_SGD[case["path"]]))
    if deep:
        # Behind dozens of ReLU masks a change of one bit anywhere moves a gradient by percents (tests/test_oracle_conditioning.py),
        # so two correct implementations cannot be compared by it: it shows in what it is for, the updated parameters.
        state.update(grads_of=[], updated={"parameters": _side_by_side(named), "buffers": _side_by_side(net.named_buffers())})
    else:
        # a convolution's bias in front of a BatchNorm has no gradient but rounding
        kept = [p for name, p in named if not (case["path"] == "mnist" and name.startswith("layer1") and name.endswith("bias") and
                                               name.split(".")[1] in ("0", "4", "8"))]
        state.update(grads_of=kept, updated={name: torch_view(t._native_array, math.prod(t.shape)) for name, t in named + list(net.named_buffers())})
    if case["mode"] == "graph":
        # the optimizer's first step sets its momentum buffers and cannot be replayed: it runs before the capture
        _training_step(state)
        captured = dict(state)  # without the graph itself: the program that drops its state drops the graph at once
        state["graph"] = _Captured(lambda: _training_step(captured))
        state["result"] = _training_outputs(state, *state["graph"].result)
    return state


def _training_step(state):
    logits = state["net"](state["x"])
    loss = F.cross_entropy(logits, state["target"])
    state["opt"].zero_grad()
    loss.backward()
    state["opt"].step()
    return loss, logits


def _training_outputs(state, loss, logits):
    return {"results": state["views"]([loss, logits] + [p.grad for p in state["grads_of"]]), "updated": state["updated"]}


def _prepare_mlp(case, seed):
    rng = np.random.default_rng(seed)
    mt.manual_seed(seed)
    net = nn.Sequential(nn.Linear(case["fin"], case["hidden"]), nn.ReLU(), nn.Linear(case["hidden"], case["hidden"]), nn.ReLU(),
                        nn.Linear(case["hidden"], case["fout"]))
    net.to(DEVICE)
    x = _dev(rng.standard_normal((case["batch"], case["fin"]), dtype=np.float32))
    t = _dev(rng.standard_normal((case["batch"], case["fout"]), dtype=np.float32))
    params = list(net.parameters())
    return {"case": case, "net": net, "x": x, "t": t, "opt": SGD(params, lr=0.01, momentum=0.9), "params": params, "views": _Views(),
            "updated": [torch_view(p._native_array, math.prod(p.shape)) for p in params]}


def _prepare_conv(case, seed):
    rng = np.random.default_rng(seed)
    n, cin, cout, hw, k = (case[key] for key in ("n", "cin", "cout", "hw", "k"))
    out = _conv_out(case)
    bound = 1 / math.sqrt(cin * k * k)
    return {"case": case, "views": _Views(), "x": _dev(rng.standard_normal((n, cin, hw, hw), dtype=np.float32), True),
            "w": _dev(rng.uniform(-bound, bound, (cout, cin, k, k)).astype(np.float32), True),
            "b": _dev(rng.uniform(-bound, bound, cout).astype(np.float32), True),
            "dy": _dev(rng.standard_normal((n, cout, out, out), dtype=np.float32))}


def _prepare_bn_relu_pool(case, seed):
    rng = np.random.default_rng(seed)
    n, c, hw = case["n"], case["c"], case["hw"]
    x = rng.standard_normal((n, c, hw, hw), dtype=np.float32)
    x *= 2.0
    x += 0.5
    running = [_dev(np.zeros(c, np.float32)), _dev(np.ones(c, np.float32))]
    return {"case": case, "views": _Views(), "x": _dev(x, True), "dy": _dev(rng.standard_normal((n, c, hw // 2, hw // 2), dtype=np.float32)),
            "gamma": _dev(rng.uniform(0.5, 1.5, c).astype(np.float32), True), "beta": _dev(rng.normal(0, 0.1, c).astype(np.float32), True),
            "running": running, "updated": [torch_view(t._native_array, c) for t in running]}


def prepare(case, seed):
    return {"mlp": _prepare_mlp, "conv": _prepare_conv, "bn_relu_pool": _prepare_bn_relu_pool}.get(case["path"], _prepare_model)(case, seed)


# ------------------------------------------------------------------------------ one pass

def _run_mlp(s):
    prediction = s["net"](s["x"])
    loss = ((prediction - s["t"]) ** 2).mean()
    s["opt"].zero_grad()
    loss.backward()
    s["opt"].step()
    return s["views"]([loss, prediction] + [p.grad for p in s["params"]]) + s["updated"]


def _run_conv(s):
    stride, pad = (s["case"]["stride"],) * 2, (s["case"]["pad"],) * 2
    y = _op("conv2d")(s["x"], s["w"], s["b"], stride, pad)
    dx, dw, db = _op("conv2d_backward")(s["dy"], s["x"], s["w"], s["b"], stride, pad)
    return s["views"]([y, dx, dw, db])


def _run_bn_relu_pool(s):
    x, gamma, beta = s["x"], s["gamma"], s["beta"]
    normal, mean, var = _op("batch_norm2d")(x, gamma, beta, 1e-5, True, 0.1, *s["running"])
    active = _op("relu")(normal)
    y = _op("max_pool2d")(active, (2, 2), (2, 2), (0, 0))
    d_active, = _op("max_pool2d_backward")(s["dy"], y, active, (2, 2), (2, 2), (0, 0))
    d_normal, = _op("relu_backward")(d_active, normal)
    dx, d_gamma, d_beta = _op("batch_norm2d_backward")(d_normal, mean, var, x, gamma, beta, 1e-5)
    return s["views"]([y, mean, var, dx, d_gamma, d_beta]) + s["updated"]


def run(state):
    case = state["case"]
    if case["path"] == "mlp":
        return _run_mlp(state)
    if case["path"] == "conv":
        return _run_conv(state)
    if case["path"] == "bn_relu_pool":
        return _run_bn_relu_pool(state)
    if case["mode"] == "infer":
        with mt.no_grad():
            return state["views"]([state["net"](state["x"])])
    if case["mode"] == "graph":
        state["graph"].replay()
        return state["result"]
    return _training_outputs(state, *_training_step(state))


# ------------------------------------------------------------------------------ what a pass needs

def _conv_out(case):
    return (case["hw"] + 2 * case["pad"] - case["k"]) // case["stride"] + 1


def _layers(path, size):
    """Multiply-adds per image, parameters and BatchNorm channels of a model's forward pass."""
    macs, params, bn = [], [], []

    def conv(cin, cout, k, out, bias=False, norm=True):
        macs.append(cin * cout * k * k * out * out)
        params.append(cin * cout * k * k + (cout if bias else 0) + (2 * cout if norm else 0))
        bn.append(cout if norm else 0)

    def linear(fin, fout):
        macs.append(fin * fout)
        params.append(fin * fout + fout)

    if path == "mnist":
        conv(1, 32, 3, 28, True), conv(32, 128, 3, 14, True), conv(128, 32, 3, 7, True)
        linear(288, 128), linear(128, 10)
    elif path == "small_cnn":
        conv(1, 32, 3, 26, True, False), conv(32, 64, 3, 24, True, False)
        linear(9216, 128), linear(128, 10)
    elif path == "resnet18":
        conv(3, 64, 3, 32)
        cin, hw = 64, 32
        for stage, width in enumerate((64, 128, 256, 512)):
            for block in range(2):
                hw = hw // 2 if stage and not block else hw
                conv(cin, width, 3, hw), conv(width, width, 3, hw)
                if cin != width:
                    conv(cin, width, 1, hw)
                cin = width
        linear(512, 10)
    else:
        hw = (size - 1) // 2 + 1
        conv(3, 64, 7, hw)
        hw = (hw - 1) // 2 + 1
        cin = 64
        for stage, (mid, count) in enumerate(zip((64, 128, 256, 512), (3, 4, 6, 3))):
            for block in range(count):
                conv(cin, mid, 1, hw)
                hw = (hw - 1) // 2 + 1 if stage and not block else hw
                conv(mid, mid, 3, hw), conv(mid, 4 * mid, 1, hw)
                if not block:
                    conv(cin, 4 * mid, 1, hw)
                cin = 4 * mid
        linear(2048, 1000)
    return sum(macs), macs[0], sum(params), sum(bn)


def work(case):
    path = case["path"]
    if path == "conv":
        out = _conv_out(case)
        x, y = case["n"] * case["cin"] * case["hw"] ** 2, case["n"] * case["cout"] * out ** 2
        w = case["cin"] * case["cout"] * case["k"] ** 2 + case["cout"]
        return {"bytes": 4 * (2 * x + 2 * y + 2 * w), "flops": 6 * case["n"] * out ** 2 * case["cout"] * case["cin"] * case["k"] ** 2}
    if path == "bn_relu_pool":
        x = case["n"] * case["c"] * case["hw"] ** 2
        y = case["n"] * case["c"] * (case["hw"] // 2) ** 2
        return {"bytes": 4 * (2 * x + 2 * y + 10 * case["c"]), "flops": 20 * x}
    if path == "mlp":
        b, fin, hidden, fout = (case[k] for k in ("batch", "fin", "hidden", "fout"))
        params = fin * hidden + hidden * hidden + hidden * fout + 2 * hidden + fout
        return {"bytes": 4 * (b * (fin + 2 * fout) + 6 * params), "flops": 2 * b * (2 * fin * hidden + 3 * hidden * hidden + 3 * hidden * fout)}
    macs, first, params, channels = _layers(path, case.get("size", 224))
    _, cin, size, classes = _MODELS[path]
    batch, pixels = case["batch"], cin * case.get("size", size) ** 2
    if case["mode"] == "infer":
        return {"bytes": 4 * (batch * (pixels + classes) + params + 2 * channels), "flops": 2 * batch * macs}
    # parameters, momentum and gradients: read and written; the first layer has no data gradient
    return {"bytes": 4 * (batch * (pixels + classes) + 5 * params + 4 * channels) + 8 * batch, "flops": 2 * batch * (3 * macs - first)}


def tolerance(case):
    path = case["path"]
    if path == "bn_relu_pool":  # 32-bit arithmetic throughout
        return {"rel": 1e-4, "max": 0.5}
    if path == "conv":  # one product with operands in TF32
        return {"rel": 2e-3, "max": 0.05}
    if case.get("mode") == "infer":
        return {"rel": 5e-3}
    # several TF32 products in a row, ReLU masks that turn on the last bit, and an update that feeds the next pass
    return {"rel": 1e-2 if path in ("resnet18", "resnet50") else 2e-2, "max": 0.5}
