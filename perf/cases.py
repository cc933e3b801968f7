"""Workloads of this framework, as a user's program drives them through its public entry points, for timing one build
against another.

Three kinds of work:

  dense / conv   one SNN_dense / SNN_conv layer on device tensors, "train" (forward, then backward on an upstream
                 gradient through autograd) or "infer" (evaluation under no_grad: spike times only)
  net            a whole network of nets.py (MNIST-, CIFAR-, ImageNet-shaped):
                   "step"   encoding, forward, loss, constraint cost, backward, Adam -- a training step on one GPU
                   "grad"   the same up to the flat gradient, which a data-parallel rank hands to the all-reduce
                   "infer"  encoding and forward under no_grad
                 launched op by op, or (graph) as the captured whole-step CUDA graph of graph.py

Layer sizes, value families and batch sizes are those of the benchmark configurations and the parity tests, and the
space around them.
"""
import math

import torch

from snntc_2023_b200 import nets, train
from snntc_2023_b200.SNN_TC_Modules import SNN_conv, SNN_dense
from snntc_2023_b200.graph import GraphedStep

NO_SPIKE = 1e5
CONSTRAINT_K, CONSTRAINT_K2 = 100.0, 1e-2   # as in the benchmark's training step
NETS = {"mlp": (nets.MNIST_MLP, (784,), 10),
        "cifar": (nets.CIFAR_CNN, (32, 32, 3), 10),
        "imagenet": (nets.IMAGENET_CNN, (224, 224, 3), 1000)}


# ------------------------------------------------------------------------------------------------- the cases
def _dense(B, I, J, mode, bias=True, family="hidden", grads=1.0):
    return dict(kind="dense", B=B, I=I, J=J, mode=mode, bias=bias, family=family, grads=grads)


def _conv(B, H, W, C, J, k, stride, padding, mode, bias=True, family="hidden", grads=1.0):
    return dict(kind="conv", B=B, H=H, W=W, C=C, J=J, k=k, stride=stride, padding=padding, mode=mode, bias=bias,
                family=family, grads=grads)


def _net(net, batch, mode, graph=False):
    return dict(kind="net", net=net, batch=batch, mode=mode, graph=graph)


def listed():
    named = [
        # one digit at a time through the MLP: nothing but call overhead and kernel latency
        ("mlp infer 1", _net("mlp", 1, "infer")),
        # the trainer's loop written op by op on small batches
        ("mlp step 32", _net("mlp", 32, "step")),
        # first benchmark configuration: one dense layer, no bias, dense random upstream gradient
        ("dense 784-400 256", _dense(256, 784, 400, "train", bias=False, family="input")),
        # second configuration: the MLP's training step as one CUDA graph
        ("mlp step graph 1024", _net("mlp", 1024, "step", graph=True)),
        # classifier head on flattened features: the weight matrix (103 MB) is larger than a batch's work
        ("dense 25088-1024 64", _dense(64, 25088, 1024, "train")),
        # one image through the CIFAR-shaped network: latency of a chain of small kernels
        ("cifar infer 1", _net("cifar", 1, "infer")),
        # a test pass: forward only, batch that divides nothing
        ("cifar infer 250", _net("cifar", 250, "infer")),
        # odd sizes off the tuned path: 5x5, stride 2, VALID, channel counts that are no multiple of 16
        ("conv 5x5s2 20-52 37", _conv(37, 45, 39, 20, 52, 5, 2, "VALID", "train", grads=0.25)),
        # third configuration: one conv layer whose every input spikes and every output has a gradient
        ("conv 3x3 64-128 128", _conv(128, 32, 32, 64, 128, 3, 1, "SAME", "train", bias=False, family="input")),
        # fine-tuning on small batches without a graph: launches and small grids
        ("cifar grad 16", _net("cifar", 16, "grad")),
        # fourth configuration: the benchmark's headline workload
        ("cifar grad graph 256", _net("cifar", 256, "grad", graph=True)),
        # fifth configuration: the largest
        ("imagenet grad graph 64", _net("imagenet", 64, "grad", graph=True)),
    ]
    return [dict(c, name=n) for n, c in named]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        what = rng.choice(["dense", "dense", "dense", "conv", "conv", "conv", "conv", "net", "net"])
        mode = rng.choice(["train", "train", "infer"])
        family = rng.choice(["hidden", "hidden", "input"])
        grads = rng.choice([1.0, 0.35, 0.12])   # no pooling behind the layer / pooling in front / pooling behind
        bias = rng.random() < 0.75
        if what == "dense":
            c = _dense(_log(rng, 1, 1024), _log(rng, 32, 25088), _log(rng, 10, 1024), mode, bias, family, grads)
        elif what == "conv":
            k, stride = rng.choice([(1, 1), (3, 1), (3, 1), (3, 1), (3, 2), (5, 1), (5, 2), (7, 2)])
            C = rng.choice([1, 3, 16, 32, 64, 128, 256, _log(rng, 2, 256)])
            J = rng.choice([16, 32, 64, 128, 256, _log(rng, 8, 256)])
            c = _conv(_log(rng, 1, 256), _log(rng, 7, 64), _log(rng, 7, 64), C, J, k, stride,
                      rng.choice(["SAME", "SAME", "VALID"]), mode, bias, family, grads)
        else:
            net = rng.choice(["mlp", "mlp", "cifar", "cifar", "imagenet"])
            batch = _log(rng, 2, {"mlp": 2048, "cifar": 256, "imagenet": 32}[net])
            mode = rng.choice(["grad", "grad", "infer"] if net != "mlp" else ["step", "step", "infer"])
            c = _net(net, batch, mode, mode != "infer" and rng.random() < 0.5)
        # at most the work of the largest listed case, and the sorted lists of a layer in a few GB
        if c["kind"] == "net" or (_layer_rij(c)[0] * _layer_rij(c)[1] < 6e8 and math.prod(_layer_rij(c)) < 3e10):
            return c


# ------------------------------------------------------------------------------------------------- inputs
def _out_size(c):
    if c["padding"] == "SAME":
        return math.ceil(c["H"] / c["stride"]), math.ceil(c["W"] / c["stride"])
    return (c["H"] - c["k"]) // c["stride"] + 1, (c["W"] - c["k"]) // c["stride"] + 1


def _layer_rij(c):
    """Rows (samples or receptive fields), fan-in with the bias row, fan-out."""
    if c["kind"] == "dense":
        return c["B"], c["I"] + int(c["bias"]), c["J"]
    Nh, Nw = _out_size(c)
    return c["B"] * Nh * Nw, c["k"] * c["k"] * c["C"] + int(c["bias"]), c["J"]


def _spikes(shape, family, g):
    """Spike times. "input": exp(U[0,1)), what the encoding of pixels gives. "hidden": exp(1.5*U[0,1)) with half of the
    entries at the no-spike value, what a layer's outputs look like."""
    t = torch.rand(shape, generator=g, device="cuda")
    if family == "input":
        return torch.exp(t)
    return torch.where(torch.rand(shape, generator=g, device="cuda") < 0.5, torch.full_like(t, NO_SPIKE), torch.exp(1.5 * t))


def _weight(fan_in, J, bias, family, g):
    """"input": N(2/I, 1/I), the single-layer configurations' family. "hidden": the layers' own initialisation,
    randn*sqrt(15/I). A zero bias row last where there is a bias."""
    w = torch.randn((fan_in, J), generator=g, device="cuda")
    w = w / math.sqrt(fan_in) + 2.0 / fan_in if family == "input" else w * math.sqrt(15.0 / fan_in)
    return torch.cat([w, torch.zeros((1, J), device="cuda")]) if bias else w


def _prepare_layer(c, g):
    if c["kind"] == "dense":
        shape, out, fan_in = (c["B"], c["I"]), (c["B"], c["J"]), c["I"]
        make, args = SNN_dense, (c["I"], c["J"])
    else:
        shape, out, fan_in = (c["B"], c["H"], c["W"], c["C"]), (c["B"],) + _out_size(c) + (c["J"],), c["k"] * c["k"] * c["C"]
        make, args = SNN_conv, (c["C"], c["J"], c["k"], c["stride"], c["padding"])
    w = _weight(fan_in, c["J"], c["bias"], c["family"], g)
    layer = make(*args, biasvolt=1.0 if c["bias"] else 0.0, weight=w).cuda()
    x = _spikes(shape, c["family"], g)
    state = dict(mode=c["mode"], layer=layer, x=x)
    if c["mode"] == "train":
        x.requires_grad_(True)
        grad = torch.randn(out, generator=g, device="cuda")
        if c["grads"] < 1.0:   # pooling and outputs that never spike leave most outputs without a gradient
            grad = grad * (torch.rand(out, generator=g, device="cuda") < c["grads"])
        state["grad"] = grad
    return state


def _prepare_net(c, g):
    specs, shape, classes = NETS[c["net"]]
    weights = []
    for s in specs:
        if s[0] in ("conv", "dense"):
            fan_in, fan_out = (s[3] * s[3] * s[1], s[2]) if s[0] == "conv" else (s[1], s[2])
            weights.append(_weight(fan_in, fan_out, True, "hidden", g))
    net = nets.SnnNet(specs, weights=weights, device="cuda")
    t = torch.rand((c["batch"],) + shape, generator=g, device="cuda")
    labels = torch.randint(0, classes, (c["batch"],), generator=g, device="cuda")
    state = dict(mode=c["mode"], net=net, t=t, labels=labels)
    if c["mode"] == "infer":
        return state
    opt = train.Adam(net.flat_param, net.flat_grad, lr=1e-5) if c["mode"] == "step" else None

    def step(t, labels):
        loss = net.loss(train.encode(t, one_minus=False), labels)
        net.backward(loss + net.constraint_cost(CONSTRAINT_K, CONSTRAINT_K2))
        if opt is not None:
            opt.step()
        return loss.detach()

    state.update(opt=opt, step=GraphedStep(step, [t, labels]) if c["graph"] else step)
    return state


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return _prepare_net(case, g) if case["kind"] == "net" else _prepare_layer(case, g)


# ------------------------------------------------------------------------------------------------- one pass
def run(state):
    mode = state["mode"]
    if "net" in state:
        if mode == "infer":
            with torch.no_grad():
                return state["net"](train.encode(state["t"], one_minus=False))
        loss = state["step"](state["t"], state["labels"])
        out = dict(loss=loss, grad=state["net"].flat_grad)
        if mode == "step":
            out["param"] = state["net"].flat_param
        return out
    if mode == "infer":
        with torch.no_grad():
            return state["layer"](state["x"])
    y = state["layer"](state["x"])
    dx, dw = torch.autograd.grad(y, [state["x"], state["layer"].weight], state["grad"])
    return dict(y=y.detach(), dx=dx, dw=dw)


# ------------------------------------------------------------------------------------------------- what a pass must do
def work(case):
    """Every operand once from and to memory; per (row, input that spikes, output) three flops forward (the two running
    sums), and per output with a gradient two for dX and three for dW. About half of a hidden layer's inputs spike; in the
    networks about a quarter of the outputs carry a gradient."""
    if case["kind"] != "net":
        R, I, J = _layer_rij(case)
        n_in = case["B"] * (case["I"] if case["kind"] == "dense" else case["H"] * case["W"] * case["C"])
        spiking = R * I * J * (1.0 if case["family"] == "input" else 0.5)
        if case["mode"] == "infer":
            return dict(bytes=4.0 * (n_in + I * J + R * J), flops=3.0 * spiking)
        # forward x, w, y; backward the upstream gradient, dX and dW on top
        return dict(bytes=4.0 * (2 * n_in + 2 * I * J + 2 * R * J), flops=spiking * (3.0 + 5.0 * case["grads"]))
    specs, shape, _ = NETS[case["net"]]
    n = case["batch"]
    layers = nets.layer_work(specs, shape)
    params = sum(l["I"] * l["J"] for l in layers)
    acts = sum(n * l["R"] * l["J"] for l in layers)
    nbytes, flops = 4.0 * (n * math.prod(shape) + params + layers[-1]["J"] * n), 0.0
    for l in layers:
        spiking = n * l["R"] * l["I"] * l["J"] * (0.5 if l["needs_dx"] else 1.0)
        flops += 3.0 * spiking
        if case["mode"] != "infer":
            flops += 0.25 * spiking * (5.0 if l["needs_dx"] else 3.0)
    if case["mode"] != "infer":
        nbytes += 4.0 * (2 * acts + params * (1 if case["mode"] == "grad" else 6))
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """Sums of 32-bit floats; a network's gradient is such sums chained through all its layers. A spike decision is a
    comparison that a last bit can tip, and one tipped output of a step moves its whole gradient: where the weights have
    been updated from gradients that differ by 3e-7, the next step's gradient was measured to differ by up to 2e-3
    (largest element 8e-3)."""
    if case["kind"] != "net" or case["mode"] == "infer":
        return {"rel": 1e-5}
    return {"rel": 1e-4} if case["mode"] == "grad" else {"rel": 5e-3, "max": 0.1}
