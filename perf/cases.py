"""The work that programs built on this framework give it, as cases that can be timed and compared.

Six kinds, one per public way in: ``compiled`` (CompiledLogicNet, the deployed discretised network), ``packed`` (bit-packed
inference through the modules), ``eval`` (float evaluation with arg-max gates, what a validation pass runs), ``train`` (the plain
modules with torch's cross-entropy, gradients left in ``.grad`` for an optimizer of the caller's own), ``step`` (the whole
training step: fused flat layers and loss, gradients in one bucket, Adam) and ``block`` / ``flat`` (one ConvLogic block, one stack
of flat layers, forward and backward, as parts of a model of the caller's own).  The shapes of the stacks are those of
``ConvLogicCifarModel`` and ``ConvLogicMnistModel`` for a width ``k``.
"""

import torch

import convlogic_b200 as cb

DEV = "cuda"


def listed():
    return [
        # one request to a deployed MNIST-sized network: launches and host time only
        {"name": "compiled mnist k16 b1", "kind": "compiled", "stack": "mnist", "k": 16, "batch": 1, "input": "bool"},
        # the same network on one test batch (configuration 1 of the benchmark)
        {"name": "compiled mnist k16 b256", "kind": "compiled", "stack": "mnist", "k": 16, "batch": 256, "input": "bool"},
        # a small CIFAR network on a ragged batch of float pixels, three thermometer levels per colour
        {"name": "compiled cifar k32 b1000", "kind": "compiled", "stack": "cifar", "k": 32, "batch": 1000, "input": "float", "levels": 3},
        # bulk inference with the largest network: one streamed chunk of byte pixels (configuration 4)
        {"name": "compiled cifar k1024 b8192", "kind": "compiled", "stack": "cifar", "k": 1024, "batch": 8192, "input": "byte", "levels": 31},
        # a flat network on a whole test set, 32 samples per word (the default of PackBitsTensor)
        {"name": "packed flat 64000x4 b10000", "kind": "packed", "in": 3072, "width": 64000, "depth": 4, "batch": 10000, "bits": 32},
        # validation pass of a small CIFAR network during training
        {"name": "eval cifar k32 b500", "kind": "eval", "stack": "cifar", "k": 32, "batch": 500, "levels": 3},
        # drop-in training of the small MNIST network
        {"name": "train mnist k16 b128", "kind": "train", "stack": "mnist", "k": 16, "batch": 128, "levels": 1},
        # training step of a small CIFAR network, batch not a power of two
        {"name": "step cifar k32 b100", "kind": "step", "stack": "cifar", "k": 32, "batch": 100, "levels": 3},
        # training step of the middle CIFAR network (configuration 3, the headline of the benchmark)
        {"name": "step cifar k256 b256", "kind": "step", "stack": "cifar", "k": 256, "batch": 256, "levels": 3},
        # one first block with its input gradient (configuration 2)
        {"name": "block 9-256 32x32 b256", "kind": "block", "cin": 9, "cout": 256, "side": 32, "batch": 256, "values": "bits"},
        # a small flat network
        {"name": "flat 784-8000x3 b100", "kind": "flat", "in": 784, "width": 8000, "depth": 3, "batch": 100},
        # the large flat stack (configuration 5)
        {"name": "flat 3072-256000x8 b1024", "kind": "flat", "in": 3072, "width": 256000, "depth": 8, "batch": 1024},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["compiled", "compiled", "packed", "eval", "train", "step", "step", "block", "block", "flat", "flat"])
    if kind == "compiled":
        if rng.random() < 0.4:
            return {"kind": kind, "stack": "mnist", "k": _log(rng, 8, 64), "batch": _log(rng, 1, 4096), "input": "bool"}
        k = _log(rng, 16, 1024)
        return {"kind": kind, "stack": "cifar", "k": k, "batch": _log(rng, 1, min(8192, 8192 * 1024 // k)),
                "input": rng.choice(["float", "byte"]), "levels": rng.randint(1, 31)}
    if kind == "packed":
        width, depth = 10 * _log(rng, 200, 12800), rng.randint(2, 6)
        return {"kind": kind, "in": _log(rng, 64, min(4096, 2 * width)), "width": width, "depth": depth, "batch": _log(rng, 16, 20000),
                "bits": rng.choice([8, 16, 32, 64])}
    if kind in ("eval", "train", "step"):
        stack = rng.choice(["mnist", "cifar", "cifar"])
        k = _log(rng, 8, 64 if stack == "mnist" else 256)
        return {"kind": kind, "stack": stack, "k": k, "batch": _log(rng, 16, min(512, 65536 // k)), "levels": 1 if stack == "mnist" else rng.randint(1, 5)}
    if kind == "block":
        side = rng.choice([4, 8, 12, 16, 28, 32])
        cout = _log(rng, 16, 1024)
        return {"kind": kind, "cin": _log(rng, 1, 256), "cout": cout, "side": side,
                "batch": _log(rng, 8, min(512, 256 * 256 * 1024 // (cout * side * side))), "values": rng.choice(["bits", "real"])}
    width, depth = 10 * _log(rng, 100, 25600), rng.randint(2, 8)
    return {"kind": "flat", "in": _log(rng, 64, min(4096, 2 * width)), "width": width, "depth": depth, "batch": _log(rng, 16, 1024)}


# ------------------------------------------------------------------------------------------ models
def _stack(case, seed):
    """The nn.Sequential of a case on the GPU, gate logits N(0, 1); connections and logits come from the seed."""
    torch.manual_seed(seed)
    if case["stack"] == "cifar":
        net = cb.ConvLogicCifarModel(k_param=case["k"], input_channels=3 * case["levels"], tau=20).network
    else:
        net = cb.ConvLogicMnistModel(k_param=case["k"], tau=6.5).network
    return _gates(net, seed)


def _flat(case, seed):
    torch.manual_seed(seed)
    dims = [case["in"]] + [case["width"]] * case["depth"]
    return _gates(torch.nn.Sequential(*[cb.LogicLayer(i, o, residual_init=True) for i, o in zip(dims[:-1], dims[1:])], cb.GroupSum(10, 30.0)), seed)


def _gates(net, seed):
    net = net.to(DEV)
    g = torch.Generator(device=DEV).manual_seed(seed)
    for p in net.parameters():
        p.data.normal_(generator=g)
    return net


_deployed = {}  # the one network a serving program holds: requests (seeds) differ, the network does not


def _deployed_net(case):
    key = (case["stack"], case["k"], case.get("levels"))
    if key not in _deployed:
        _deployed.clear()
        shape = (1, 28, 28) if case["stack"] == "mnist" else (3 * case["levels"], 32, 32)
        _deployed[key] = cb.CompiledLogicNet(_stack(case, 3).eval(), input_shape=shape).compile()
    return _deployed[key]


def _deployed_flat(case):
    key = (case["in"], case["width"], case["depth"])
    if key not in _deployed:
        _deployed.clear()
        _deployed[key] = _flat(case, 3).eval()
    return _deployed[key]


def _images(case, g):
    """Thermometer bits of CIFAR-like pixels (each bit set with probability 1/2) or MNIST-like ones (1/5), as float."""
    n = case["batch"]
    shape, p = ((n, 1, 28, 28), 0.2) if case["stack"] == "mnist" else ((n, 3 * case["levels"], 32, 32), 0.5)
    return (torch.rand(shape, device=DEV, generator=g) < p).float()


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind, n = case["kind"], case["batch"]
    s = {"kind": kind}
    if kind == "compiled":
        s["net"] = _deployed_net(case)
        if case["input"] == "bool":
            s["x"] = torch.rand((n, 1, 28, 28), device=DEV, generator=g) < 0.2
        else:
            levels = case["levels"]
            s["thresholds"] = torch.arange(1, levels + 1, device=DEV, dtype=torch.float32) / (levels + 1)
            x = torch.randint(0, 256, (n, 3, 32, 32), device=DEV, generator=g, dtype=torch.uint8)
            s["x"] = x if case["input"] == "byte" else x.float() / 255
    elif kind == "packed":
        s["net"], s["bits"] = _deployed_flat(case), case["bits"]
        s["x"] = torch.rand((n, case["in"]), device=DEV, generator=g) < 0.5
    elif kind == "eval":
        s["net"], s["x"] = _stack(case, seed).eval(), _images(case, g)
    elif kind in ("train", "step"):
        net, s["x"] = _stack(case, seed).train(), _images(case, g)
        s["labels"] = torch.randint(0, 10, (n,), device=DEV, generator=g)
        if kind == "train":
            s["net"] = net
        else:
            net = cb.fuse_logic_layers(net).train()
            s["bucket"] = cb.GradBucket(net).direct()
            s["adam"] = cb.FlatAdam(s["bucket"], lr=0.01)
            s["body"], s["trees"], s["sum"] = net[:-2], net[-2], net[-1]
    elif kind == "block":
        torch.manual_seed(seed)
        s["net"] = _gates(cb.ConvLogicLayer(case["cin"], case["cout"], residual_init=True, complete=True), seed).train()
        x = torch.rand((n, case["cin"], case["side"], case["side"]), device=DEV, generator=g)
        s["x"] = ((x < 0.5).float() if case["values"] == "bits" else x).requires_grad_(True)
        s["grad"] = torch.randn((n, case["cout"], case["side"] // 2, case["side"] // 2), device=DEV, generator=g)
    else:
        s["net"] = _flat(case, seed).train()
        s["x"] = (torch.rand((n, case["in"]), device=DEV, generator=g) < 0.5).float()
        s["grad"] = torch.randn((n, 10), device=DEV, generator=g)
    return s


def run(s):
    kind, x = s["kind"], s["x"]
    if kind == "compiled":
        return s["net"].forward_pixels(x, s["thresholds"]) if "thresholds" in s else s["net"](x)
    if kind == "packed":
        return s["net"](cb.PackBitsTensor(x, s["bits"]))
    if kind == "eval":
        with torch.no_grad():
            return s["net"](x)
    if kind == "step":
        loss = s["trees"].cross_entropy(s["body"](x), s["labels"], s["sum"].k, s["sum"].tau)
        loss.backward()
        s["adam"].step()
        return {"loss": loss.detach(), "gradients": s["bucket"].flat, "logits": s["adam"].params}
    net = s["net"]
    for p in net.parameters():
        p.grad = None
    x.grad = None
    y = net(x)
    if kind == "train":
        y = torch.nn.functional.cross_entropy(y, s["labels"])
        y.backward()
    else:
        y.backward(s["grad"])
    out = {"y": y.detach(), "gates": [p.grad for p in net.parameters()]}
    if kind == "block":
        out["x"] = x.grad
    return out


# -------------------------------------------------------------------------------------------- work
def _layers(case):
    """(features in, features out, positions at which its gates are evaluated, neurons) of every layer of a stack."""
    k = case["k"]
    if case["stack"] == "cifar":
        ch, size, flat = [3 * case["levels"], k, 4 * k, 16 * k, 32 * k], [32, 16, 8, 4, 2], 128 * k
        e = 2 if k >= 1024 else 1
        dims = [flat, 10 * e * flat, 5 * e * flat, e * flat * 10 // 4]
        conv = [(ch[i] * size[i] ** 2, ch[i + 1] * size[i + 1] ** 2, size[i] ** 2, 7 * ch[i + 1]) for i in range(4)]
    else:
        conv = [(784, k * 144, 576, 7 * k), (k * 144, 3 * k * 36, 144, 21 * k), (3 * k * 36, 9 * k * 9, 36, 63 * k)]
        dims = [81 * k, 1280 * k, 640 * k, 320 * k]
    return conv, [(i, o, 1, o) for i, o in zip(dims[:-1], dims[1:])]


def work(case):
    """Bytes: inputs, weights and results of the call, each once -- for a network of float modules those of every module (the three
    flat layers that ``step`` fuses count as one).  Operations: three multiply-adds per gate in the forward pass, six more for
    its gradients; one per gate and 32 samples on packed bits."""
    kind, n = case["kind"], case["batch"]
    if kind == "compiled":
        conv, flat = _layers(case)
        pixel = {"bool": 784, "byte": 3072, "float": 4 * 3072}[case["input"]]
        gates = sum(c[3] for c in conv + flat)
        # connections and gate of a neuron: one byte per gate, 32 per conv channel (7 gates), 8 per flat neuron of the first layer
        params = gates + sum(c[3] for c in conv) // 7 * 32 + 8 * flat[0][1]
        return {"bytes": n * (pixel + 40) + params, "flops": sum(c[2] * c[3] for c in conv + flat) * n / 32}
    if kind == "packed":
        width, depth = case["width"], case["depth"]
        row = (n + 7) // 8
        return {"bytes": n * (case["in"] + 40) + 2 * case["in"] * row + 2 * depth * width * row + 17 * depth * width, "flops": depth * width * n / 32}
    if kind == "block":
        x, y, gates = case["cin"] * case["side"] ** 2, case["cout"] * (case["side"] // 2) ** 2, 7 * case["cout"]
        return {"bytes": 4 * n * (3 * x + 2 * y) + 4 * 16 * 3 * gates, "flops": 18 * n * gates * case["side"] ** 2}
    if kind == "flat":
        layers = [(case["in"], case["width"], 1, case["width"])] + [(case["width"], case["width"], 1, case["width"])] * (case["depth"] - 1)
    else:
        conv, flat = _layers(case)
        layers = conv + ([(flat[0][0], flat[-1][1], 1, sum(c[3] for c in flat))] if kind == "step" else flat)
    gates = sum(c[3] for c in layers)
    forward = 4 * n * (sum(c[0] + c[1] for c in layers) + layers[-1][1]) + 64 * gates
    flops = 6 * n * sum(c[2] * c[3] for c in layers)
    if kind == "eval":
        return {"bytes": forward, "flops": flops}
    # backward: upstream gradient and input of every layer read, input gradient of all but the first and every gate gradient written
    backward = 4 * n * (sum(2 * c[0] + c[1] for c in layers) - layers[0][0]) + 2 * 64 * gates
    adam = 7 * 64 * gates if kind == "step" else 0
    return {"bytes": forward + backward + adam, "flops": 3 * flops}


def tolerance(case):
    """Counts are whole numbers.  Flat layers: sums in fp32 whose order is free.  Behind a 2x2 max pool the gradient of a window goes
    to the candidate that wins, and two candidates may differ by less than a rounding: logits moved by 3e-8 move the gate
    gradients of the stacks by up to 5e-5."""
    if case["kind"] in ("compiled", "packed"):
        return "exact"
    return {"rel": 1e-4 if case["kind"] in ("train", "step", "block") else 1e-5}
