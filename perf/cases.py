"""The work this framework is used for, as cases to be timed: training steps, predictions and
short epochs of the four network classes, through their public Python entry points.

A case is one network with one batch (or one small data set).  ``prepare`` builds and configures
the network and makes its inputs, ``run`` is one call (or the few calls of one epoch) as a training
or serving program makes it, and its outputs are the energies or predictions that the call returns
together with the network's own state: beliefs, errors, weights, biases, feedback weights and Adam
moments (views of the library's device memory, no copies).

Dense networks: ``widths`` lists the layer widths, input first.  Convolutions: ``convs`` lists the
layers as <channels>k<kernel>s<stride>p<padding>.
"""
import math

import numpy as np
import torch

import deepity_b200 as dp

ACTS = {"sigmoid": dp.Sigmoid, "tanh": dp.TanH, "relu": dp.ReLU, "gelu": dp.GeLU,
        "esigmoid": dp.ESigmoid, "hard_tanh": dp.HardTanH}


# ------------------------------------------------------------------------------ the cases
def _dense(name, kind, call, widths, batch, steps, act, **more):
    return dict(name=name, kind=kind, call=call, widths=widths, batch=batch, steps=steps, act=act,
                optimizer=more.pop("optimizer", "SGD"), psi_optimizer=more.pop("psi_optimizer", "SGD"),
                precision=more.pop("precision", "fp32"), options=more.pop("options", ""),
                batches=more.pop("batches", 1))


def listed():
    return [
        # The reference's MNIST classifier: small host batches, one training step per call.
        _dense("simple_mnist_train", "simple", "train", "784-128-128-10", 64, 20, "sigmoid"),
        # The same classifier serving requests: latency of one prediction.
        _dense("simple_mnist_predict", "simple", "predict", "784-128-128-10", 64, 20, "sigmoid"),
        # The medium-depth DKP classifier trained from host batches.
        _dense("dkp_mlp_train", "dkp", "train", "784" + "-256" * 8 + "-10", 256, 2, "tanh"),
        # An epoch over a small tabular data set with fit(): widths and batch that fit no tile,
        # AdamW weights and Adam feedback weights.
        _dense("dkp_ragged_fit", "dkp", "fit", "100-300-200-77-10", 50, 6, "relu",
               optimizer="ADAMW", psi_optimizer="ADAM", batches=16),
        # The depth-scaling stack (width 512, batch 1024), inputs already on the GPU.
        _dense("dkp_deep_stack", "dkp", "device", "512" + "-512" * 512 + "-10", 1024, 2, "tanh"),
        # A shallower stack of that width in the single-pass TF32 mode that a user may choose.
        _dense("dkp_stack_tf32", "dkp", "device", "512" + "-512" * 12 + "-10", 1024, 2, "tanh",
               precision="tf32"),
        # The wide CIFAR-shaped classifier: cross-entropy head, Adam, large batch.
        _dense("full_wide_train", "full", "device", "3072" + "-1024" * 4 + "-10", 4096, 20, "gelu",
               optimizer="ADAM", psi_optimizer="ADAM", options="ce"),
        # A deep residual network with muPC scaling and momentum in the state updates.
        _dense("full_residual_train", "full", "device", "784" + "-256" * 30 + "-10", 256, 5, "relu",
               options="mupc residual momentum"),
        # Batch inference with the wide classifier from host memory.
        _dense("full_wide_predict", "full", "predict", "3072" + "-1024" * 4 + "-10", 1024, 10,
               "gelu", options="ce"),
        # A wide classic predictive-coding network on a large batch.
        _dense("simple_wide_train", "simple", "device", "784" + "-1024" * 4 + "-10", 4096, 20,
               "tanh"),
        # The CIFAR-shaped convolutional network: four host batches, then the weights are read
        # back as a checkpoint would.
        dict(name="conv_cifar_epoch", kind="conv", call="epoch", channels=3, side=32,
             convs="32k3s2p1 64k3s2p1 128k3s2p1 10k4s1p0", batch=128, steps=10, act="relu",
             optimizer="SGD", batches=4),
        # A small MNIST-shaped convolutional network serving an odd batch.
        dict(name="conv_mnist_predict", kind="conv", call="predict", channels=1, side=28,
             convs="8k5s2p2 16k3s2p1 10k7s1p0", batch=50, steps=10, act="tanh",
             optimizer="SGD", batches=1),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """Half of the sizes that users choose are round, the others are whatever the data gave."""
    n = _log_int(rng, lo, hi)
    if rng.random() < 0.5:
        return n
    step = 256 if n >= 512 else 64 if n >= 96 else 16 if n >= 16 else 4
    return max(lo, min(hi, (n + step // 2) // step * step))


def _draw_dense(rng):
    kind = rng.choice(("simple", "dkp", "full"))
    call = rng.choices(("train", "device", "predict", "fit"), (40, 25, 20, 15))[0]
    batch = _size(rng, 1, 4096)
    width = _size(rng, 16, 1024)
    inputs = rng.choice((784, 3072, width, _size(rng, 8, 2048)))
    outputs = rng.choice((10, 10, 2, 16, 100, _log_int(rng, 2, 64)))
    hidden = rng.randint(1, 4) if kind == "simple" else _log_int(rng, 1, 64)
    steps = rng.randint(hidden + 2, 20) if kind == "simple" else rng.choice((2, 2, 3, 4, 6, 10))
    act = rng.choice(sorted(ACTS))
    opts = []
    if kind == "full":
        # stacks of more than a dozen layers are residual and muPC-scaled, or use tanh
        if rng.random() < (0.7 if hidden > 12 else 0.2):
            opts += ["mupc", "residual"]
        for name, share in (("momentum", 0.3), ("ce", 0.4), ("ipc", 0.1), ("epc", 0.1)):
            if rng.random() < share:
                opts.append(name)
    elif kind == "simple" and rng.random() < 0.2:
        opts.append("ce")
    if hidden > 12 and "mupc" not in opts:
        act = "tanh"
    optimizer = rng.choice(("SGD", "SGD", "ADAM", "ADAMW"))
    case = _dense("", kind, call, "-".join(map(str, [inputs] + [width] * hidden + [outputs])), batch,
                  steps, act, optimizer=optimizer,
                  psi_optimizer=rng.choice(("SGD", "ADAM")) if kind != "simple" else "SGD",
                  precision="tf32" if rng.random() < 0.1 else "fp32", options=" ".join(opts),
                  batches=rng.randint(4, 16) if call == "fit" else 1)
    del case["name"]
    return case


def _draw_conv(rng):
    side = rng.choice((8, 16, 28, 32, rng.randint(8, 32)))
    count = rng.randint(1, 3)
    convs, s, ch = [], side, _log_int(rng, 4, 32)
    for _ in range(count):
        k = rng.choice((3, 3, 5))
        stride = 2 if s >= 8 and rng.random() < 0.7 else 1
        convs.append(f"{ch}k{k}s{stride}p{k // 2}")
        s = (s + 2 * (k // 2) - k) // stride + 1
        ch = min(128, ch * 2)
    convs.append(f"{rng.choice((10, 10, 2, 37))}k{s}s1p0")
    call = rng.choice(("epoch", "epoch", "predict"))
    return dict(kind="conv", call=call, channels=rng.choice((1, 3)), side=side,
                convs=" ".join(convs), batch=_size(rng, 1, 128), steps=rng.randint(2, 10),
                act=rng.choice(sorted(ACTS)), optimizer=rng.choice(("SGD", "SGD", "ADAM")),
                batches=rng.randint(1, 4) if call == "epoch" else 1)


def draw(rng):
    while True:
        case = _draw_conv(rng) if rng.random() < 0.18 else _draw_dense(rng)
        # far inside the largest listed case's work; state of at most about 2 GB
        if work(case)["flops"] <= (5e10 if case["kind"] == "conv" else 2.5e11) and \
                _state_floats(case) <= 5e8:
            return case


# ------------------------------------------------------------------------------ geometry
def _widths(case):
    return [int(v) for v in case["widths"].split("-")]


def _conv_layers(case):
    """(in channels, in side, out channels, kernel, stride, padding, out side) per weight layer"""
    out, c, s = [], case["channels"], case["side"]
    for text in case["convs"].split():
        o, rest = text.split("k")
        k, rest = rest.split("s")
        st, p = rest.split("p")
        o, k, st, p = int(o), int(k), int(st), int(p)
        t = (s + 2 * p - k) // st + 1
        out.append((c, s, o, k, st, p, t))
        c, s = o, t
    return out


def _state_floats(case):
    if case["kind"] == "conv":
        return sum(6 * case["batch"] * o * t * t for _, _, o, _, _, _, t in _conv_layers(case))
    w = _widths(case)
    data = 20 * case["batch"] * case["batches"] * w[0]  # uploaded every epoch: keep it modest
    return sum(6 * case["batch"] * v for v in w) + 4 * sum(a * b for a, b in zip(w, w[1:])) + data


# ------------------------------------------------------------------------------ state
class _Device:
    """A float tensor in the library's device memory, for torch.as_tensor."""

    def __init__(self, ptr, shape, strides):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "version": 3,
                                         "strides": tuple(4 * s for s in strides),
                                         "data": (ptr, False)}


def _views(net, widths, simple, optimizer, psi_optimizer):
    """The network's state as torch views.  Neighbouring layers of one shape make one view with
    the layer as its outermost dimension."""
    names = [("z", True), ("e", True), ("W", False), ("b", False)]
    if not simple:
        names.append(("Psi", False))
    if optimizer != "SGD":
        names += [(n, False) for n in ("weight.m", "weight.v", "bias.m", "bias.v")]
    if not simple and psi_optimizer != "SGD":
        names += [("psi.m", False), ("psi.v", False)]
    out = {}
    for name, beliefs in names:
        layers = []
        for l in range(len(widths) if beliefs else len(widths) - 1):
            if beliefs:
                shape = (net.batch_size, widths[l])
            elif name in ("W", "weight.m", "weight.v"):
                shape = (widths[l + 1], widths[l])
            elif name in ("b", "bias.m", "bias.v"):
                shape = (1, widths[l + 1])
            else:
                shape = (widths[l], widths[-1])
            layers.append((net.tensor_ptr(l, name), shape))
        l = 0
        while l < len(layers):
            ptr, shape = layers[l]
            end, step = l + 1, shape[0] * shape[1]
            if end < len(layers) and layers[end][1] == shape:
                step = (layers[end][0] - ptr) // 4
            while end < len(layers) and layers[end][1] == shape and \
                    layers[end][0] - layers[end - 1][0] == 4 * step:
                end += 1
            view = _Device(ptr, (end - l,) + shape, (step, shape[1], 1))
            out[f"{name}.{l}"] = torch.as_tensor(view, device="cuda")
            l = end
    return out


def _one_hot(rows, classes, gen):
    index = torch.randint(classes, (rows,), generator=gen, device="cuda")
    return torch.nn.functional.one_hot(index, classes).float()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    host = lambda t: np.ascontiguousarray(t.cpu().numpy())  # noqa: E731
    batch, rows = case["batch"], case["batch"] * case["batches"]
    if case["kind"] == "conv":
        arch, spec = [], _conv_layers(case)
        for i, (_, _, o, k, s, p, _) in enumerate(spec):
            arch.append(dp.Convolution(o, k, k, s, s, p, p))
            if i + 1 < len(spec):
                arch.append(ACTS[case["act"]]())
        arch.append(dp.Convolution(0, 1, 1))
        net = dp.SimpleConvolutionalPCN(*arch, input_shape=(case["channels"],) + (case["side"],) * 2,
                                        batch_size=batch)
        net.configure(learning_rate=1e-3, inference_rate=0.1, lmbda=1e-4,
                      optimizer=case["optimizer"], seed=seed % 2 ** 31)
        x = torch.randn(rows, case["channels"], case["side"], case["side"], generator=gen,
                        device="cuda")
        y = _one_hot(rows, spec[-1][2], gen)
        return dict(case=case, net=net, x=host(x), y=host(y), weights=len(spec))

    kind, widths, opts = case["kind"], _widths(case), case["options"].split()
    arch = []
    for a, b in zip(widths, widths[1:]):
        arch += [dp.Linear(a, b), ACTS[case["act"]]()]
    cls = {"simple": dp.SimplePCN, "dkp": dp.DKPPCN, "full": dp.FullPCN}[kind]
    net = cls(*arch, batch_size=batch)
    kw = dict(learning_rate=1e-3, inference_rate=0.1, lmbda=1e-4, optimizer=case["optimizer"],
              seed=seed % 2 ** 31, precision=case["precision"])
    if kind != "simple":
        kw.update(feedback_rate=1e-3, psi_optimizer=case["psi_optimizer"])
    if kind == "simple":
        kw.update(use_cross_entropy="ce" in opts)
    if kind == "full":
        kw.update(use_mu_pc_scaling="mupc" in opts, use_residual_connections="residual" in opts,
                  use_momentum="momentum" in opts, use_cross_entropy="ce" in opts,
                  use_ipc="ipc" in opts, use_epc="epc" in opts)
    net.configure(**kw)
    if case["act"] in ("sigmoid", "esigmoid"):  # image data in [0, 1)
        x = torch.rand(rows, widths[0], generator=gen, device="cuda")
    else:
        x = torch.randn(rows, widths[0], generator=gen, device="cuda")
    y = _one_hot(rows, widths[-1], gen)
    for l, n in enumerate(widths[1:]):  # biases as a network that has been trained holds them
        net.set_tensor(l, "b", 0.1 * torch.randn(n, generator=gen, device="cuda"))
    state = dict(case=case, net=net)
    if case["call"] == "device":
        state.update(x=x, y=y)
    else:
        state.update(x=host(x), y=host(y))
    if case["call"] != "predict":
        state["views"] = _views(net, widths, kind == "simple", case["optimizer"],
                                case["psi_optimizer"])
    return state


def run(state):
    case, net, x, y = state["case"], state["net"], state["x"], state["y"]
    steps, call = case["steps"], case["call"]
    if case["kind"] == "conv":
        if call == "predict":
            return net.predict_with_projection(x, steps)
        n = case["batch"]
        out = {"energy": [net.train_step(x[i * n:(i + 1) * n], y[i * n:(i + 1) * n], steps)
                          for i in range(case["batches"])]}
        for l in range(state["weights"]):
            out[f"W.{l}"], out[f"b.{l}"] = net.layers[l].weights, net.layers[l].biases
        return out
    if call == "predict":
        return net.predict(x, steps)
    out = dict(state["views"])
    if call == "train":
        out["energy"] = net.train_step(x, y, steps)
    elif call == "device":
        out["energy"] = net.train_step_device(x, y, steps)
    else:
        net.fit(x, y, 1, steps, shuffle=False)
    return out


# ------------------------------------------------------------------------------ what it costs
def work(case):
    """Bytes: inputs, parameters and optimizer state read once and written once, beliefs and errors
    written once (a prediction: inputs and parameters in, outputs out).  FLOPs: the products that
    the algorithm asks for; the clamped input layer's prediction is computed once per step."""
    batch, steps, train = case["batch"], case["steps"], case["call"] != "predict"
    adam = case["optimizer"] != "SGD"
    if case["kind"] == "conv":
        flops, params = 0.0, 0.0
        spec = _conv_layers(case)
        states = batch * case["channels"] * case["side"] ** 2
        for i, (c, _, o, k, _, _, t) in enumerate(spec):
            product = 2.0 * batch * o * t * t * c * k * k
            flops += product * ((1 if i == 0 else 2 * steps + 1) + (1 if train else 0))
            params += o * c * k * k + o
            states += batch * o * t * t
        inputs = batch * (case["channels"] * case["side"] ** 2 + spec[-1][2])
    else:
        flops, params = 0.0, 0.0
        w, kind = _widths(case), case["kind"]
        for i, (a, b) in enumerate(zip(w, w[1:])):
            product = 2.0 * batch * a * b
            settle = 0 if i == 0 else steps
            if kind == "simple":
                forward, learn = settle + 1, 1 if train else 0
            else:
                # sweep; with training also the refresh before learning and the closing energy
                forward = settle + (1 if i == 0 else 3 if train else 1)
                learn = 2 if i + 2 < len(w) else 1
                if "ipc" in case["options"].split():
                    learn += steps - 1
                if not train:
                    learn = 0
            flops += product * (forward + settle + learn)
            params += a * b + b
            if kind != "simple" and train:
                params += a * w[-1]
                flops += 2.0 * batch * w[-1] * (a + (b if i + 2 < len(w) else 0))
        states, inputs = batch * sum(w), batch * (w[0] + w[-1])
    count = case["batches"]
    if not train:
        return {"bytes": 4.0 * (inputs + params), "flops": flops}
    per = inputs + 2 * states + params * (2 + (4 if adam else 0))
    return {"bytes": 4.0 * per * count, "flops": flops * count}


def tolerance(case):
    """Beliefs, weights and energies of two correct fp32 implementations agree to 1e-6 .. 1e-5.  The
    errors (belief minus prediction) are differences of nearly equal numbers: where a short settling
    has moved the beliefs by a hundredth of their size they carry that rounding a hundred times
    larger, and where muPC scaling makes the feedback another factor of ten smaller, a thousand."""
    if "mupc" in case.get("options", ""):
        return {"rel": 2e-2, "max": 0.5}
    if case.get("precision") == "tf32":  # 10-bit operands: 5e-4 each, with the same amplification
        return {"rel": 3e-2, "max": 0.5}
    if case["optimizer"] != "SGD" or case.get("psi_optimizer", "SGD") != "SGD":
        # an element whose gradient is of the size of the rounding may step the other way
        return {"rel": 4e-3, "max": 0.5}
    if case["kind"] in ("simple", "conv"):
        return {"rel": 1e-4, "max": 4e-3}
    return {"rel": 1e-3, "max": 4e-2}
