"""What the performance of this library is measured on: training and inference passes as a host program makes them
through the public entry points (myea_b200.net.Net and the C ABI behind it), over the range of networks it is used for.

A case is a dict of plain values:
  mode       "step"     `steps` times the training sequence forward, compute_error, backward, update_derivative_weight,
                        update_parameter, each on a batch of its own; then the loss and the trained parameters are read
             "epoch"    train_epoch over `steps` mini-batches of a dataset that lies on the device; then the same
             "predict"  one inference-mode forward pass; the network's outputs are read into host memory
  source     where the batches come from: "device" memory, pinned "host" memory (then the loss is read after every step,
             as a host loop that watches its training does), or the "dataset" of an epoch
  kind       "mlp", "residual" (blocks of two fully connected layers with ShakeDrop) or "lstm"
  layers     hidden layers, residual blocks or LSTM layers;  hidden: their width (per direction for LSTM layers)
  resume     the optimizer's moments are read as well (what a program needs to continue the training elsewhere); without
             it the parameters and normalization averages, which are what a checkpoint file holds
"""
import ctypes as C
import math

import torch

from myea_b200 import capi
from myea_b200.net import Net

ACTIVATIONS = {"tanh": capi.AF_TANH, "relu": capi.AF_RELU, "elu": capi.AF_ELU, "sigmoid": capi.AF_SIGMOID, "leaky_relu": capi.AF_LEAKY_RELU}
NORMS = {"none": capi.NORM_NONE, "bn": capi.NORM_BN, "brn": capi.NORM_BRN}
DROPOUTS = {"none": capi.DROP_NONE, "inverted": capi.DROP_BERNOULLI_INVERTED, "bernoulli": capi.DROP_BERNOULLI}
DEFAULTS = {"mode": "step", "source": "device", "kind": "mlp", "layers": 2, "activation": "tanh", "norm": "none", "dropout": "none", "keep": 0.5,
            "time": 1, "last_step_only": False, "bidirectional": False, "zoneout": 0.0, "loss": "mse", "optimizer": "adam", "clip": 0.0,
            "decay": 0.0, "rate": 1e-3, "steps": 1, "resume": False}


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    small = dict(inputs=64, hidden=256, outputs=10, layers=2, activation="tanh", loss="ce")
    wide = dict(inputs=4096, hidden=4096, outputs=1024, layers=8, activation="relu", norm="bn", dropout="inverted", keep=0.5,
                rate=1e-4)
    res = dict(kind="residual", inputs=1024, hidden=2048, outputs=1000, layers=6, activation="elu", norm="brn", loss="ce", optimizer="adabound", decay=1e-4,
               rate=1e-4)
    lstm = dict(kind="lstm", inputs=512, hidden=1024, outputs=1024, layers=2, time=64, last_step_only=True, optimizer="amsgrad")
    return [
        # one answer from the 64-256-256-10 classifier: a host program that asks for a single row, where only latency counts
        _case("small mlp, predict one", mode="predict", source="host", batch=1, **small),
        # an epoch of that classifier over a dataset on the device: mini-batches of 128, all launches and no arithmetic
        _case("small mlp, epoch", mode="epoch", source="dataset", batch=128, steps=16, resume=True, **small),
        # a classifier of ordinary size fed from host memory batch by batch
        _case("classifier from host", source="host", inputs=784, hidden=1024, outputs=10, layers=2, activation="relu", dropout="inverted", keep=0.8,
              loss="ce", batch=256, steps=8, resume=True),
        # widths and a batch that divide by nothing, smooth activations, momentum descent: a regression network
        _case("ragged regression", inputs=75, hidden=333, outputs=21, layers=4, activation="tanh", norm="bn", optimizer="nesterov", batch=203, steps=8,
              resume=True),
        # eight layers of 4096 units with batch normalization and dropout at the full batch: the largest training step
        _case("wide mlp", batch=4096, steps=6, **wide),
        # the same network on the rows one of eight GPUs gets of that batch
        _case("wide mlp, eighth batch", batch=512, steps=8, **wide),
        # and its answers for a full batch
        _case("wide mlp, predict", mode="predict", batch=4096, **wide),
        # residual network with batch renormalization and ShakeDrop
        _case("residual", batch=2048, steps=8, **res),
        # two peephole LSTM layers, full back-propagation through 64 steps, error on the last one
        _case("lstm", batch=256, steps=4, resume=True, **lstm),
        # its answers for a few sequences at a time, as a service asks for them
        _case("lstm, predict", mode="predict", source="host", batch=16, **lstm),
        # a small recurrent network of a width that is no multiple of anything, error on every step
        _case("small lstm", kind="lstm", inputs=39, hidden=150, outputs=161, layers=2, time=40, batch=50, steps=4, resume=True),
        # bidirectional LSTM with zoneout and clipping, the rows one of eight GPUs gets of a batch of 1024
        _case("bidirectional lstm", kind="lstm", inputs=1024, hidden=2048, outputs=1024, layers=1, time=128, bidirectional=True, zoneout=0.1, clip=1.0,
              batch=128, steps=2),
    ]


def _log(rng, lo, hi, multiple=32):
    """log-uniform in [lo, hi]: half of the values as they fall, half rounded to a multiple where they are large enough"""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if v >= multiple and rng.random() < 0.5:
        v = v // multiple * multiple
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["mlp", "mlp", "mlp", "residual", "lstm", "lstm"])
    mode = rng.choice(["step", "step", "epoch", "predict"])
    source = "dataset" if mode == "epoch" else rng.choice(["device", "host"])
    c = _case(mode=mode, source=source, kind=kind, loss=rng.choice(["mse", "ce"]), optimizer=rng.choice(["adam", "amsgrad", "adabound", "nesterov"]))
    if kind == "mlp":
        c.update(inputs=_log(rng, 16, 4096), hidden=_log(rng, 32, 4096), outputs=_log(rng, 4, 1024), layers=rng.randint(1, 8),
                 activation=rng.choice(["tanh", "relu", "sigmoid", "leaky_relu"]), norm=rng.choice(["none", "bn"]),
                 dropout=rng.choice(["none", "none", "inverted", "bernoulli"]), keep=rng.choice([0.5, 0.8]),
                 batch=_log(rng, 1 if mode == "predict" else 32, 4096))
    elif kind == "residual":
        c.update(inputs=_log(rng, 64, 1024), hidden=_log(rng, 128, 2048), outputs=_log(rng, 10, 1000), layers=rng.randint(1, 6),
                 activation=rng.choice(["elu", "relu", "tanh"]), norm=rng.choice(["bn", "brn"]), batch=_log(rng, 64, 2048), decay=rng.choice([0.0, 1e-4]))
    else:
        c.update(inputs=_log(rng, 16, 1024), hidden=_log(rng, 32, 2048), outputs=_log(rng, 4, 1024), layers=rng.randint(1, 2), time=_log(rng, 4, 128),
                 batch=_log(rng, 4, 256), loss="mse", last_step_only=rng.random() < 0.5, clip=rng.choice([0.0, 1.0]))
        if c["layers"] == 1 and rng.random() < 0.5:
            c.update(bidirectional=True, zoneout=0.1, last_step_only=False)
        else:   # the library asks for a next layer at least as wide (the reference's bias runs overlap)
            c["outputs"] = max(c["outputs"], c["hidden"])
    if mode != "predict":
        c["steps"] = rng.choice([2, 4, 8])
    c["rate"] = 1e-3 if c["hidden"] < 512 and kind != "residual" else 1e-4   # wide and deep networks are trained with small steps
    most = max(_cost(x) for x in listed())
    while _cost(c) > most:
        if c["steps"] > 1:
            c["steps"] //= 2
        elif c["time"] > 8:
            c["time"] //= 2
        else:
            c["batch"] = max(4, c["batch"] // 2)
    c["resume"] = mode != "predict" and _parameters(c) < 20e6
    return c


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def _fc_widths(c):
    """[inputs, outputs] of every fully connected layer in order, and of every LSTM layer"""
    if c["kind"] == "lstm":
        dirs = 2 if c["bidirectional"] else 1
        rec, n_in = [], c["inputs"]
        for _ in range(c["layers"]):
            rec.append((n_in, c["hidden"]))
            n_in = c["hidden"] * dirs
        return [(n_in, c["outputs"])], rec
    n = c["layers"] if c["kind"] == "mlp" else 1 + 2 * c["layers"]
    w = [c["inputs"]] + [c["hidden"]] * n + [c["outputs"]]
    return list(zip(w[:-1], w[1:])), []


def _parameters(c):
    fc, rec = _fc_widths(c)
    dirs = 2 if c["bidirectional"] else 1
    return sum(i * o + o for i, o in fc) + sum(dirs * 4 * h * (i + h + 1) for i, h in rec)


def work(case):
    c = case
    fc, rec = _fc_widths(c)
    dirs = 2 if c["bidirectional"] else 1
    rows, P = float(c["batch"] * c["time"]), float(_parameters(c))
    train = c["mode"] != "predict"
    # contractions: forward, error propagation (not below the first layer), weight derivatives
    flops = 0.0
    for k, (i, o) in enumerate(fc):
        flops += 2.0 * rows * i * o * ((3 if k or rec else 2) if train else 1)
    for k, (i, h) in enumerate(rec):
        flops += dirs * 2.0 * rows * 4 * h * ((i + h) * (2 if train else 1) + ((h + (i if k else 0)) if train else 0))
    moments = {"adam": 2, "amsgrad": 3, "adabound": 2, "nesterov": 1}[c["optimizer"]]
    io = rows * (c["inputs"] + c["outputs"]) * 4
    if not train:
        return {"bytes": P * 4 + io, "flops": flops}
    # every step reads its batch and reads and writes the parameters and the optimizer's state; the results once at the end
    read_back = P * 4 * (1 + (1 if c["resume"] else 0))
    return {"bytes": c["steps"] * (io + 2 * P * 4 * (1 + moments)) + read_back, "flops": c["steps"] * flops}


def tolerance(case):
    # Products carry 2e-6 of a tensor's scale whoever computes them in 32 bits.
    if case["mode"] == "predict":
        return {"rel": 4e-5, "max": 1e-3}
    # Through training two things enlarge that.  A pre-activation within rounding distance of a kink (ReLU, ELU) takes the
    # other branch on another correct implementation, which changes its derivative altogether; and the first steps of
    # Adam-type updates are lr * sign(g), so that a derivative which is zero up to the rounding of its sum moves its
    # weight by lr to either side (in a residual block all biases in front of the normalization are of that kind, and the
    # running means follow them).  Both touch few elements: a small share of the 2-norm, a large `max`.
    # Measured between two products that are exact to 2e-6 and 5e-7: up to 8e-3 on deep narrow networks, 1e-3 on wide ones.
    kinks = case["kind"] == "residual" or (case["kind"] == "mlp" and case["activation"] in ("relu", "leaky_relu"))
    if case["optimizer"] == "nesterov":   # linear in the derivatives
        return {"rel": 2e-2, "max": 0.5} if kinks else {"rel": 1e-4, "max": 2e-2}
    return {"rel": 2e-2 if kinks else 1e-2 if case["norm"] != "none" else 1e-3, "max": 0.5}


def _network(c):
    af, loss = ACTIVATIONS[c["activation"]], capi.LOSS_CE if c["loss"] == "ce" else capi.LOSS_MSE
    norm, drop = NORMS[c["norm"]], DROPOUTS[c["dropout"]]
    layers = [capi.fc(c["inputs"])]
    if c["kind"] == "mlp":
        layers += [capi.fc(c["hidden"], af, norm, drop, (c["keep"], 0.0, 0.0)) for _ in range(c["layers"])]
    elif c["kind"] == "residual":
        layers.append(capi.fc(c["hidden"], af))
        for _ in range(c["layers"]):
            layers += [capi.residual(2, capi.DROP_SHAKEDROP, (0.5, 0.0, 0.0)), capi.fc(c["hidden"], af), capi.fc(c["hidden"], af, norm)]
    else:
        z = c["zoneout"]
        layers += [capi.lstm(c["hidden"], bidirectional=c["bidirectional"], dropout=capi.DROP_ZONEOUT if z else capi.DROP_NONE, p=(z, z, 0.0))
                   for _ in range(c["layers"])]
    layers.append(capi.fc(c["outputs"], capi.AF_SOFTMAX if c["loss"] == "ce" else capi.AF_LINEAR))
    desc = capi.net(layers, c["batch"], T=c["time"], loss=loss, accuracy=capi.ACC_CE if c["loss"] == "ce" else capi.ACC_DISTANCE,
                    time_delays=c["time"] - 1 if c["last_step_only"] else 0, r_max=3.0, d_max=5.0)
    kw = {"clip": c["clip"] or None, "weight_decay": c["decay"], "lr": c["rate"]}
    # derivatives are sums over the batch: rates that multiply them directly are stated per example
    opt = {"adam": lambda: capi.opt(capi.OPT_ADAM, **kw), "amsgrad": lambda: capi.opt(capi.OPT_AMSGRAD, **kw),
           "adabound": lambda: capi.opt(capi.OPT_ADABOUND, final_lr=0.1 / c["batch"], **kw),
           "nesterov": lambda: capi.opt(capi.OPT_GD, gd_lr=c["rate"] / c["batch"], momentum=0.9, nesterov=True, **kw)}[c["optimizer"]]()
    return layers, desc, opt


def _initial_parameters(net, layers, gen):
    """Glorot-uniform weights with the gain of the activation function, biases 0, normalization scales 1 and shifts 0"""
    gain = {capi.AF_TANH: 5.0 / 3.0, capi.AF_RELU: math.sqrt(2.0), capi.AF_LEAKY_RELU: math.sqrt(2.0)}
    p = torch.zeros(net.P, device="cuda")
    for l in range(1, len(layers)):
        li = net.layer_index(l)
        a, b = int(li.first_connection_index), int(li.last_connection_index)
        if layers[l].type_layer not in (capi.LAYER_FC, capi.LAYER_LSTM) or b <= a:
            continue
        n_in, n_out = int(li.number_inputs), int(li.number_outputs)
        if layers[l].type_layer == capi.LAYER_LSTM:
            bound = math.sqrt(6.0 / (n_in + n_out))
        else:
            bound = gain.get(layers[l].type_activation_function, 1.0) * math.sqrt(6.0 / (n_in + n_out))
        p[a:b].uniform_(-bound, bound, generator=gen)
    p[net.W + net.n_bias:net.W + net.n_bias + net.n_norm] = 1.0
    return p


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def _upload(net, which, values):
    host = _pinned(values.numel())
    host.copy_(values)
    net._ck(net.lib.myea_b200_upload(net.h, which, host.data_ptr(), 0, host.numel()), "upload")


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    layers, desc, opt = _network(c)
    net = Net(desc, opt)
    _upload(net, capi.BUF_PARAMETERS, _initial_parameters(net, layers, gen))
    if net.n_norm:
        _upload(net, capi.BUF_NORM_VARIANCE_AVERAGE, torch.ones(net.n_norm * net.T))
    if c["decay"]:   # weights decay, biases and normalization parameters do not
        mask = torch.zeros(net.P)
        mask[:net.W] = 1.0
        _upload(net, capi.BUF_MASK_REGULARIZED, mask)
    state = {"case": c, "net": net, "opt": opt, "seed": seed % 1000003 + 1, "step": 0,
             "masks": c["dropout"] != "none" or c["zoneout"] > 0 or c["kind"] == "residual", "last": len(layers) - 1}
    T, B, n = c["time"], c["batch"], c["steps"]

    def batches(units, kind, count):
        """`count` batches [T, B, units] of inputs (standard normal) or targets (normal or one-hot)"""
        if kind == "labels":
            lab = torch.randint(units, (count, T, B), generator=gen, device="cuda")
            return torch.nn.functional.one_hot(lab, units).float()
        return torch.randn((count, T, B, units), generator=gen, device="cuda")

    X = batches(c["inputs"], "normal", n if c["mode"] != "predict" else 1)
    Y = batches(c["outputs"], "labels" if c["loss"] == "ce" else "normal", n) if c["mode"] != "predict" else None
    if c["mode"] == "epoch":
        # example-major rows [T * width], shuffled by the host
        xs = X.permute(0, 2, 1, 3).reshape(n * B, -1).contiguous().cpu()
        ys = Y.permute(0, 2, 1, 3).reshape(n * B, -1).contiguous().cpu()
        net._ck(net.lib.myea_b200_dataset_set(net.h, n * B, xs.data_ptr(), ys.data_ptr()), "dataset_set")
        state["order"] = torch.randperm(n * B, generator=gen, device="cuda").cpu().numpy().astype("uint64")
    elif c["source"] == "host":
        state["X"] = [x.cpu().pin_memory() for x in X]
        state["Y"] = [y.cpu().pin_memory() for y in Y] if Y is not None else None
    else:
        state["X"], state["Y"] = list(X), list(Y) if Y is not None else None
    if c["mode"] == "predict":
        state["outputs"] = _pinned(T, B, c["outputs"])
    else:
        state["parameters"] = _pinned(net.P)
        state["moment"] = _pinned(net.P) if c["resume"] else None
        state["averages"] = _pinned(2, net.n_norm * net.T) if net.n_norm else None
    net.synchronize()
    return state


def _train(state):
    """the training sequence on each of the state's batches; (loss sum, loss terms, accuracy hits)"""
    c, net, opt = state["case"], state["net"], state["opt"]
    lib, h, B = net.lib, net.h, c["batch"]
    host = c["source"] == "host"
    forward, error = (lib.myea_b200_forward, lib.myea_b200_compute_error) if host else (lib.myea_b200_forward_device, lib.myea_b200_compute_error_device)
    net.reset_loss()
    loss = None
    for x, y in zip(state["X"], state["Y"]):
        if state["masks"]:
            net.generate_masks(state["seed"], state["step"])
        state["step"] += 1
        net._ck(forward(h, B, x.data_ptr(), 1), "forward")
        net._ck(error(h, B, y.data_ptr()), "compute_error")
        net._ck(lib.myea_b200_backward(h, B), "backward")
        net._ck(lib.myea_b200_update_derivative_weight(h, B), "update_derivative_weight")
        net._ck(lib.myea_b200_update_parameter(h, B, B * c["steps"], C.byref(opt)), "update_parameter")
        if host:
            loss = net.loss()
    return loss or net.loss()


def run(state):
    c, net = state["case"], state["net"]
    lib, h = net.lib, net.h
    if c["mode"] == "predict":
        x, out = state["X"][0], state["outputs"]
        forward = lib.myea_b200_forward if c["source"] == "host" else lib.myea_b200_forward_device
        net._ck(forward(h, c["batch"], x.data_ptr(), 0), "forward")
        net._ck(lib.myea_b200_get_outputs(h, state["last"], out.data_ptr(), out.numel()), "get_outputs")
        return {"outputs": out}
    if c["mode"] == "epoch":
        loss = net.train_epoch(state["order"], c["batch"], mask_seed=state["seed"] if state["masks"] else 0, first_step=state["step"])
        state["step"] += c["steps"]
    else:
        loss = _train(state)
    got = {"loss": float(loss[0]), "hits": float(loss[-1])}
    wanted = [("parameters", capi.BUF_PARAMETERS, state["parameters"])]
    if state["moment"] is not None:
        wanted.append(("moment", capi.BUF_PREVIOUS_DELTA if c["optimizer"] == "nesterov" else capi.BUF_FIRST_MOMENT, state["moment"]))
    if state["averages"] is not None:
        wanted += [("mean", capi.BUF_NORM_MEAN_AVERAGE, state["averages"][0]), ("deviation", capi.BUF_NORM_VARIANCE_AVERAGE, state["averages"][1])]
    for name, which, host in wanted:
        net._ck(lib.myea_b200_download(h, which, host.data_ptr(), 0, host.numel()), "download")
        got[name] = host
    return got
