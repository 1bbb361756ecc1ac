"""What a user of this framework has it do: training runs, training windows, inference and table standardisation.

A case is a dict of plain values.  Every case runs through the package's public entry points (glades-ml_b200/capi.py
and include/glades_b200.h).  Network shapes, activations, learning rates and batch sizes come from the
repository's benchmark configurations, or are generic; data is synthetic, made from the seed.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

g = importlib.import_module("glades-ml_b200")

DEV = "cuda:0"


# ---- cases ------------------------------------------------------------------------------------------------
def listed():
    return [
        # the tiny tabular classifier: online SGD in the reference's own arithmetic, 150 rows; the shortest training
        # runs there are, one sample after the other
        dict(name="tiny_classifier", kind="reference", net="4-16-3", act="sigmoid", head="sigmoid", out="classification",
             rows=150, batch=1, epochs=10, lr=0.001, momentum=0.9),
        # parity of ten bits, minibatches of 32: a small network trained for many epochs in one call
        dict(name="parity_net", kind="epochs", net="10-32-32-1", act="tanh", head="sigmoid", out="regression", rows=1024,
             batch=32, epochs=20, lr=0.05, momentum=0.0),
        # an ordinary tabular classifier with odd sizes and a short last minibatch
        dict(name="tabular_classifier", kind="epochs", net="57-200-90-7", act="relu", head="softmax", out="classification",
             rows=10007, batch=250, epochs=1, lr=0.05, momentum=0.9),
        # one epoch of the time-series window regressor, momentum and 1024-row minibatches
        dict(name="window_regressor", kind="epochs", net="32-256-256-1", act="relu", head="linear", out="regression",
             rows=131072, batch=1024, epochs=1, lr=1e-3, momentum=0.9),
        # one epoch over image-shaped rows, sizes that people choose by hand (none a multiple of a tile), a short last
        # minibatch, momentum
        dict(name="digits_classifier", kind="epochs", net="784-1000-500-10", act="relu", head="softmax",
             out="classification", rows=20300, batch=1000, epochs=1, lr=0.05, momentum=0.9),
        # the wide teacher-student network: sixteen 8192-row windows, then the weights are read
        dict(name="wide_mlp", kind="windows", net="1024-4096-4096-1024", act="relu", head="softmax", out="classification",
             window=8192, count=16, lr=1e-2, momentum=0.0),
        # the same network with an eighth of the window: what one of eight GPUs computes
        dict(name="wide_mlp_small_window", kind="windows", net="1024-4096-4096-1024", act="relu", head="softmax",
             out="classification", window=1024, count=32, lr=1e-2, momentum=0.0),
        # the same training fed from host memory, two windows in flight
        dict(name="wide_mlp_from_host", kind="stream", net="1024-4096-4096-1024", act="relu", head="softmax",
             out="classification", window=8192, count=8, lr=1e-2, momentum=0.0),
        # batched inference over rows that lie on the GPU: class and probabilities come back
        dict(name="batched_inference", kind="infer", net="784-2048-2048-10", act="relu", head="softmax",
             out="classification", rows=65536),
        # the same network asked for one row from host memory: the latency of a single request
        dict(name="single_request", kind="serve", net="784-2048-2048-10", act="relu", head="softmax",
             out="classification", rows=1),
        # standardisation of the window regressor's raw table, min-max
        dict(name="standardize_minmax", kind="standardize", rows=1 << 20, cols=33, categorical=0, zscore=0),
        # standardisation of a mixed table, z-score, some columns one-hot encoded
        dict(name="standardize_zscore", kind="standardize", rows=100003, cols=24, categorical=5, zscore=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A layer's width: a multiple of 128, a multiple of 8, or any number."""
    n, how = _log(rng, lo, hi), rng.randrange(3)
    if how < 2:
        m = 128 if how == 0 and n >= 128 else 8
        n = max(m, int(round(n / m)) * m)
    return max(lo, min(hi, n))


def _net(*sizes):
    return "-".join(str(s) for s in sizes)


def draw(rng):
    kind = rng.choice(["reference", "small", "middle", "large", "windows", "stream", "infer", "serve", "standardize"])
    act = rng.choice(["relu", "relu", "tanh", "sigmoid"])
    if kind == "reference":
        # one or two hidden layers; what follows a hidden layer stays narrow (the reference doubles a node's error once
        # for each node above it)
        hidden = [_log(rng, 4, 64)] + ([_log(rng, 3, 8)] if rng.random() < 0.5 else [])
        rows = _log(rng, 50, 1000)
        return dict(kind="reference", net=_net(_log(rng, 2, 32), *hidden, rng.randint(2, 4)), act=rng.choice(["sigmoid", "tanh"]),
                    head="sigmoid", out=rng.choice(["classification", "regression"]), rows=rows, batch=rng.choice([1, 1, 8, 32]),
                    epochs=max(1, min(10, 2000 // rows)), lr=0.001, momentum=rng.choice([0.0, 0.9]))
    if kind in ("small", "middle", "large"):
        if kind == "small":
            sizes = [_log(rng, 4, 64)] + [_log(rng, 8, 64) for _ in range(rng.randint(1, 2))]
            rows, batch, epochs = _log(rng, 200, 4000), _log(rng, 16, 128), rng.randint(1, 10)
        elif kind == "middle":
            sizes = [_width(rng, 16, 256)] + [_width(rng, 64, 512) for _ in range(rng.randint(1, 2))]
            rows, batch, epochs = _log(rng, 4000, 131072), _log(rng, 64, 2048), 1
        else:
            sizes = [_width(rng, 256, 1024)] + [_width(rng, 500, 2048) for _ in range(2)]
            rows, batch, epochs = _log(rng, 8000, 32768), _log(rng, 256, 4096), 1
        softmax = rng.random() < 0.6
        sizes.append(rng.randint(2, 16) if softmax else rng.randint(1, 4))
        return dict(kind="epochs", net=_net(*sizes), act=act, head="softmax" if softmax else "linear",
                    out="classification" if softmax else "regression", rows=rows, batch=min(batch, rows), epochs=epochs,
                    lr=0.02 if softmax else 1e-3, momentum=rng.choice([0.0, 0.9]))
    if kind in ("windows", "stream"):
        net = _net(_width(rng, 256, 1024), _width(rng, 1024, 4096), _width(rng, 1024, 4096), _width(rng, 64, 1024))
        window = _log(rng, 256, 8192)
        return dict(kind=kind, net=net, act=act, head="softmax", out="classification", window=window,
                    count=max(2, min(16, 32768 // window)), lr=1e-2, momentum=rng.choice([0.0, 0.0, 0.9]))
    if kind in ("infer", "serve"):
        net = _net(_width(rng, 64, 1024), _width(rng, 256, 2048), _width(rng, 256, 2048), rng.randint(2, 64))
        return dict(kind=kind, net=net, act=act, head="softmax", out="classification",
                    rows=_log(rng, 1024, 65536) if kind == "infer" else _log(rng, 1, 256))
    cols = _log(rng, 4, 96)
    zscore = rng.randrange(2)
    return dict(kind="standardize", rows=_log(rng, 10000, 200000 if zscore else 1 << 20), cols=cols,
                categorical=rng.choice([0, cols // 4]), zscore=zscore)


# ---- inputs -----------------------------------------------------------------------------------------------
def _sizes(case):
    return [int(s) for s in case["net"].split("-")]


class State:
    """What the program keeps between calls: the network's handle and the tensors it works on."""


def _network(case, gen, mode, batch):
    """A network with seeded weights: uniform, scaled by fan-in as a user would start a training run."""
    sizes = _sizes(case)
    layers = len(sizes) - 1
    acts = [case["act"]] * (layers - 1) + [case["head"]]
    desc = g.make_desc(sizes, acts, case["out"], batch=batch, lr=case.get("lr", 0.0), momentum=case.get("momentum", 0.0),
                       params=[0.01] * (layers - 1) + [1.0], mode=mode)
    net = g.Net(desc)
    w = torch.cat([(torch.rand(o * i, generator=gen, device=DEV) * 2 - 1) * math.sqrt(1.5 / i) for i, o in zip(sizes, sizes[1:])])
    b = (torch.rand(layers - 1, generator=gen, device=DEV) * 2 - 1) * 0.05
    net.set_weights(w.cpu().numpy(), b.cpu().numpy())
    return net


def _rows(case, gen, rows, n_in, n_out):
    """Inputs and expected rows.  Classes come from a seeded linear teacher (one-hot rows, 0.99 / 0.01 under the sigmoid head
    as the one-hot encoder writes them), regression targets from the same teacher squashed into (0, 1)."""
    x = torch.randn(rows, n_in, generator=gen, device=DEV)
    teacher = torch.randn(n_in, n_out, generator=gen, device=DEV) / math.sqrt(n_in)
    score = x @ teacher
    if case["out"] == "regression":
        return x, torch.sigmoid(score)
    on, off = (1.0, 0.0) if case["head"] == "softmax" else (0.99, 0.01)
    y = torch.full((rows, n_out), off, device=DEV)
    y.scatter_(1, score.argmax(1, keepdim=True), on)
    return x, y


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    s = State()
    s.case, s.kind = case, case["kind"]
    if s.kind == "standardize":
        return _prepare_table(s, case, gen)
    sizes = _sizes(case)
    if s.kind in ("infer", "serve"):
        s.net = _network(case, gen, g.MODE_BATCHED, case["rows"])
        s.x = torch.rand(case["rows"], sizes[0], generator=gen, device=DEV)  # pixel-like values
        if s.kind == "serve":
            s.x = s.x.cpu().numpy()
        else:
            s.net.set_data_device(s.x.data_ptr(), 0, case["rows"])
        torch.cuda.synchronize()
        return s
    if s.kind in ("reference", "epochs"):
        rows, batch = case["rows"], case["batch"]
    else:
        rows, batch = case["window"] * case["count"], case["window"]
    s.net = _network(case, gen, g.MODE_REFERENCE if s.kind == "reference" else g.MODE_BATCHED, batch)
    if s.kind == "stream":
        # pinned host windows that a data loader would fill in turn
        s.host = []
        for _ in range(min(4, case["count"])):
            x, y = _rows(case, gen, batch, sizes[0], sizes[-1])
            s.host.append((x.cpu().pin_memory().numpy(), y.cpu().pin_memory().numpy()))
    else:
        s.x, s.y = _rows(case, gen, rows, sizes[0], sizes[-1])
        s.net.set_data_device(s.x.data_ptr(), s.y.data_ptr(), rows)
    torch.cuda.synchronize()
    return s


def _prepare_table(s, case, gen):
    """A raw table in device memory: numeric columns of mixed scales, categorical ones as category indices."""
    rows, cols, ncat = case["rows"], case["cols"], case["categorical"]
    s.raw = torch.randn(rows, cols, generator=gen, device=DEV) * torch.linspace(0.5, 40.0, cols, device=DEV) + 3.0
    kind, classes, outs = np.zeros(cols, np.int32), np.zeros(cols, np.int32), np.zeros(cols, np.int32)
    for k in range(ncat):
        c = k * (cols // max(1, ncat))
        kind[c], classes[c] = 1, 2 + k % 11
        s.raw[:, c] = torch.randint(0, int(classes[c]), (rows,), generator=gen, device=DEV).float()
    outs[-1] = 1
    s.plan = (kind, classes, outs)
    s.nx, s.ny = ctypes.c_int32(), ctypes.c_int32()
    torch.cuda.synchronize()
    _standardize(s, None, None, None)
    s.x = torch.empty(rows, s.nx.value, device=DEV)
    s.y = torch.empty(rows, s.ny.value, device=DEV)
    return s


# ---- one pass -----------------------------------------------------------------------------------------------
def _standardize(s, x, y, stats):
    at = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    st = g.lib().gl_standardize_table(s.raw.data_ptr(), s.case["rows"], s.case["cols"], at(s.plan[0]), at(s.plan[1]), at(s.plan[2]),
                                      s.case["zscore"], x.data_ptr() if x is not None else None, ctypes.byref(s.nx),
                                      y.data_ptr() if y is not None else None, ctypes.byref(s.ny),
                                      at(stats) if stats is not None else None, 0)
    if st != 0:
        raise g.GladesError(st, g.lib().gl_last_error().decode())


def run(s):
    c, kind = s.case, s.kind
    if kind == "standardize":
        stats = np.zeros((c["cols"], 4), np.float32)
        _standardize(s, s.x, s.y, stats)
        return dict(x=s.x, y=s.y, stats=stats)
    if kind == "infer":
        out, cls, _ = s.net.forward(0, c["rows"])
        return dict(probabilities=out, classes=cls)
    if kind == "serve":
        out, cls, _ = s.net.forward_host(s.x)
        return dict(probabilities=out, classes=cls)
    if kind in ("reference", "epochs"):
        m = s.net.train_epochs(c["epochs"])
    elif kind == "windows":
        for k in range(c["count"] - 1):
            s.net.train_window(k * c["window"], c["window"], want_metrics=False)
        m = s.net.train_window((c["count"] - 1) * c["window"], c["window"])
    else:
        for k in range(c["count"]):
            if k >= 2:
                m = s.net.window_result()
            s.net.submit_window_host(*s.host[k % len(s.host)])
        for _ in range(min(2, c["count"])):
            m = s.net.window_result()
    w, b = s.net.get_weights()
    out = dict(weights=w, bias=b, error=m.total_error, accuracy=m.total_accuracy)
    if kind == "reference":
        out["last"] = s.net.last_outputs()
        if c["out"] == "classification":
            out["confusion"] = s.net.confusion()
    return out


# ---- what a pass cannot do without ------------------------------------------------------------------------
def work(case):
    if case["kind"] == "standardize":
        rows, cols, ncat = case["rows"], case["cols"], case["categorical"]
        wide = sum(2 + k % 11 for k in range(ncat))
        return {"bytes": 4.0 * rows * (cols + cols - ncat + wide), "flops": 3.0 * rows * (cols - ncat)}
    sizes = _sizes(case)
    weights = sum(i * o for i, o in zip(sizes, sizes[1:]))
    if case["kind"] in ("infer", "serve"):
        return {"bytes": 4.0 * (case["rows"] * (sizes[0] + sizes[-1] + 1) + weights), "flops": 2.0 * weights * case["rows"]}
    if case["kind"] in ("reference", "epochs"):
        rows, samples = case["rows"], case["rows"] * case["epochs"]
    else:
        rows = samples = case["window"] * case["count"]
    # forward, error propagation (not into the inputs) and weight gradient
    return {"bytes": 4.0 * (rows * (sizes[0] + sizes[-1]) + 2 * weights),
            "flops": float(samples) * (6.0 * weights - 2.0 * sizes[0] * sizes[1])}


def tolerance(case):
    if case["kind"] in ("reference", "standardize"):
        return "exact"  # these reproduce a fixed order of separately rounded fp32 operations, bit for bit
    if case["kind"] in ("infer", "serve"):
        return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}  # fp32 sums in any order; a class may change where two are level
    # fp32 sums in any order, carried through a run of updates; the activations' threshold may fall either way for single rows
    return {"rel": 2e-5, "max": 2e-3}
