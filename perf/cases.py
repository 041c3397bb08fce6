"""The work that users of this framework have it do, as timed cases: whole training steps of the five workloads through
``DataParallelTrainer`` (captured once, replayed per step, fed the three ways the trainer can be fed), the same kind of model
written op by op against the eager engine (training step and evaluation), and the C ABI called directly on the caller's own
device buffers (products with their gradients, optimizer steps over a whole model).

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges; ``prepare`` / ``run`` / ``work`` / ``tolerance`` take a
case.  All data is fp32, the only type the framework computes in.
"""
import ctypes as C
import math

import numpy as np
import torch

import rusttensor_b200 as rt
from rusttensor_b200.capi import CApi
from rusttensor_b200.workloads import kaiming_uniform, one_hot

CONFIG = {"mlp": 1, "elementwise": 2, "cnn": 3, "conv": 4, "lstm": 5}  # workload numbers of the trainer; 100 + c: fused forward ops
OPTIMIZERS = {"sgd": 0, "adam": 1, "momentum": 2, "adagrad": 3}
MINIBATCHES = 4  # rows of an attached data set, in batches


def listed():
    return [
        # A small classifier's training step, a new host batch uploaded for every step: launches and the upload are what counts.
        dict(name="mlp_step", kind="mlp", fused=False, feed="pipelined", batch=64, inputs=784, hidden=128, classes=10),
        # The same with the data set on the device, a large and uneven batch and the fused forward ops.
        dict(name="mlp_dataset", kind="mlp", fused=True, feed="dataset", batch=1000, inputs=784, hidden=300, classes=10),
        # The convolutional classifier at the batch size that it is benchmarked at, batches uploaded.
        dict(name="cnn_step", kind="cnn", fused=False, feed="pipelined", batch=256, hw=28, c1=32, c2=64, fc=128, classes=10),
        # A smaller one with uneven channel counts, fused forward ops, data set on the device.
        dict(name="cnn_dataset", kind="cnn", fused=True, feed="dataset", batch=90, hw=20, c1=24, c2=40, fc=100, classes=10),
        # Convolution, pooling, transposed convolution at image-model sizes: dense contractions in both directions.
        dict(name="conv_step", kind="conv", fused=False, feed="resident", batch=128, cin=64, hw=56, cmid=128),
        # The character LSTM written from fundamental ops (how the reference's example is written): thousands of small calls.
        dict(name="lstm_step", kind="lstm", fused=False, feed="pipelined", vocab=65, hidden=512, seq=128, batch=64),
        # The same model from the fused ops, a smaller and uneven size.
        dict(name="lstm_fused", kind="lstm", fused=True, feed="pipelined", vocab=50, hidden=200, seq=60, batch=30),
        # A chain of elementwise ops with a broadcast operand and a reduction, forward and backward, on one large matrix.
        dict(name="elementwise_chain", kind="elementwise", fused=False, feed="resident", rows=4096, cols=4096),
        # A small regression model trained op by op from the eager engine: host work per op.
        dict(name="eager_step", kind="eager", batch=64, inputs=8, hidden=64, optimizer="adam"),
        # Evaluation of the convolutional classifier on a test batch, op by op, no gradients.
        dict(name="cnn_eval", kind="eval", batch=1000, hw=28, c1=32, c2=64, fc=128, classes=10),
        # A large product and its two gradients through the C ABI.
        dict(name="matmul_large", kind="matmul", m=4096, k=4096, n=4096),
        # One optimizer step over all tensors of a model, uneven tensor sizes.
        dict(name="adam_model", kind="optimizer", optimizer="adam", tensors=20, total=20000003),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cnn_dims(rng):
    return dict(hw=4 * rng.randint(4, 8), c1=rng.randint(8, 32), c2=rng.randint(16, 64), fc=rng.randint(32, 128), classes=rng.randint(5, 20))


def draw(rng):
    kind = rng.choice(["mlp", "cnn", "conv", "lstm", "elementwise", "eager", "eval", "matmul", "optimizer"])
    fused, feed = rng.random() < 0.5, rng.choice(["pipelined", "dataset"])
    if kind == "mlp":
        return dict(kind=kind, fused=fused, feed=feed, batch=_log(rng, 16, 2048), inputs=rng.randint(100, 1000),
                    hidden=_log(rng, 32, 1024), classes=rng.randint(5, 20))
    if kind == "cnn":
        return dict(kind=kind, fused=fused, feed=feed, batch=_log(rng, 16, 512), **_cnn_dims(rng))
    if kind == "conv":
        return dict(kind=kind, fused=fused, feed="resident", batch=_log(rng, 4, 128), cin=rng.randint(16, 64), hw=2 * rng.randint(7, 28),
                    cmid=rng.randint(32, 128))
    if kind == "lstm":
        return dict(kind=kind, fused=fused, feed="pipelined", vocab=rng.randint(30, 100), hidden=_log(rng, 64, 512), seq=_log(rng, 16, 96),
                    batch=_log(rng, 8, 64))
    if kind == "elementwise":
        return dict(kind=kind, fused=False, feed="resident", rows=_log(rng, 64, 4096), cols=_log(rng, 64, 4096))
    if kind == "eager":
        return dict(kind=kind, batch=_log(rng, 16, 1024), inputs=rng.randint(1, 64), hidden=_log(rng, 16, 256),
                    optimizer=rng.choice(sorted(OPTIMIZERS)))
    if kind == "eval":
        return dict(kind=kind, batch=_log(rng, 1, 2048), **_cnn_dims(rng))
    if kind == "matmul":
        return dict(kind=kind, m=_log(rng, 32, 4096), k=_log(rng, 32, 4096), n=_log(rng, 32, 4096))
    return dict(kind=kind, optimizer=rng.choice(sorted(OPTIMIZERS)), tensors=rng.randint(1, 40), total=_log(rng, 100000, 60000000))


# ---- what a program has in hand before the call -------------------------------------------------------------------------------


class _View:
    """A device buffer of the engine as torch sees it (no copy)."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (ptr, False), "version": 2}


def _pointer(tensor):
    out = C.c_void_p()
    tensor.engine._call("tensor_device_ptr", C.c_int64(tensor.handle), C.byref(out))
    return out.value


def _view(tensor):
    return torch.as_tensor(_View(_pointer(tensor), tensor.shape), device="cuda")


def _dims(c):
    names = {"mlp": "batch inputs hidden classes", "elementwise": "rows cols", "cnn": "batch hw c1 c2 fc classes",
             "conv": "batch cin hw cmid", "lstm": "vocab hidden seq batch"}[c["kind"]]
    return [c[n] for n in names.split()]


def _cnn_params(r, c):
    flat = c["c2"] * (c["hw"] // 4) ** 2
    return [kaiming_uniform(r, 9, (c["c1"], 1, 3, 3)), r.uniform(-0.1, 0.1, c["c1"]),
            kaiming_uniform(r, 9 * c["c1"], (c["c2"], c["c1"], 3, 3)), r.uniform(-0.1, 0.1, c["c2"]),
            kaiming_uniform(r, flat, (flat, c["fc"])), r.uniform(-0.1, 0.1, c["fc"]),
            kaiming_uniform(r, c["fc"], (c["fc"], c["classes"])), r.uniform(-0.1, 0.1, c["classes"])]


def _net_params(r, c):
    if c["kind"] == "mlp":
        return [kaiming_uniform(r, c["inputs"], (c["inputs"], c["hidden"])), r.uniform(-0.1, 0.1, c["hidden"]),
                kaiming_uniform(r, c["hidden"], (c["hidden"], c["classes"])), r.uniform(-0.1, 0.1, c["classes"])]
    if c["kind"] == "cnn":
        return _cnn_params(r, c)
    if c["kind"] == "conv":
        return [kaiming_uniform(r, 9 * c["cin"], (c["cmid"], c["cin"], 3, 3)), r.uniform(-0.1, 0.1, c["cmid"]),
                kaiming_uniform(r, 16 * c["cmid"], (c["cmid"], c["cin"], 4, 4)), r.uniform(-0.1, 0.1, c["cin"])]
    v, h = c["vocab"], c["hidden"]  # recurrent weights at the scale at which a trained LSTM is stable
    return [r.uniform(-1, 1, (v + h, 4 * h)) / math.sqrt(h), r.uniform(-0.1, 0.1, 4 * h), kaiming_uniform(r, h, (h, v)), r.uniform(-0.1, 0.1, v)]


def _rows(r, c, rows):
    """Host arrays of `rows` samples for the workloads that are fed batches."""
    if c["kind"] == "mlp":
        return [r.random((rows, c["inputs"]), dtype=np.float32), one_hot(r, rows, c["classes"])]
    if c["kind"] == "cnn":
        return [r.random((rows, 1, c["hw"], c["hw"]), dtype=np.float32), one_hot(r, rows, c["classes"])]
    return [one_hot(r, rows, c["vocab"]), one_hot(r, rows, c["vocab"])]  # lstm: time-major characters and their successors


def _prepare_trainer(c, seed):
    """A trainer in the middle of training: parameters, optimizer moments and a step count as a resumed run has them."""
    r = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    tr = rt.DataParallelTrainer(CONFIG[c["kind"]] + (100 if c["fused"] else 0), _dims(c))
    s = {"trainer": tr, "feed": c["feed"]}
    if c["kind"] == "elementwise":
        for p in tr.params:
            _view(p).normal_(generator=g)
    else:
        for p, a in zip(tr.params, _net_params(r, c)):
            p.update_from_host(a)
    if tr.optimizer_kind:
        for i, p in enumerate(tr.params):
            tr.set_state(0, i, 1e-3 * r.standard_normal(p.shape, dtype=np.float32))
            if tr.optimizer_kind == 1:
                tr.set_state(1, i, 1e-5 * r.uniform(0.5, 2, p.shape))
        tr.step_count = 100
    if c["feed"] == "resident":
        for x in tr.inputs:
            _view(x).normal_(generator=g)
    elif c["feed"] == "pipelined":
        n = c["seq"] * c["batch"] if c["kind"] == "lstm" else c["batch"]
        s["batches"] = [_rows(r, c, n) for _ in range(MINIBATCHES)]
    else:
        n = MINIBATCHES * c["batch"]
        tr.attach_dataset(_rows(r, c, n))
        s["batches"] = np.split(r.permutation(n), MINIBATCHES)
    torch.cuda.synchronize()
    tr.capture()
    s["loss"] = tr.loss_tensor()
    s["out"] = [_view(s["loss"])] + [_view(p) for p in tr.params]
    if c["kind"] == "elementwise":
        s["out"] = s["out"][:1] + [_view(p.grad) for p in tr.params]
    elif c["kind"] == "conv":
        s["out"].append(_view(tr.inputs[0].grad))
    if tr.optimizer_kind:
        for which in range(2 if tr.optimizer_kind == 1 else 1):
            s["out"] += [_view(tr.state(which, i)) for i in range(len(tr.params))]
    return s


def _run_trainer(s):
    tr = s["trainer"]
    if s["feed"] == "resident":
        tr.step()
        return s["out"]
    k = s["at"] = (s.get("at", -1) + 1) % MINIBATCHES
    if s["feed"] == "pipelined":
        for i, a in enumerate(s["batches"][k]):
            np.copyto(tr.pipeline_buffer(i), a)
        tr.step_pipelined()
    else:
        tr.step_dataset(s["batches"][k])
    return s["out"]


def _views(s, tensors):
    """Torch views of tensors that the pass has made; kept per address, since the engine's allocator hands out the same ones again."""
    s["keep"] = tensors
    out = []
    for i, t in enumerate(tensors):
        key = (i, _pointer(t))
        if key not in s["views"]:
            s["views"][key] = _view(t)
        out.append(s["views"][key])
    return out


def _prepare_eager(c, seed):
    r = np.random.default_rng(seed)
    eng = rt.engine()
    h = c["hidden"]
    shapes = [(c["inputs"], h), (h,), (h, h), (h,), (h, 1), (1,)]
    params = [eng.tensor(r.uniform(-1, 1, s) / math.sqrt(s[0]), requires_grad=True) for s in shapes]
    x = r.uniform(-2, 2, (c["batch"], c["inputs"]))
    make = {"sgd": lambda p: eng.Sgd(p, 0.01), "adam": lambda p: eng.Adam(p, 1e-3), "momentum": lambda p: eng.MomentumSGD(p, 0.01, 0.9),
            "adagrad": lambda p: eng.AdaGrad(p, 0.01)}[c["optimizer"]]
    return {"params": params, "x": eng.tensor(x), "y": eng.tensor(np.sin(x.sum(1, keepdims=True))), "ops": eng.ops, "optimizer": make(params), "views": {}}


def _run_eager(s):
    ops, (w1, b1, w2, b2, w3, b3) = s["ops"], s["params"]
    h = ops.tanh(ops.add(ops.matmul(s["x"], w1), b1))
    h = ops.tanh(ops.add(ops.matmul(h, w2), b2))
    loss = ops.mse_loss(ops.add(ops.matmul(h, w3), b3), s["y"])
    s["optimizer"].zero_grad()
    loss.backward()
    grads = [p.grad for p in s["params"]]
    s["optimizer"].step()
    return _views(s, [loss] + grads + s["params"])


def _prepare_eval(c, seed):
    r = np.random.default_rng(seed)
    eng = rt.engine()
    x = eng.tensor(r.random((c["batch"], 1, c["hw"], c["hw"]), dtype=np.float32))
    return {"params": [eng.tensor(p) for p in _cnn_params(r, c)], "x": x, "ops": eng.ops, "flat": (c["batch"], c["c2"] * (c["hw"] // 4) ** 2), "views": {}}


def _run_eval(s):
    ops, (c1, d1, c2, d2, w1, b1, w2, b2) = s["ops"], s["params"]
    h = s["x"]
    for w, b in ((c1, d1), (c2, d2)):
        h = ops.max_pool2d(ops.relu(ops.conv2d(h, w, b, (1, 1), (1, 1))), (2, 2), (2, 2), (0, 0))
    h = ops.relu(ops.add(ops.matmul(ops.view(h, s["flat"]), w1), b1))
    return _views(s, [ops.log_softmax(ops.add(ops.matmul(h, w2), b2), 1)])


def _api():
    return CApi(ctx=rt.context_handle())


def _p(t):
    return C.c_void_p(t.data_ptr())


def _prepare_matmul(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    m, k, n = c["m"], c["k"], c["n"]
    a, b, up = (torch.randn(s, generator=g, device="cuda") for s in ((m, k), (k, n), (m, n)))
    out = y, da, db = torch.empty(m, n, device="cuda"), torch.empty(m, k, device="cuda"), torch.empty(k, n, device="cuda")
    i = C.c_int64
    forward = (0, 0, i(m), i(n), i(k), _p(a), i(k), _p(b), i(n), _p(y), i(n), 0)
    backward = (_p(a), _p(b), _p(up), i(m), i(k), i(n), _p(da), _p(db))
    return {"api": _api(), "forward": forward, "backward": backward, "out": list(out), "keep": (a, b, up)}


def _run_matmul(s):
    s["api"].call("gemm", *s["forward"])
    s["api"].call("matmul_backward", *s["backward"])
    return s["out"]


def _sizes(c):
    """Uneven tensor sizes that add up to the total: a few large matrices, many small ones."""
    w = [1.0 / (1 + i) for i in range(c["tensors"])]
    sizes = [max(1, int(c["total"] * x / sum(w))) for x in w]
    sizes[0] += c["total"] - sum(sizes)
    return sizes


def _prepare_optimizer(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    sizes = _sizes(c)
    kind, n = OPTIMIZERS[c["optimizer"]], len(sizes)
    new = lambda scale: [scale * torch.randn(k, generator=g, device="cuda") for k in sizes]  # noqa: E731
    p, grad, s1, s2 = new(0.05), new(1e-2), new(1e-3), new(1e-3)
    if c["optimizer"] != "momentum":
        s2 = [t.square_() for t in s2]
        s1 = [t.square_() for t in s1] if c["optimizer"] == "adagrad" else s1
    lists = [(C.c_void_p * n)(*[t.data_ptr() for t in ts]) for ts in (p, grad, s1, s2)]
    f = C.c_float
    args = (kind, n, *lists, (C.c_int64 * n)(*sizes), f(1e-3), f(0.9), f(0.999), f(1e-8), f(0.9), C.c_int64(100), f(1.0), 0, f(0), f(0))
    out = p + (s1 if kind else []) + (s2 if kind == 1 else [])
    return {"api": _api(), "args": args, "out": out[:64], "keep": (p, grad, s1, s2)}


def _run_optimizer(s):
    s["api"].call("optimizer_step_multi", *s["args"])
    return s["out"]


_KINDS = {"eager": (_prepare_eager, _run_eager), "eval": (_prepare_eval, _run_eval), "matmul": (_prepare_matmul, _run_matmul),
          "optimizer": (_prepare_optimizer, _run_optimizer)}


def prepare(case, seed):
    make, step = _KINDS.get(case["kind"], (_prepare_trainer, _run_trainer))
    state = make(case, seed)
    state["step"] = step
    torch.cuda.synchronize()
    return state


def run(state):
    return state["step"](state)


# ---- what a pass cannot do without --------------------------------------------------------------------------------------------


def _conv_flops(c, backward):
    """The classifier with two 3x3 convolutions: multiply-adds x 2 of the forward pass, or of forward + gradients."""
    b, px = c["batch"], c["hw"] ** 2
    first, second = 2 * b * px * 9 * c["c1"], 2 * b * (px // 4) * 9 * c["c1"] * c["c2"]
    dense = 2 * b * (c["c2"] * (px // 16) * c["fc"] + c["fc"] * c["classes"])
    return 2 * first + 3 * (second + dense) if backward else first + second + dense


def work(case):
    c, kind = case, case["kind"]
    if kind == "optimizer":
        words, flops = {"sgd": (3, 2), "adam": (7, 12), "momentum": (5, 4), "adagrad": (5, 6)}[c["optimizer"]]
        return {"bytes": 4 * words * c["total"], "flops": flops * c["total"]}
    if kind == "matmul":
        m, k, n = c["m"], c["k"], c["n"]
        return {"bytes": 4 * (2 * m * k + 2 * k * n + 2 * m * n), "flops": 6 * m * k * n}
    if kind == "elementwise":
        n = c["rows"] * c["cols"]
        return {"bytes": 4 * (2 * n + 2 * c["cols"]), "flops": 40 * n}
    if kind == "conv":
        b, px, ch = c["batch"], c["hw"] ** 2, c["cin"] * c["cmid"]
        p = ch * 25 + c["cmid"] + c["cin"]  # momentum: parameter and velocity read and written
        return {"bytes": 4 * (3 * b * c["cin"] * px + 4 * p), "flops": 6 * b * px * ch * 9 + 6 * b * (px // 4) * ch * 16}
    if kind == "eager":
        h = c["hidden"]
        p = c["inputs"] * h + h * h + 4 * h + 1
        return {"bytes": 4 * (c["batch"] * (c["inputs"] + 1) + 7 * p), "flops": 2 * c["batch"] * (2 * c["inputs"] * h + 3 * h * h + 3 * h)}
    if kind == "eval":
        p = c["c1"] * 10 + c["c2"] * (9 * c["c1"] + 1) + c["c2"] * (c["hw"] // 4) ** 2 * c["fc"] + c["fc"] * (c["classes"] + 1)
        return {"bytes": 4 * (c["batch"] * (c["hw"] ** 2 + c["classes"]) + p), "flops": _conv_flops(c, False)}
    # Adam: parameter and both moments read and written
    if kind == "mlp":
        b, i, h, o = c["batch"], c["inputs"], c["hidden"], c["classes"]
        return {"bytes": 4 * (b * (i + o) + 6 * (i * h + h + h * o + o)), "flops": 2 * b * (2 * i * h + 3 * h * o)}
    if kind == "cnn":
        p = c["c1"] * 10 + c["c2"] * (9 * c["c1"] + 1) + c["c2"] * (c["hw"] // 4) ** 2 * c["fc"] + c["fc"] * (c["classes"] + 1) + c["classes"]
        return {"bytes": 4 * (c["batch"] * (c["hw"] ** 2 + c["classes"]) + 6 * p), "flops": _conv_flops(c, True)}
    v, h, rows = c["vocab"], c["hidden"], c["seq"] * c["batch"]
    p = (v + h + 1) * 4 * h + (h + 1) * v
    return {"bytes": 4 * (2 * rows * v + 6 * p), "flops": 2 * rows * (4 * h * (2 * v + 3 * h) + 3 * h * v)}


def tolerance(case):
    kind = case["kind"]
    if kind == "optimizer":
        return {"rel": 2e-6, "max": 1e-4}
    if kind == "matmul":  # 3xTF32: each product to about 2^-21, fp32 accumulation
        return {"rel": 1e-5, "max": 1e-4}
    if kind in ("elementwise", "eval"):
        return {"rel": 2e-5, "max": 1e-3}
    if kind in ("cnn", "conv"):
        # relu and max-pooling select: of the hundreds of thousands of windows a few have two candidates (or a winner and zero) that
        # are equal to within rounding, and the gradient of such a window goes to one position or the other
        return {"rel": 1e-3, "max": 0.5}
    if kind in ("lstm", "mlp"):  # the gradients of a hundred timesteps; a relu input may lie within rounding of zero
        return {"rel": 1e-4, "max": 5e-2}
    return {"rel": 1e-4, "max": 2e-2}  # eager: Adam divides by the root of young second moments
