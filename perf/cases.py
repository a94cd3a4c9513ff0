"""The work this framework is used for, as measurable cases.

Seven kinds of work, each through the public entry points (vtl_b200.capi.Device, vtl_b200.host.Session / Model /
DataLoader):

  int8_linear   one quantised Linear forward: dynamic row quantisation of f32 activations, INT8 product, fused
                dequantisation + bias (+ ReLU)
  int8_mlp      INT8 MLP inference: wide and narrow layers in turn, row maxima handed from layer to layer
  mlp_fit       steps of a small MLP on one batch that stays, then the weights read back (Model.train_step)
  mlp_epoch     one epoch over a device-resident dataset: shuffled batches, BatchNorm1D, any optimizer
  f32_step      one AdamW training step of a deep f32 MLP through the device entry points
  cnn_fit       steps of a small CNN, then the weights read back (Model.train_step)
  conv_layer    one convolution layer, forward and backward
  checkpoint    parameters to checkpoint text and back
"""
import numpy as np
import torch

from vtl_b200 import capi, host

_session = None


def _ses():
    """The one Session (and device context) of the process, as a program keeps it."""
    global _session
    if _session is None:
        _session = host.Session(0)
    return _session


def _dev():
    return _ses().dev


# ---------------------------------------------------------------- the cases
def listed():
    mlp = {"kind": "int8_mlp", "d": 8192, "h": 28672, "layers": 4}
    return [
        # a single token through one quantised layer: launch latency, and 16 MiB of weights read once
        {"name": "int8_linear_1row", "kind": "int8_linear", "m": 1, "n": 4096, "k": 4096, "relu": True},
        # sizes that nothing divides: a batch of 999 rows, 2047 inputs, 3001 outputs
        {"name": "int8_linear_odd", "kind": "int8_linear", "m": 999, "n": 3001, "k": 2047, "relu": False},
        # the benchmark's headline: 4096 rows, 4096 inputs and outputs
        {"name": "int8_linear_4096", "kind": "int8_linear", "m": 4096, "n": 4096, "k": 4096, "relu": True},
        # decoding for eight users at once: 0.94 GB of weights read once for a few rows
        {"name": "int8_mlp_decode8", "m": 8, **mlp},
        # the benchmark's inference batch (prefill): 16384 tokens
        {"name": "int8_mlp_16384", "m": 16384, **mlp},
        # the smallest training run: 784-256-10, batch 64, Adam, mean squared error
        {"name": "mlp_fit_784_256_10", "kind": "mlp_fit", "batch": 64, "in": 784, "hidden": 256, "out": 10, "depth": 1,
         "steps": 30},
        # an ordinary classifier on features: 20 shuffled batches with BatchNorm and softmax cross-entropy
        {"name": "mlp_epoch_bn", "kind": "mlp_epoch", "rows": 5120, "batch": 256, "in": 600, "hidden": 512, "out": 100,
         "opt": "adamw"},
        # one eighth of the benchmark's data-parallel batch: 8 layers of width 4096, 8192 rows
        {"name": "f32_step_4096", "kind": "f32_step", "rows": 8192, "width": 4096, "layers": 8},
        # the benchmark's CNN on 32 x 32 colour images, batch 256
        {"name": "cnn_fit_32x32", "kind": "cnn_fit", "batch": 256, "c": 3, "hw": 32, "o1": 32, "o2": 64, "k": 3, "pad": 1,
         "pool1": False, "hidden": 0, "steps": 10},
        # grey 28 x 28 images, channel counts and planes that no tile divides, a hidden Linear, batch 50
        {"name": "cnn_fit_28x28", "kind": "cnn_fit", "batch": 50, "c": 1, "hw": 28, "o1": 20, "o2": 50, "k": 5, "pad": 0,
         "pool1": True, "hidden": 500, "steps": 10},
        # a down-sampling layer: 3 x 3 with stride 2
        {"name": "conv_layer_stride2", "kind": "conv_layer", "batch": 32, "c": 64, "hw": 56, "o": 128, "k": 3, "pad": 1,
         "stride": 2},
        # a model of 16 million parameters written as a checkpoint and read again
        {"name": "checkpoint_16M", "kind": "checkpoint", "n": 16777213},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of lo..hi; one in three rounded to a multiple of 32 (where it is large)."""
    v = int(round(lo * (hi / lo) ** rng.random()))
    if v >= 64 and rng.random() < 1 / 3:
        v = v // 32 * 32
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["int8_linear", "int8_linear", "int8_mlp", "mlp_fit", "mlp_epoch", "f32_step", "cnn_fit", "conv_layer",
                       "checkpoint"])
    if kind == "int8_linear":
        return {"kind": kind, "m": _log(rng, 1, 8192), "n": _log(rng, 128, 8192), "k": _log(rng, 128, 8192),
                "relu": rng.random() < 0.5}
    if kind == "int8_mlp":
        d = 128 * _log(rng, 8, 64)
        return {"kind": kind, "m": _log(rng, 1, 8192), "d": d, "h": d * 7 // 2, "layers": 2 * rng.randint(1, 2)}
    if kind == "mlp_fit":
        return {"kind": kind, "batch": _log(rng, 8, 256), "in": _log(rng, 16, 1024), "hidden": _log(rng, 16, 512),
                "out": _log(rng, 2, 32), "depth": rng.randint(1, 2), "steps": 30}
    if kind == "mlp_epoch":
        batch = _log(rng, 32, 512)
        return {"kind": kind, "rows": batch * rng.randint(8, 20) + rng.randint(0, batch - 1), "batch": batch,
                "in": _log(rng, 64, 1024), "hidden": _log(rng, 64, 1024), "out": _log(rng, 4, 200),
                "opt": rng.choice(["adam", "adamw", "sgd", "rmsprop"])}
    if kind == "f32_step":
        return {"kind": kind, "rows": _log(rng, 256, 8192), "width": _log(rng, 256, 4096), "layers": rng.randint(2, 8)}
    if kind == "cnn_fit":
        k = rng.choice([3, 5])
        return {"kind": kind, "batch": _log(rng, 16, 256), "c": rng.choice([1, 3, 4, 16]), "hw": rng.choice([20, 24, 28, 32]),
                "o1": _log(rng, 8, 32), "o2": _log(rng, 16, 64), "k": k, "pad": rng.choice([0, k // 2]),
                "pool1": rng.random() < 0.5, "hidden": rng.choice([0, 0, 100, 500]), "steps": 5}
    if kind == "conv_layer":
        k = rng.choice([1, 3, 5])
        return {"kind": kind, "batch": _log(rng, 4, 64), "c": _log(rng, 3, 64), "hw": _log(rng, 14, 56), "o": _log(rng, 8, 128),
                "k": k, "pad": rng.choice([0, k // 2]), "stride": rng.choice([1, 1, 2])}
    return {"kind": "checkpoint", "n": _log(rng, 1000, 33554432)}


# ---------------------------------------------------------------- sizes
def _cnn_dims(c):
    h1 = c["hw"] + 2 * c["pad"] - c["k"] + 1
    p1 = h1 // 2 if c["pool1"] else h1
    h2 = p1 + 2 * c["pad"] - c["k"] + 1
    return h1, p1, h2, h2 // 2


def _conv_out(c):
    return (c["hw"] + 2 * c["pad"] - c["k"]) // c["stride"] + 1


def work(c):
    """Bytes: inputs once, outputs once (weights, moments and activations handed back included).  Operations: the products."""
    k = c["kind"]
    if k == "int8_linear":
        m, n, kk = c["m"], c["n"], c["k"]
        return {"bytes": 5 * m * kk + 4 * m + n * kk + 8 * n + 4 * m * n, "flops": 2 * m * n * kk}
    if k == "int8_mlp":
        w = c["layers"] * c["d"] * c["h"]
        return {"bytes": w + 8 * c["m"] * c["d"], "flops": 2 * c["m"] * w}
    if k in ("mlp_fit", "mlp_epoch"):
        hid = [c["hidden"]] * c.get("depth", 1)
        dims = [c["in"], *hid, c["out"]]
        p = sum(a * b + b for a, b in zip(dims, dims[1:]))
        rows = c["batch"] * (c["steps"] if k == "mlp_fit" else c["rows"] // c["batch"])
        data = (c["batch"] if k == "mlp_fit" else c["rows"]) * (c["in"] + c["out"])
        return {"bytes": 24 * p + 4 * data, "flops": 6 * rows * p}
    if k == "f32_step":
        p = c["layers"] * (c["width"] ** 2 + c["width"])
        return {"bytes": 24 * p + 8 * c["rows"] * c["width"], "flops": (6 * c["layers"] - 2) * c["rows"] * c["width"] ** 2}
    if k == "cnn_fit":
        h1, p1, h2, p2 = _cnn_dims(c)
        kk = c["k"] ** 2
        conv = 2 * c["batch"] * (h1 * h1 * c["o1"] * c["c"] * kk + h2 * h2 * c["o2"] * c["o1"] * kk)
        flat = c["o2"] * p2 * p2
        fc = flat * c["hidden"] + c["hidden"] * 10 if c["hidden"] else flat * 10
        p = c["o1"] * c["c"] * kk + c["o2"] * c["o1"] * kk + fc
        return {"bytes": 24 * p + 4 * c["batch"] * (c["c"] * c["hw"] ** 2 + 10),
                "flops": 3 * c["steps"] * (conv + 2 * c["batch"] * fc)}
    if k == "conv_layer":
        q = _conv_out(c)
        x, y, w = c["batch"] * c["c"] * c["hw"] ** 2, c["batch"] * c["o"] * q * q, c["o"] * c["c"] * c["k"] ** 2
        # forward: x, w in, y and the pre-activation out; backward: g, x, w in, dx, dw out
        return {"bytes": 4 * (3 * x + 3 * w + 3 * y), "flops": 6 * c["batch"] * q * q * w}
    n = c["n"]
    return {"bytes": 2 * (4 * n + capi.load().vtlb_ckpt_text_len(n)), "flops": 0}


def tolerance(c):
    k = c["kind"]
    if k in ("int8_linear", "int8_mlp", "checkpoint"):
        return "exact"  # whole-number sums, and f32 operations that each round on their own
    if k == "conv_layer":
        return {"rel": 5e-6, "max": 5e-5}  # against the same sums in 64 bits: 1.2e-6 at most, 4e-6 in one value
    if k == "f32_step":
        # the products are off by 1e-5 of 64-bit ones; a pre-activation that is zero within that changes sides and
        # takes its row's part of the gradient with it (4e-4 over all gradients, 7e-2 in one)
        return {"rel": 2e-3, "max": 0.3}
    # two sum orders over a run of Adam steps: 1e-6 as a rule; where an activation or a gradient is zero within
    # rounding the runs part (4e-3 in the worst of 220, 6e-2 in one weight)
    return {"rel": 1e-2, "max": 0.25}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape, std=1.0):
    return torch.randn(*shape, generator=g, device="cuda").mul_(std)


def _one_hot(g, n, classes):
    t = torch.zeros(n, classes, device="cuda")
    t[torch.arange(n, device="cuda"), torch.randint(0, classes, (n,), generator=g, device="cuda")] = 1.0
    return t


def _buf(t):
    """A torch tensor's memory as the framework's device buffer."""
    return capi.DBuf(_dev(), t.data_ptr(), t.shape, np.float32)


class _Kept:
    """A model (or loader) that is closed when the program drops it."""

    def __init__(self, obj):
        self.obj = obj

    def __del__(self):
        self.obj.close()


def _quant_weight(g, n, k):
    """An [n, k] weight ~ N(0, 0.02), quantised per output channel: codes and scales."""
    dev = _dev()
    w = _normal(g, n, k, std=0.02)
    q = torch.zeros(n, dev.i8_ld(k), dtype=torch.int8, device="cuda")
    s = torch.empty(n, device="cuda")
    torch.cuda.synchronize()
    dev.quant_rows_i8(w.data_ptr(), n, k, q.data_ptr(), s.data_ptr())
    dev.sync()
    return q, s


def _set_params(model, seed, fans):
    """Kaiming-uniform weights; vectors (biases, BatchNorm) keep the values they start with."""
    rng = np.random.default_rng(int(seed))
    for i, fan in enumerate(fans):
        if fan:
            lim = (6.0 / fan) ** 0.5
            model.set_param(i, rng.uniform(-lim, lim, model.param_size(i)).astype(np.float32))


def prepare(case, seed):
    c = case
    dev = _dev()
    g = _gen(seed)
    st = {"case": c}
    k = c["kind"]
    if k == "int8_linear":
        m, n, kk = c["m"], c["n"], c["k"]
        st["w"], st["sw"] = _quant_weight(g, n, kk)
        st["bias"] = _normal(g, n, std=0.01)
        st["x"] = _normal(g, m, kk)
        st["q"] = torch.zeros(m, dev.i8_ld(kk), dtype=torch.int8, device="cuda")
        st["sa"] = torch.empty(m, device="cuda")
        st["y"] = torch.empty(m, n, device="cuda")
    elif k == "int8_mlp":
        dims = [c["d"], c["h"]] * (c["layers"] // 2) + [c["d"]]
        st["dims"], m = dims, c["m"]
        st["w"] = [_quant_weight(g, n, kk) + (_normal(g, n, std=0.01),) for kk, n in zip(dims, dims[1:])]
        st["x"] = _normal(g, m, dims[0])
        big = max(dims)
        st["q"] = [torch.zeros(m * dev.i8_ld(big), dtype=torch.int8, device="cuda") for _ in range(2)]
        st["sa"], st["amax"] = torch.empty(m, device="cuda"), torch.empty(m, device="cuda")
        st["hidden"], st["y"] = torch.empty(m * big, device="cuda"), torch.empty(m, dims[-1], device="cuda")
    elif k in ("mlp_fit", "mlp_epoch"):
        model = host.Model(_ses())
        model.input([c["in"]])
        fans, width = [], c["in"]
        for _ in range(c.get("depth", 1)):
            model.linear(c["hidden"])
            fans += [width, 0]
            model.relu()
            if k == "mlp_epoch":
                model.batchnorm1d(c["hidden"])
                fans += [0, 0]
            width = c["hidden"]
        model.linear(c["out"])
        fans += [width, 0]
        if k == "mlp_fit":
            model.mse_loss()
            model.adam(1e-4)
            st["x"] = torch.rand(c["batch"], c["in"], generator=g, device="cuda")
            st["t"] = _one_hot(g, c["batch"], c["out"])
        else:
            model.softmax_cross_entropy_loss()
            getattr(model, c["opt"])(1e-3 if c["opt"] == "sgd" else 1e-4)
            st["x"], st["t"] = _normal(g, c["rows"], c["in"]), _one_hot(g, c["rows"], c["out"])
            torch.cuda.synchronize()
            st["loader"] = _Kept(host.DataLoader(_ses(), _buf(st["x"]), _buf(st["t"]), c["batch"], True, True, int(seed) & 0xffff))
        _set_params(model, seed, fans)
        st["model"] = _Kept(model)
    elif k == "f32_step":
        L, n, rows = c["layers"], c["width"], c["rows"]
        pw, pb = -(-n * n // 64) * 64, -(-n // 64) * 64  # every tensor starts on a 256-byte boundary
        st["theta"], st["grad"], st["m"], st["v"] = (torch.zeros(L * (pw + pb), device="cuda") for _ in range(4))
        for i in range(L):
            st["theta"][i * pw:i * pw + n * n].uniform_(-1, 1, generator=g).mul_((6.0 / n) ** 0.5)
        views = lambda t: ([t[i * pw:] for i in range(L)], [t[L * pw + i * pb:] for i in range(L)])  # noqa: E731
        st["W"], st["b"] = views(st["theta"])
        st["dW"], st["db"] = views(st["grad"])
        ptr = [[t.data_ptr() for t in ts] for w in ("theta", "grad", "m", "v") for ts in views(st[w])]
        st["table"] = capi.Device.adam_table(
            [(ptr[2][i], ptr[0][i], ptr[4][i], ptr[6][i], n * n) for i in range(L)] +
            [(ptr[3][i], ptr[1][i], ptr[5][i], ptr[7][i], n) for i in range(L)])
        st["x"], st["t"] = _normal(g, rows, n), _normal(g, rows, n)
        st["pre"], st["act"] = ([torch.empty(rows, n, device="cuda") for _ in range(L)] for _ in range(2))
        st["g"] = [torch.empty(rows, n, device="cuda") for _ in range(2)]
        st["loss"] = torch.zeros(1, device="cuda")
        st["step"] = 0
    elif k == "cnn_fit":
        h1, p1, h2, p2 = _cnn_dims(c)
        kk, pad = (c["k"], c["k"]), (c["pad"], c["pad"])
        model = host.Model(_ses())
        model.input([c["c"], c["hw"], c["hw"]])
        model.conv2d(c["c"], c["o1"], kk, pad)
        model.relu()
        if c["pool1"]:
            model.maxpool2d((2, 2), (0, 0), (2, 2))
        model.conv2d(c["o1"], c["o2"], kk, pad)
        model.relu()
        model.maxpool2d((2, 2), (0, 0), (2, 2))
        model.flatten()
        flat = c["o2"] * p2 * p2
        fans = [c["c"] * c["k"] ** 2, 0, c["o1"] * c["k"] ** 2, 0, flat, 0]
        if c["hidden"]:
            model.linear(c["hidden"])
            model.relu()
            fans += [c["hidden"], 0]
        model.linear(10)
        model.softmax_cross_entropy_loss()
        model.adam(1e-4)
        _set_params(model, seed, fans)
        st["model"] = _Kept(model)
        st["x"] = _normal(g, c["batch"], c["c"], c["hw"], c["hw"])
        st["t"] = _one_hot(g, c["batch"], 10)
    elif k == "conv_layer":
        q = _conv_out(c)
        st["x"] = _normal(g, c["batch"], c["c"], c["hw"], c["hw"])
        st["w"] = _normal(g, c["o"], c["c"], c["k"], c["k"], std=(2.0 / (c["c"] * c["k"] ** 2)) ** 0.5)
        st["bias"] = _normal(g, c["o"], std=0.01)
        st["g"] = _normal(g, c["batch"], c["o"], q, q)
        for name, like in (("y", "g"), ("pre", "g"), ("dx", "x"), ("dw", "w"), ("db", "bias")):
            st[name] = torch.empty_like(st[like])
    else:
        n = c["n"]
        st["x"] = _normal(g, n, std=0.02)
        st["text"] = torch.zeros(dev.ckpt_text_len(n), dtype=torch.uint8, device="cuda")
        st["back"] = torch.empty(n, device="cuda")
    return st


# ---------------------------------------------------------------- one pass
def _run_int8_linear(st, c, dev):
    m, n, k = c["m"], c["n"], c["k"]
    dev.quant_rows_i8(st["x"].data_ptr(), m, k, st["q"].data_ptr(), st["sa"].data_ptr())
    dev.linear_i8_fwd(st["q"].data_ptr(), st["sa"].data_ptr(), st["w"].data_ptr(), st["sw"].data_ptr(),
                      st["bias"].data_ptr(), st["y"].data_ptr(), m, n, k, c["relu"])
    return st["y"], st["q"], st["sa"]


def _run_int8_mlp(st, c, dev):
    m, dims = c["m"], st["dims"]
    sa_t, amax_t = st["sa"], st["amax"]
    sa, amax, hid = sa_t.data_ptr(), amax_t.data_ptr(), st["hidden"].data_ptr()
    q = [t.data_ptr() for t in st["q"]]
    dev.quant_rows_i8(st["x"].data_ptr(), m, dims[0], q[0], sa)
    for i, (wq, sw, bias) in enumerate(st["w"]):
        k, n = dims[i], dims[i + 1]
        a = q[i & 1]
        if i + 1 == len(st["w"]):
            dev.linear_i8_fwd(a, sa, wq.data_ptr(), sw.data_ptr(), bias.data_ptr(), st["y"].data_ptr(), m, n, k, False)
        else:
            dev.linear_i8_fwd_amax(a, 1, sa, wq.data_ptr(), sw.data_ptr(), bias.data_ptr(), hid, m, n, k, True, amax)
            dev.quant_rows_i8(hid, m, n, q[1 - (i & 1)], sa, amax)
    return st["y"], st["hidden"], sa_t, amax_t


def _weights(model):
    return [model.get_param(i) for i in range(model.num_params())]


def _run_fit(st, c, dev):
    model, steps = st["model"].obj, c["steps"]
    x, t = st["x"].data_ptr(), st["t"].data_ptr()
    for i in range(steps):
        loss = model.train_step(x, st["x"].shape, t, st["t"].shape, want_loss=i + 1 == steps)
    return [loss] + _weights(model)


def _run_mlp_epoch(st, c, dev):
    model, loader = st["model"].obj, st["loader"].obj
    loader.reset()
    for i in range(len(loader)):
        feat, lab = loader.batch_with_labels(i)
        loss = model.train_step(feat, feat.shape, lab, lab.shape, want_loss=i + 1 == len(loader))
        feat.free()
        lab.free()
    stats = [model.running_stat(0, c["hidden"], v) for v in (False, True)]
    return [loss] + _weights(model) + stats


def _run_f32_step(st, c, dev):
    L, n, rows = c["layers"], c["width"], c["rows"]
    W, b, dW, db = ([t.data_ptr() for t in st[k]] for k in ("W", "b", "dW", "db"))
    pre, act, g = ([t.data_ptr() for t in st[k]] for k in ("pre", "act", "g"))
    ins = [st["x"].data_ptr()] + act[:-1]
    for i in range(L):
        last = i + 1 == L
        dev.linear_fwd_f32(ins[i], W[i], b[i], act[i], rows, n, n, relu=not last, pre=None if last else pre[i])
    dev.mse_fwd_bwd_f32(act[-1], st["t"].data_ptr(), rows * n, rows * n, st["loss"].data_ptr(), g[0])
    for i in reversed(range(L)):
        # the gradient of the layer below comes out masked by that layer's ReLU
        dev.linear_bwd_f32_planes(g[0], ins[i], W[i], g[1] if i else None, dW[i], db[i], rows, n, n,
                                  relu_mask_src=pre[i - 1] if i else None)
        g.reverse()
    st["step"] += 1
    t = st["step"]
    lr_t = 1e-4 * (1.0 - 0.999 ** t) ** 0.5 / (1.0 - 0.9 ** t)
    dev.adamw_step_f32(st["table"], 0.9, 0.999, lr_t, 1e-8, 0.01, zero_grad=False)
    return st["loss"], st["theta"], st["m"], st["v"]


def _run_conv_layer(st, c, dev):
    dims = (c["batch"], c["c"], c["hw"], c["hw"], c["o"], c["k"], c["k"], c["pad"], c["pad"], c["stride"], c["stride"])
    p = {k: v.data_ptr() for k, v in st.items() if k != "case"}
    dev.conv2d_fwd_f32(p["x"], p["w"], p["bias"], p["y"], *dims, relu=True, pre=p["pre"])
    dev.conv2d_bwd_f32(p["g"], p["x"], p["w"], p["dx"], p["dw"], p["db"], *dims)
    return st["y"], st["pre"], st["dx"], st["dw"], st["db"]


def _run_checkpoint(st, c, dev):
    n = c["n"]
    dev.ckpt_encode_f32(st["x"].data_ptr(), n, st["text"].data_ptr())
    dev.ckpt_decode_f32(st["text"].data_ptr(), st["text"].numel(), st["back"].data_ptr(), n)
    return st["text"], st["back"]


_RUN = {"int8_linear": _run_int8_linear, "int8_mlp": _run_int8_mlp, "mlp_fit": _run_fit, "mlp_epoch": _run_mlp_epoch,
        "f32_step": _run_f32_step, "cnn_fit": _run_fit, "conv_layer": _run_conv_layer, "checkpoint": _run_checkpoint}


def run(state):
    return _RUN[state["case"]["kind"]](state, state["case"], _dev())
