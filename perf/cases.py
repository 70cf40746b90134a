"""The work that programs have this framework do, as cases that can be timed.

Every case is a pass through the public entry points on device arrays: the
ndarray functions of ``owl_gb300.dense.NN`` (convolutions and poolings, all
directions), the layers of ``owl_gb300.layers`` and the Algodiff training step.
Inputs are drawn from a seed: activations uniform in [-1, 1] (pixels in [0, 1]),
kernels N(0, 2 / fan_in), output gradients N(0, 1).
"""

from __future__ import annotations

import math

import torch

from owl_gb300 import _lib
from owl_gb300 import algodiff as A
from owl_gb300.dense import NN, SAME, GpuBackend
from owl_gb300.layers import ACT_NONE, ACT_RELU, Layers

# The most multiply-add work (FLOPs) that a drawn case may have, by how its
# convolutions are computed: no drawn case costs more than the largest listed.
DRAW_FLOPS = {"fp32": 2.0e10, "tf32": 6e10, "bf16": 1.6e11, "bf16x3": 1.0e11, "f64": 1.2e9}


def listed():
    return [
        # a single small call in the default precision, as a user's first program makes it:
        # latency and launches (conv2d, then max_pool2d with argmax on its output)
        {"name": "small_conv_pool_fp32", "kind": "conv_pool", "prec": "fp32", "b": 8, "side": 32,
         "ci": 16, "co": 32, "k": 3},
        # training a wide layer of a vision network in BF16: forward and both gradients
        {"name": "conv2d_bf16", "kind": "conv", "prec": "bf16", "b": 64, "dims": "56x56",
         "ci": 128, "co": 128, "k": 3, "s": 1, "rate": 1, "padding": "SAME"},
        # a downsampling layer: stride 2, VALID, twice the channels
        {"name": "conv2d_strided_bf16", "kind": "conv", "prec": "bf16", "b": 64, "dims": "28x28",
         "ci": 256, "co": 256, "k": 3, "s": 2, "rate": 1, "padding": "VALID"},
        # a dilated layer at float32 accuracy (split BF16)
        {"name": "dilated_conv2d_split", "kind": "conv", "prec": "bf16x3", "b": 64,
         "dims": "56x56", "ci": 128, "co": 128, "k": 3, "s": 1, "rate": 2, "padding": "SAME"},
        # the default precision, plain float32, on odd sizes
        {"name": "conv2d_fp32_ragged", "kind": "conv", "prec": "fp32", "b": 16, "dims": "57x43",
         "ci": 96, "co": 160, "k": 3, "s": 1, "rate": 1, "padding": "SAME"},
        # Owl's D module: a gradient check's convolution in float64
        {"name": "conv2d_f64", "kind": "conv", "prec": "f64", "b": 8, "dims": "28x28", "ci": 32,
         "co": 64, "k": 5, "s": 1, "rate": 1, "padding": "SAME"},
        # a volumetric encoder stage (conv3d) and decoder stage (transpose_conv3d), trained in BF16
        {"name": "conv3d_pair_bf16", "kind": "conv3d_pair", "prec": "bf16", "b": 4, "side": 32,
         "ci": 32, "co": 64},
        # volumetric pooling, max and average, forward and backward
        {"name": "pool3d", "kind": "pool", "b": 4, "dims": "32x32x32", "ch": 64, "k": 2, "s": 2},
        # overlapping windows, as after the stem of a residual network
        {"name": "pool2d_overlap", "kind": "pool", "b": 16, "dims": "112x112", "ch": 64, "k": 3,
         "s": 2},
        # a whole training step's gradients (two convolutions, two pools, two dense layers) in
        # the default precision
        {"name": "cnn_step_fp32", "kind": "cnn", "prec": "fp32", "b": 256},
        # the layers of that network trained in BF16: convolution with bias and ReLU, dense
        # layers, and their backward passes
        {"name": "train_layers_bf16", "kind": "layers", "prec": "bf16", "b": 256, "side": 14,
         "ci": 32, "co": 64, "units": 1024, "k": 5},
        # a downsampling block of the serving stack, its kernels declared constant
        {"name": "serve_block_bf16", "kind": "block", "prec": "bf16", "b": 16, "side": 28,
         "ci": 128, "co": 256},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_conv(rng):
    prec = rng.choice(("fp32", "bf16", "bf16", "bf16", "bf16x3", "tf32", "f64"))
    nd = 3 if rng.random() < 0.2 else 2
    while True:
        c = {"kind": "conv", "prec": prec, "b": _log(rng, 1, 64),
             "dims": "x".join(str(_log(rng, 5, 112 if nd == 2 else 32)) for _ in range(nd)),
             "ci": _log(rng, 3, 512), "co": _log(rng, 8, 512), "k": rng.choice((1, 3, 3, 3, 5)),
             "s": rng.choice((1, 1, 1, 2)), "rate": 1, "padding": rng.choice(("SAME", "VALID"))}
        if rng.random() < 0.75:  # most layers have round channel counts
            c["ci"], c["co"] = ((v + 15) // 16 * 16 for v in (c["ci"], c["co"]))
        if c["s"] == 1 and nd == 2 and c["k"] == 3 and rng.random() < 0.25:
            c["rate"] = 2
        x, y, _ = _conv_shapes(c)
        ok = min(y[1:-1]) >= 1 and max(math.prod(x), math.prod(y)) <= 64 * 56 * 56 * 128
        if ok and 0.002 * DRAW_FLOPS[prec] <= work(c)["flops"] <= DRAW_FLOPS[prec]:
            return c


def draw(rng):
    kind = rng.choice(("conv", "conv", "conv", "conv_pool", "conv3d_pair", "pool", "pool",
                       "cnn", "layers", "block"))
    if kind == "conv":
        return _draw_conv(rng)
    if kind == "conv_pool":
        return {"kind": kind, "prec": "fp32", "b": _log(rng, 1, 16), "side": _log(rng, 8, 48),
                "ci": rng.choice((1, 3, 8, 16, 20, 32)), "co": rng.choice((8, 16, 24, 32, 64)),
                "k": rng.choice((1, 3, 5))}
    if kind == "conv3d_pair":
        return {"kind": kind, "prec": rng.choice(("bf16", "bf16", "fp32", "bf16x3")),
                "b": _log(rng, 1, 4), "side": 2 * _log(rng, 4, 16),
                "ci": rng.choice((8, 16, 24, 32)), "co": rng.choice((16, 32, 48, 64))}
    if kind == "pool":
        if rng.random() < 0.4:
            dims = "x".join(str(_log(rng, 6, 40)) for _ in range(3))
            k, s = rng.choice(((2, 2), (2, 2), (3, 2), (3, 3)))
        else:
            dims = "x".join(str(_log(rng, 7, 112)) for _ in range(2))
            k, s = rng.choice(((2, 2), (3, 2), (3, 2), (3, 1), (3, 3)))
        n = math.prod(int(d) for d in dims.split("x"))
        ch = rng.choice((3, 16, 32, 64, 96, 128, 256))
        return {"kind": kind, "b": max(1, min(_log(rng, 1, 64), 16 * 112 * 112 * 64 // (n * ch))),
                "dims": dims, "ch": ch, "k": k, "s": s}
    if kind == "cnn":
        return {"kind": kind, "prec": "fp32", "b": _log(rng, 16, 256)}
    if kind == "layers":
        return {"kind": kind, "prec": rng.choice(("bf16", "bf16", "bf16x3", "fp32")),
                "b": _log(rng, 16, 256), "side": rng.choice((7, 10, 14, 15)),
                "ci": rng.choice((16, 32)), "co": rng.choice((32, 48, 64)),
                "units": rng.choice((104, 256, 512, 1000, 1024)), "k": rng.choice((3, 5))}
    side, ci = rng.choice(((56, 64), (28, 128), (28, 128), (14, 256), (7, 256)))
    return {"kind": "block", "prec": "bf16", "b": _log(rng, 1, 64 if side < 56 else 32),
            "side": side, "ci": ci, "co": 2 * ci}


# ---- shapes --------------------------------------------------------------------


def _out(n, k, s, padding):
    return -(-n // s) if padding == "SAME" else -(-(n - k + 1) // s)


def _conv_shapes(c):
    dims = [int(d) for d in c["dims"].split("x")]
    ext = (c["k"] - 1) * c["rate"] + 1
    od = [_out(n, ext, c["s"], c["padding"]) for n in dims]
    return ((c["b"], *dims, c["ci"]), (c["b"], *od, c["co"]),
            (*[c["k"]] * len(dims), c["ci"], c["co"]))


def _conv_flops(out_shape, w_shape):
    return 2.0 * math.prod(out_shape[:-1]) * math.prod(w_shape)


def _pool_out(c):
    return (c["b"], *[_out(int(d), c["k"], c["s"], "SAME") for d in c["dims"].split("x")], c["ch"])


# ---- inputs --------------------------------------------------------------------


class _Gen:
    """Seeded device arrays."""

    def __init__(self, seed, prec="fp32"):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype = torch.float64 if prec == "f64" else torch.float32

    def uniform(self, shape, lo=-1.0, hi=1.0):
        return torch.empty(shape, dtype=self.dtype, device="cuda").uniform_(lo, hi,
                                                                           generator=self.g)

    def normal(self, shape, std=1.0):
        return torch.empty(shape, dtype=self.dtype, device="cuda").normal_(0.0, std,
                                                                          generator=self.g)

    def kernel(self, shape):
        return self.normal(shape, math.sqrt(2.0 / math.prod(shape[:-1])))


class _Declared:
    """Kernel tensors declared constant to the library, as a serving stack
    holds them: forgotten before they are freed."""

    def __init__(self, tensors):
        self.tensors = tensors
        for t in tensors:
            _lib.call("owlgpu_weights_declare", t.data_ptr(), 0)

    def __del__(self):
        for t in self.tensors:
            _lib.call("owlgpu_weights_forget", t.data_ptr())


def _nn(prec):
    return NN(GpuBackend("fp32" if prec == "f64" else prec))


def _inputs(c, seed):
    g = _Gen(seed, c.get("prec", "fp32"))
    k = c["kind"]
    if k == "conv":
        x, y, w = _conv_shapes(c)
        return {"x": g.uniform(x), "w": g.kernel(w), "dy": g.normal(y)}
    if k == "conv_pool":
        return {"x": g.uniform((c["b"], c["side"], c["side"], c["ci"])),
                "w": g.uniform((c["k"], c["k"], c["ci"], c["co"]))}
    if k == "conv3d_pair":
        b, n, h, ci, co = c["b"], c["side"], c["side"] // 2, c["ci"], c["co"]
        return {"x": g.uniform((b, n, n, n, ci)), "w": g.kernel((3, 3, 3, ci, co)),
                "dy": g.normal((b, n, n, n, co)), "tx": g.uniform((b, h, h, h, co)),
                "tw": g.kernel((2, 2, 2, co, ci)), "tdy": g.normal((b, n, n, n, ci))}
    if k == "pool":
        dims = [int(d) for d in c["dims"].split("x")]
        return {"x": g.uniform((c["b"], *dims, c["ch"])), "dy": g.normal(_pool_out(c))}
    if k == "cnn":
        p = {n: g.kernel(s) if n.startswith("w") else g.uniform(s, -0.05, 0.05)
             for n, s in A.MNIST_CNN}
        labels = torch.randint(0, 10, (c["b"],), generator=g.g, device="cuda")
        return {"x": g.uniform((c["b"], 28, 28, 1), 0.0, 1.0), "params": p,
                "onehot": torch.nn.functional.one_hot(labels, 10).to(g.dtype)}
    if k == "layers":
        b, n, ci, co, u = c["b"], c["side"], c["ci"], c["co"], c["units"]
        f = (n // 2) * (n // 2) * co
        return {"x": g.uniform((b, n, n, ci), 0.0, 1.0), "w": g.kernel((c["k"], c["k"], ci, co)),
                "b": g.uniform((co,), -0.05, 0.05), "dy": g.normal((b, n, n, co)),
                "yact": torch.relu(g.normal((b, n, n, co))), "a": torch.relu(g.normal((b, f))),
                "wd": g.kernel((f, u)), "bd": g.uniform((u,), -0.05, 0.05),
                "dz": g.normal((b, u)), "w2": g.kernel((u, 10)), "b2": g.uniform((10,))}
    b, n, ci, co = c["b"], c["side"], c["ci"], c["co"]
    m = -(-n // 2)
    return {"x": torch.relu(g.normal((b, n, n, ci))), "h": torch.relu(g.normal((b, m, m, co))),
            "w1": g.kernel((3, 3, ci, co)), "w2": g.kernel((3, 3, co, co)),
            "wp": g.kernel((1, 1, ci, co))}


def prepare(case, seed):
    st = {"case": case, "nn": _nn(case.get("prec", "fp32")), **_inputs(case, seed)}
    k = case["kind"]
    if k == "cnn":
        st["ad"] = A.Algodiff(st["nn"])
    elif k in ("layers", "block"):
        st["layers"] = Layers(st["nn"])
    if k == "block":
        st["declared"] = _Declared([st["w1"], st["w2"], st["wp"]])
    return st


# ---- one pass ------------------------------------------------------------------


def run(st):
    c, nn = st["case"], st["nn"]
    k = c["kind"]
    if k == "conv":
        x, w, dy, p = st["x"], st["w"], st["dy"], c["padding"]
        s = [c["s"]] * (x.dim() - 2)
        if c["rate"] > 1:
            r = [c["rate"]] * len(s)
            return (nn.dilated_conv2d(x, w, s, r, p),
                    nn.dilated_conv2d_backward_input(x, w, s, r, dy),
                    nn.dilated_conv2d_backward_kernel(x, w, s, r, dy))
        if x.dim() == 5:
            return (nn.conv3d(x, w, s, p), nn.conv3d_backward_input(x, w, s, dy),
                    nn.conv3d_backward_kernel(x, w, s, dy))
        return (nn.conv2d(x, w, s, p), nn.conv2d_backward_input(x, w, s, dy),
                nn.conv2d_backward_kernel(x, w, s, dy))
    if k == "conv_pool":
        y = nn.conv2d(st["x"], st["w"], [1, 1], SAME)
        return (y, *nn.max_pool2d_argmax(y, [2, 2], [2, 2], SAME))
    if k == "conv3d_pair":
        x, w, dy, one, two = st["x"], st["w"], st["dy"], [1, 1, 1], [2, 2, 2]
        tx, tw, tdy = st["tx"], st["tw"], st["tdy"]
        return (nn.conv3d(x, w, one, SAME), nn.conv3d_backward_input(x, w, one, dy),
                nn.conv3d_backward_kernel(x, w, one, dy), nn.transpose_conv3d(tx, tw, two, SAME),
                nn.transpose_conv3d_backward_input(tx, tw, two, tdy),
                nn.transpose_conv3d_backward_kernel(tx, tw, two, tdy))
    if k == "pool":
        x, dy, nd = st["x"], st["dy"], st["x"].dim() - 2
        ks, ss = [c["k"]] * nd, [c["s"]] * nd
        if nd == 3:
            return (nn.max_pool3d(x, ks, ss), nn.max_pool3d_backward(SAME, x, ks, ss, dy),
                    nn.avg_pool3d(x, ks, ss), nn.avg_pool3d_backward(SAME, x, ks, ss, dy))
        return (nn.max_pool2d(x, ks, ss), nn.max_pool2d_backward(SAME, x, ks, ss, dy),
                nn.avg_pool2d(x, ks, ss), nn.avg_pool2d_backward(SAME, x, ks, ss, dy))
    if k == "cnn":
        loss, grads = A.loss_and_grads(st["ad"], st["params"], st["x"], st["onehot"])
        return loss, grads
    L = st["layers"]
    if k == "layers":
        y = L.conv2d_bias_act(st["x"], st["w"], st["b"], [1, 1], SAME, ACT_RELU)
        dz, db = L.bias_act_backward(st["yact"], st["dy"], ACT_RELU)
        h = L.dot(st["a"], st["wd"], bias=st["bd"], act=ACT_RELU)
        da = L.dot(st["dz"], st["wd"], trans_b=True)
        dw = L.dot(st["a"], st["dz"], trans_a=True)
        z = L.dot(st["dz"], st["w2"], bias=st["b2"], act=ACT_NONE)
        return y, dz, db, h, da, dw, z
    return (L.conv2d_bias_act(st["x"], st["w1"], None, [2, 2], SAME, ACT_RELU),
            nn.conv2d(st["h"], st["w2"], [1, 1], SAME),
            nn.conv2d(st["x"], st["wp"], [2, 2], SAME))


# ---- what a pass cannot do without ---------------------------------------------


def work(c):
    k = c["kind"]
    if k == "conv":
        x, y, w = _conv_shapes(c)
        n = [math.prod(v) for v in (x, y, w)]  # three passes, each two operands in, one out
        return {"bytes": (8 if c["prec"] == "f64" else 4) * 3 * sum(n),
                "flops": 3 * _conv_flops(y, w)}
    if k == "conv_pool":
        y = (c["b"], c["side"], c["side"], c["co"])
        w = (c["k"], c["k"], c["ci"], c["co"])
        po = c["b"] * (-(-c["side"] // 2)) ** 2 * c["co"]
        return {"bytes": 4 * (c["b"] * c["side"] ** 2 * c["ci"] + math.prod(w) +
                              2 * math.prod(y)) + 12 * po, "flops": _conv_flops(y, w)}
    if k == "conv3d_pair":
        b, n, ci, co = c["b"], c["side"], c["ci"], c["co"]
        px, ph = b * n ** 3, b * (n // 2) ** 3
        return {"bytes": 4 * 3 * (px * (ci + co) + 27 * ci * co + ph * co + px * ci + 8 * ci * co),
                "flops": 3 * (2.0 * px * 27 * ci * co + 2.0 * ph * 8 * ci * co)}
    if k == "pool":
        nx = c["b"] * math.prod(int(d) for d in c["dims"].split("x")) * c["ch"]
        ny = math.prod(_pool_out(c))
        # max: x -> y, (x, dy) -> dx; average: x -> y, dy -> dx
        return {"bytes": 4 * (5 * nx + 4 * ny), "flops": 0}
    if k == "cnn":
        b, p = c["b"], sum(math.prod(s) for _, s in A.MNIST_CNN)
        conv = 2.0 * b * (784 * 800 + 196 * 51200)
        dense = 2.0 * b * (3136 * 1024 + 10240)
        acts = b * (784 + 2 * 784 * 32 + 2 * 196 * 64)  # pixels and the two layers' outputs
        return {"bytes": 4 * (3 * p + 2 * acts), "flops": 3 * (conv + dense) - 2.0 * b * 784 * 800}
    if k == "layers":
        b, n, ci, co, u = c["b"], c["side"], c["ci"], c["co"], c["units"]
        f, w = (n // 2) * (n // 2) * co, c["k"] ** 2 * ci * co
        px = b * n * n
        return {"bytes": 4 * (px * (ci + 4 * co) + w + 3 * (b * f + f * u + b * u) + b * u),
                "flops": 2.0 * px * w + 6.0 * b * f * u + 2.0 * b * u * 10}
    b, n, ci, co = c["b"], c["side"], c["ci"], c["co"]
    m = -(-n // 2)
    wn = 9 * ci * co + 9 * co * co + ci * co
    return {"bytes": 4 * (b * n * n * ci * 5 // 4 + 4 * b * m * m * co + wn),
            "flops": 2.0 * b * m * m * wn}


# ---- the same in 64 bits -------------------------------------------------------


def _same_pad(n, o, ext, s):
    p = max((o - 1) * s + ext - n, 0)
    return p // 2, p - p // 2


class _Conv64:
    """A convolution and its gradients tap by tap in float64."""

    def __init__(self, in_shape, out_shape, k, s, rate):
        self.k, self.s, self.rate, self.nd = k, s, rate, len(in_shape) - 2
        ext = (k - 1) * rate + 1
        self.n, self.o = in_shape[1:-1], out_shape[1:-1]
        self.pads = [_same_pad(n, o, ext, s) for n, o in zip(self.n, self.o)]

    def _padded(self, a):
        flat = [0, 0]
        for lo, hi in reversed(self.pads):
            flat += [lo, hi]
        return torch.nn.functional.pad(a, flat)

    def _taps(self):
        for t in range(self.k ** self.nd):
            at = []
            for _ in range(self.nd):
                at.insert(0, t % self.k)
                t //= self.k
            win = tuple(slice(i * self.rate, i * self.rate + (o - 1) * self.s + 1, self.s)
                        for i, o in zip(at, self.o))
            yield tuple(at), (slice(None), *win)

    def forward(self, x, w):
        xp, y = self._padded(x), 0.0
        for at, win in self._taps():
            y = y + xp[win] @ w[at]
        return y

    def backward_input(self, w, dy):
        shape = (dy.shape[0], *[n + lo + hi for n, (lo, hi) in zip(self.n, self.pads)],
                 w.shape[-2])
        dx = torch.zeros(shape, dtype=dy.dtype, device=dy.device)
        for at, win in self._taps():
            dx[win] += dy @ w[at].T
        return dx[(slice(None), *[slice(lo, lo + n) for n, (lo, _) in zip(self.n, self.pads)])]

    def backward_kernel(self, x, dy):
        xp, dw = self._padded(x), {}
        d = dy.reshape(-1, dy.shape[-1])
        for at, win in self._taps():
            dw[at] = xp[win].reshape(-1, x.shape[-1]).T @ d
        return torch.stack(list(dw.values())).reshape(*[self.k] * self.nd, x.shape[-1], -1)


def _pool64(x, c, mode):
    nd, k, s = x.dim() - 2, c["k"], c["s"]
    o = _pool_out(c)[1:-1]
    pads = [_same_pad(n, m, k, s) for n, m in zip(x.shape[1:-1], o)]
    flat = [0, 0]
    for lo, hi in reversed(pads):
        flat += [lo, hi]
    inside = torch.nn.functional.pad(torch.ones_like(x[:1, ..., :1]), flat)
    xp = torch.nn.functional.pad(x, flat, value=-math.inf if mode == "max" else 0.0)
    parts, cnt = [], 0
    for t in range(k ** nd):
        at = []
        for _ in range(nd):
            at.insert(0, t % k)
            t //= k
        win = (slice(None), *[slice(i, i + (m - 1) * s + 1, s) for i, m in zip(at, o)])
        parts.append(xp[win])
        cnt = cnt + inside[win]
    if mode == "avg":
        return sum(parts) / cnt
    best = parts[0]
    for p in parts[1:]:  # the first of equal values wins, as in the reference's scan
        best = torch.where(p > best, p, best)
    return best


def _grad(f, x, dy):
    x = x.detach().requires_grad_(True)
    y = f(x)
    return y.detach(), torch.autograd.grad(y, x, dy)[0]


def exact(c, seed):
    st = _inputs(c, seed)
    d = {n: (v.double() if torch.is_tensor(v) else {m: t.double() for m, t in v.items()})
         for n, v in st.items()}
    k = c["kind"]
    if k == "conv":
        cv = _Conv64(d["x"].shape, d["dy"].shape, c["k"], c["s"], c["rate"])
        return (cv.forward(d["x"], d["w"]), cv.backward_input(d["w"], d["dy"]),
                cv.backward_kernel(d["x"], d["dy"]))
    if k == "conv_pool":
        y = _Conv64(d["x"].shape, d["x"].shape, c["k"], 1, 1).forward(d["x"], d["w"])
        p = {"b": c["b"], "dims": f"{c['side']}x{c['side']}", "ch": c["co"], "k": 2, "s": 2}
        return y, _pool64(y, p, "max"), None
    if k == "conv3d_pair":
        cv = _Conv64(d["x"].shape, d["dy"].shape, 3, 1, 1)
        # the transpose is the backward pass of a stride-2 convolution whose
        # kernel is the same buffer read with its channel axes named the other way
        tv = _Conv64(d["tdy"].shape, d["tx"].shape, 2, 2, 1)
        tw = d["tw"].reshape(2, 2, 2, c["ci"], c["co"])
        return (cv.forward(d["x"], d["w"]), cv.backward_input(d["w"], d["dy"]),
                cv.backward_kernel(d["x"], d["dy"]), tv.backward_input(tw, d["tx"]),
                tv.forward(d["tdy"], tw),
                tv.backward_kernel(d["tdy"], d["tx"]).reshape(d["tw"].shape))
    if k == "pool":
        mx = _grad(lambda x: _pool64(x, c, "max"), d["x"], d["dy"])
        av = _grad(lambda x: _pool64(x, c, "avg"), d["x"], d["dy"])
        return (*mx, *av)
    if k == "cnn":
        return _cnn64(d)
    F = torch.nn.functional
    if k == "layers":
        cv = _Conv64(d["x"].shape, d["dy"].shape, c["k"], 1, 1)
        dz = d["dy"] * (d["yact"] > 0)
        return (F.relu(cv.forward(d["x"], d["w"]) + d["b"]), dz,
                dz.reshape(-1, c["co"]).sum(0), F.relu(d["a"] @ d["wd"] + d["bd"]),
                d["dz"] @ d["wd"].T, d["a"].T @ d["dz"], d["dz"] @ d["w2"] + d["b2"])
    down = _Conv64(d["x"].shape, d["h"].shape, 3, 2, 1)
    return (F.relu(down.forward(d["x"], d["w1"])),
            _Conv64(d["h"].shape, d["h"].shape, 3, 1, 1).forward(d["h"], d["w2"]),
            _Conv64(d["x"].shape, d["h"].shape, 1, 2, 1).forward(d["x"], d["wp"]))


def _cnn64(d):
    p = {n: t.requires_grad_(True) for n, t in d["params"].items()}
    F = torch.nn.functional
    h = d["x"]
    for w, b, ch in (("w1", "b1", 32), ("w2", "b2", 64)):
        cv = _Conv64(h.shape, (*h.shape[:3], ch), 5, 1, 1)
        h = F.relu(cv.forward(h, p[w]) + p[b])
        pool = {"b": h.shape[0], "dims": f"{h.shape[1]}x{h.shape[2]}", "ch": ch, "k": 2, "s": 2}
        h = _pool64(h, pool, "max")
    h = F.relu(h.reshape(h.shape[0], -1) @ p["w3"] + p["b3"])
    z = h @ p["w4"] + p["b4"]
    loss = -(d["onehot"] * F.log_softmax(z, dim=1)).sum() / z.shape[0]
    loss.backward()
    return loss.detach(), {n: t.grad for n, t in p.items()}
