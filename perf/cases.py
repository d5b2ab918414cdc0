"""The calls this library's speed is judged by: what a user of it runs, at the sizes they run it.

A case is a plain dict; ``kind`` says which public entry point it goes through:

* ``gemm``    - ``tensor.gemm`` (Y = alpha op(A) op(B) + beta C) or, with alpha = 1 and beta = 0,
  ``tensor.matmul`` on (transposed views of) row-major matrices;
* ``batched`` - ``tensor.matmul`` of two stacks of matrices;
* ``conv``    - ``gdnn.conv2d_filter``, NCHW, with the bias and optionally the residual and ReLU that
  a graph runtime fuses into it;
* ``forward`` - ``predict.Predictor``: set the images, run the operator list, take the logits;
* ``level3``  - ``tensor.trsm`` / ``trmm`` / ``symm`` and ``gblas.syrk``.
"""
import math

import numpy as np
import torch

from dlf_b200 import gblas, gdnn, predict, tensor
from dlf_b200.gblas import Diagonal, Layout, Side, Transpose, Triangle

_TYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
_BYTES = {"f16": 2, "bf16": 2, "f32": 4}


def listed():
    return [
        # one small fp32 product, sizes of nothing in particular: what a call costs
        {"name": "matmul_f32_small", "kind": "gemm", "dtype": "f32", "m": 60, "n": 72, "k": 50,
         "ta": False, "tb": False, "alpha": 1.0, "beta": 0.0},
        # the ordinary fp32 product (an sgemm of 1024^3)
        {"name": "sgemm_1024", "kind": "gemm", "dtype": "f32", "m": 1024, "n": 1024, "k": 1024,
         "ta": False, "tb": False, "alpha": 1.0, "beta": 0.0},
        # odd sizes, rows that start on odd addresses, a transposed weight matrix
        {"name": "gemm_bf16_ragged", "kind": "gemm", "dtype": "bf16", "m": 1111, "n": 1537, "k": 777,
         "ta": False, "tb": True, "alpha": 1.0, "beta": 0.0},
        # the 16-bit product the tensor cores are made for
        {"name": "gemm_f16_4096", "kind": "gemm", "dtype": "f16", "m": 4096, "n": 4096, "k": 4096,
         "ta": False, "tb": False, "alpha": 1.0, "beta": 0.0},
        # the largest: A stored K x M and passed transposed, scaled and added to half of C
        {"name": "sgemm_16384_tn", "kind": "gemm", "dtype": "f32", "m": 16384, "n": 16384, "k": 16384,
         "ta": True, "tb": False, "alpha": 0.5, "beta": 0.5},
        # many small products at once (1024 of 512 x 512 x 64, an attention's scores)
        {"name": "bmm_f16_1024", "kind": "batched", "dtype": "f16", "batch": 1024, "m": 512, "n": 512, "k": 64,
         "tb": False},
        # the fp32 convolution of a network's early layers
        {"name": "conv_f32_64x56", "kind": "conv", "dtype": "f32", "batch": 64, "cin": 64, "h": 56, "w": 56, "cout": 64,
         "kh": 3, "kw": 3, "stride": 1, "pad": 1, "dilation": 1, "group": 1, "residual": False, "relu": False},
        # the commonest 3 x 3 layer of a large-batch network through the NCHW entry, with its fused tail
        {"name": "conv_f16_256x14", "kind": "conv", "dtype": "f16", "batch": 256, "cin": 256, "h": 14, "w": 14, "cout": 256,
         "kh": 3, "kw": 3, "stride": 1, "pad": 1, "dilation": 1, "group": 1, "residual": True, "relu": True},
        # whole ResNet-50 v1 forwards: throughput in fp16, a small fp32 batch, one image at a time
        {"name": "resnet50_f16_b256", "kind": "forward", "dtype": "f16", "batch": 256, "size": 224},
        {"name": "resnet50_f32_b8", "kind": "forward", "dtype": "f32", "batch": 8, "size": 224},
        {"name": "resnet50_f16_b1", "kind": "forward", "dtype": "f16", "batch": 1, "size": 224},
        # a triangular system with many right-hand sides
        {"name": "trsm_f32_1024x512", "kind": "level3", "dtype": "f32", "routine": "trsm", "m": 1024, "n": 512,
         "left": True, "upper": False, "trans": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Log-uniform; half of them a multiple of 8, the rest whatever comes, odd ones among them."""
    v = _log(rng, lo, hi)
    return max(8, v // 8 * 8) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(("gemm", "gemm", "batched", "conv", "conv", "forward", "level3"))
    dtype = rng.choice(("f16", "bf16", "f32"))
    if kind == "gemm":
        most = 2e12 if dtype != "f32" else 1e12
        while True:
            m, n, k = (_size(rng, 24, 12000) for _ in range(3))
            if 2.0 * m * n * k <= most:
                break
        scaled = rng.random() < 0.3
        return {"kind": "gemm", "dtype": dtype, "m": m, "n": n, "k": k, "ta": rng.random() < 0.4,
                "tb": rng.random() < 0.4, "alpha": 0.5 if scaled else 1.0, "beta": 0.5 if scaled else 0.0}
    if kind == "batched":
        while True:
            b, m, n, k = _log(rng, 4, 1024), _size(rng, 16, 1024), _size(rng, 16, 1024), _size(rng, 16, 1024)
            if 2.0 * b * m * n * k <= 2e11 and b * (m * k + k * n + m * n) <= 6e8:
                break
        return {"kind": "batched", "dtype": dtype, "batch": b, "m": m, "n": n, "k": k, "tb": rng.random() < 0.4}
    if kind == "conv":
        most = 2.5e11 if dtype != "f32" else 1e11
        while True:
            group = rng.choice((1, 1, 1, 1, 1, 2, 4))
            f = rng.choice((1, 3, 3, 5, 7))
            c = {"kind": "conv", "dtype": dtype, "batch": _log(rng, 1, 256), "cin": group * _size(rng, 3, 512 // group),
                 "h": _log(rng, 7, 224), "w": _log(rng, 7, 224), "cout": group * _size(rng, 8, 512 // group), "kh": f,
                 "kw": f, "stride": rng.choice((1, 1, 2)), "pad": f // 2,
                 "dilation": 2 if f == 3 and rng.random() < 0.1 else 1, "group": group,
                 "residual": rng.random() < 0.3, "relu": rng.random() < 0.5}
            if (_filter(c).output_h > 1 and _filter(c).output_w > 1 and work(c)["flops"] <= most and
                    work(c)["bytes"] <= 8e8):
                return c
    if kind == "forward":
        batch = _log(rng, 1, 128 if dtype != "f32" else 24)
        return {"kind": "forward", "dtype": dtype, "batch": batch, "size": rng.choice((96, 160, 192, 224))}
    return {"kind": "level3", "dtype": "f32", "routine": rng.choice(("trsm", "trsm", "trmm", "symm", "syrk")),
            "m": _size(rng, 48, 2500), "n": _size(rng, 48, 2500), "left": rng.random() < 0.7,
            "upper": rng.random() < 0.5, "trans": rng.random() < 0.4}


# ------------------------------------------------------------------------------------------------


def _randn(seed, shape, dtype, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").mul_(scale).to(_TYPES[dtype])


def _filter(c):
    f = gdnn.Filter2D((c["batch"], c["cin"], c["h"], c["w"]), (c["cout"], c["cin"] // c["group"], c["kh"], c["kw"]), c["group"])
    return f.pads(c["pad"], c["pad"]).strides(c["stride"], c["stride"]).dilations(c["dilation"], c["dilation"])


_STAGES = ((3, 64, 1), (4, 128, 2), (6, 256, 2), (3, 512, 2))  # blocks, width, stride of the first block


def _resnet50(batch, size, seed, classes=1000):
    """ResNet-50 v1 as an exporter writes it after folding its batch normalisations: convolutions
    with a bias, ReLU and Add nodes, max pool, global average pool, Flatten, Gemm."""
    rng = np.random.default_rng(seed)
    g = predict.Graph()

    def conv(x, cin, cout, k, stride, pad, name, gain=1.0):
        n = g.append("Conv", kernel_shape=[k, k], strides=[stride, stride], pads=[pad] * 4)
        n.addInput(x)
        n.addInput(g.addInitializer(name + ".W", (gain * math.sqrt(2.0 / (cin * k * k))) *
                                    rng.standard_normal((cout, cin, k, k), dtype=np.float32)))
        n.addInput(g.addInitializer(name + ".B", rng.uniform(-0.1, 0.1, cout).astype(np.float32)))
        return n.addOutput(name)

    def relu(x, name):
        n = g.append("Relu")
        n.addInput(x)
        return n.addOutput(name)

    t = relu(conv(g.addInput("image", predict.DataType.FLOAT, (batch, 3, size, size)), 3, 64, 7, 2, 3, "conv1"), "relu1")
    mp = g.append("MaxPool", kernel_shape=[3, 3], strides=[2, 2], pads=[1, 1, 1, 1])
    mp.addInput(t)
    t, cin = mp.addOutput("pool1"), 64
    for stage, (blocks, width, stride) in enumerate(_STAGES):
        for b in range(blocks):
            nm = "s%db%d" % (stage + 1, b)
            st = stride if b == 0 else 1
            a = relu(conv(t, cin, width, 1, st, 0, nm + ".c1"), nm + ".r1")
            a = relu(conv(a, width, width, 3, 1, 1, nm + ".c2"), nm + ".r2")
            a = conv(a, width, 4 * width, 1, 1, 0, nm + ".c3", gain=0.5)
            sc = conv(t, cin, 4 * width, 1, st, 0, nm + ".down") if b == 0 else t
            add = g.append("Add")
            add.addInput(a).addInput(sc)
            t, cin = relu(add.addOutput(nm + ".add"), nm + ".out"), 4 * width
    gap = g.append("GlobalAveragePool")
    gap.addInput(t)
    fl = g.append("Flatten", axis=1)
    fl.addInput(gap.addOutput("gap"))
    fc = g.append("Gemm", transB=1)
    fc.addInput(fl.addOutput("flat"))
    fc.addInput(g.addInitializer("fc.W", rng.standard_normal((classes, cin), dtype=np.float32) / math.sqrt(cin)))
    fc.addInput(g.addInitializer("fc.B", rng.uniform(-0.1, 0.1, classes).astype(np.float32)))
    g.addOutput(fc.addOutput("logits"))
    return g


def prepare(case, seed):
    c = case
    kind, dtype = c["kind"], c["dtype"]
    if kind == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        s = {"c": c, "A": _randn(seed, (k, m) if c["ta"] else (m, k), dtype),
             "B": _randn(seed + 1000, (n, k) if c["tb"] else (k, n), dtype, 1.0 / math.sqrt(k)),
             "Y": torch.empty((m, n), dtype=_TYPES[dtype], device="cuda")}
        if c["beta"] != 0:
            s["C"] = _randn(seed + 2000, (m, n), dtype)
        return s
    if kind == "batched":
        b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
        return {"c": c, "A": _randn(seed, (b, m, k), dtype),
                "B": _randn(seed + 1000, (b, n, k) if c["tb"] else (b, k, n), dtype, 1.0 / math.sqrt(k)),
                "Y": torch.empty((b, m, n), dtype=_TYPES[dtype], device="cuda")}
    if kind == "conv":
        f = _filter(c)
        fan = (c["cin"] // c["group"]) * c["kh"] * c["kw"]
        s = {"c": c, "f": f, "X": _randn(seed, (c["batch"], c["cin"], c["h"], c["w"]), dtype),
             "W": _randn(seed + 1000, (c["cout"], c["cin"] // c["group"], c["kh"], c["kw"]), dtype, math.sqrt(2.0 / fan)),
             "b": _randn(seed + 2000, (c["cout"],), dtype, 0.1),
             "Y": torch.empty(f.output_shape(), dtype=_TYPES[dtype], device="cuda")}
        s["R"] = _randn(seed + 3000, f.output_shape(), dtype) if c["residual"] else None
        return s
    if kind == "forward":
        p = predict.Predictor(_resnet50(c["batch"], c["size"], seed), dtype=_TYPES[dtype])
        images = _randn(seed + 1000, (c["batch"], 3, c["size"], c["size"]), dtype)
        p.set(0, images)
        for _ in range(2):  # a program's first two calls: the launches one by one, then the graph
            p.predict()
        return {"c": c, "p": p, "images": images}
    m, n = c["m"], c["n"]
    q = m if c["left"] or c["routine"] == "syrk" else n
    # a well-conditioned factor: what a Cholesky or LU factorisation leaves
    T = _randn(seed, (q, q), dtype, 0.5 / math.sqrt(q))
    T.diagonal().abs_().add_(1.0)
    s = {"c": c, "T": T, "B": _randn(seed + 1000, (m, n), dtype)}
    if c["routine"] in ("symm", "syrk"):
        s["C"] = torch.zeros((m, n) if c["routine"] == "symm" else (m, m), dtype=_TYPES[dtype], device="cuda")
    return s


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "gemm":
        A, B = state["A"], state["B"]
        if c["alpha"] == 1.0 and c["beta"] == 0.0:
            return tensor.matmul(A.t() if c["ta"] else A, B.t() if c["tb"] else B, state["Y"])
        return tensor.gemm(Transpose.Trans if c["ta"] else Transpose.NoTrans, Transpose.Trans if c["tb"] else Transpose.NoTrans,
                           c["alpha"], A, B, c["beta"], state["C"], state["Y"])
    if kind == "batched":
        return tensor.matmul(state["A"], state["B"].transpose(1, 2) if c["tb"] else state["B"], state["Y"])
    if kind == "conv":
        gdnn.conv2d_filter(state["X"], state["W"], state["Y"], state["f"], bias=state["b"], residual=state["R"],
                           activation="relu" if c["relu"] else None)
        return state["Y"]
    if kind == "forward":
        state["p"].set(0, state["images"])
        state["p"].predict()
        return state["p"].output(0)
    side = Side.Left if c["left"] else Side.Right
    uplo = Triangle.Upper if c["upper"] else Triangle.Lower
    trans = Transpose.Trans if c["trans"] else Transpose.NoTrans
    if c["routine"] == "trsm":
        return tensor.trsm(side, uplo, trans, Diagonal.NonUnit, state["T"], state["B"])
    if c["routine"] == "trmm":
        return tensor.trmm(side, uplo, trans, Diagonal.NonUnit, state["T"], state["B"])
    if c["routine"] == "symm":
        return tensor.symm(side, uplo, state["T"], state["B"], C=state["C"])
    m, n = c["m"], c["n"]
    gblas.syrk(Layout.RowMajor, uplo, Transpose.NoTrans, m, n, 1.0, state["B"].view(-1), 0, n, 0.0, state["C"].view(-1), 0, m)
    return state["C"]


def _conv_work(c):
    f = _filter(c)
    out = f.batches * f.num_kernels * f.output_h * f.output_w
    weights = f.num_kernels * (f.channels // f.group) * f.kernel_h * f.kernel_w
    elems = f.batches * f.channels * f.height * f.width + weights + f.num_kernels + out * (2 if c["residual"] else 1)
    return {"bytes": _BYTES[c["dtype"]] * elems, "flops": 2.0 * out * weights / f.num_kernels}


def _forward_work(c):
    """Every layer's arithmetic; of the bytes only what enters and leaves the network (a layer's
    output could in principle stay on the chip): images, weights, biases, logits."""
    b, h = c["batch"], c["size"]
    flops, weights = 0.0, 0

    def conv(cin, cout, k, h_out):
        nonlocal flops, weights
        flops += 2.0 * b * cout * h_out * h_out * cin * k * k
        weights += cout * cin * k * k + cout

    half = lambda v: (v - 1) // 2 + 1  # noqa: E731
    h = half(h)
    conv(3, 64, 7, h)
    h, cin = half(h), 64
    for blocks, width, stride in _STAGES:
        h = half(h) if stride == 2 else h
        for i in range(blocks):
            conv(cin, width, 1, h)
            conv(width, width, 3, h)
            conv(width, 4 * width, 1, h)
            if i == 0:
                conv(cin, 4 * width, 1, h)
            cin = 4 * width
    flops += 2.0 * b * 1000 * 2048
    weights += 1000 * 2049
    return {"bytes": _BYTES[c["dtype"]] * (weights + b * 3 * c["size"] ** 2 + b * 1000), "flops": flops}


def work(case):
    c = case
    e = _BYTES[c["dtype"]]
    if c["kind"] == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": e * (m * k + k * n + m * n * (2 if c["beta"] != 0 else 1)), "flops": 2.0 * m * n * k}
    if c["kind"] == "batched":
        b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
        return {"bytes": e * b * (m * k + k * n + m * n), "flops": 2.0 * b * m * n * k}
    if c["kind"] == "conv":
        return _conv_work(c)
    if c["kind"] == "forward":
        return _forward_work(c)
    m, n = c["m"], c["n"]
    q = m if c["left"] else n
    if c["routine"] == "syrk":  # one triangle of an m x m product
        return {"bytes": e * (m * n + m * (m + 1) // 2), "flops": 1.0 * m * (m + 1) * n}
    if c["routine"] == "symm":
        return {"bytes": e * (q * (q + 1) // 2 + 2 * m * n), "flops": 2.0 * m * n * q}
    return {"bytes": e * (q * (q + 1) // 2 + 2 * m * n), "flops": 1.0 * m * n * q}


def tolerance(case):
    """Measured against the same call in 64-bit arithmetic, times about four. A 16-bit result
    carries its own rounding (2e-4 in fp16, 1.7e-3 in bf16); a whole network carries that of every
    layer (3e-4 in fp16, 2.6e-5 in fp32); fp32 products are sums of three tf32 products: 4e-7 to 4e-6."""
    d = case["dtype"]
    if case["kind"] == "forward":
        return {"rel": {"f16": 4e-3, "bf16": 3e-2, "f32": 1e-4}[d]}
    return {"rel": {"f16": 1e-3, "bf16": 7e-3, "f32": 1.5e-5}[d]}


def exact(case, seed):
    """What ``run`` returns for these inputs in 64-bit arithmetic, written with plain torch."""
    c = case
    kind = c["kind"]
    if kind == "forward":
        return _exact_forward(c, seed)
    s = prepare(case, seed)
    if kind == "gemm":
        A, B = s["A"].double(), s["B"].double()
        y = c["alpha"] * ((A.t() if c["ta"] else A) @ (B.t() if c["tb"] else B))
        return y + c["beta"] * s["C"].double() if c["beta"] != 0 else y
    if kind == "batched":
        return torch.bmm(s["A"].double(), (s["B"].transpose(1, 2) if c["tb"] else s["B"]).double())
    if kind == "conv":
        return _conv64(s["X"].double(), s["W"].double(), s["b"].double(), c["stride"], c["pad"], c["dilation"], c["group"],
                       s["R"], c["relu"])
    T, B = s["T"].double(), s["B"].double()
    if c["routine"] == "syrk":
        full = B @ B.t()
        return torch.triu(full) if c["upper"] else torch.tril(full)
    part = torch.triu(T) if c["upper"] else torch.tril(T)
    if c["routine"] == "symm":
        part = part + part.t() - torch.diag(part.diagonal())
        return part @ B if c["left"] else B @ part
    upper = c["upper"] != c["trans"]
    part = part.t() if c["trans"] else part
    if c["routine"] == "trmm":
        return part @ B if c["left"] else B @ part
    return torch.linalg.solve_triangular(part, B, upper=upper, left=c["left"])


def _conv64(x, w, b, stride, pad, dilation, group, residual, relu):
    """One filter tap after the other: a strided window of the bordered images times its weights."""
    n, cin, h, wd = x.shape
    cout, cg, kh, kw = w.shape
    oh = (h + 2 * pad - dilation * (kh - 1) - 1) // stride + 1
    ow = (wd + 2 * pad - dilation * (kw - 1) - 1) // stride + 1
    xp = torch.nn.functional.pad(x, (pad, pad, pad, pad)) if pad else x
    y = b.view(1, group, cout // group, 1).expand(n, group, cout // group, oh * ow).contiguous()
    wg = w.view(group, cout // group, cg, kh, kw)
    for i in range(kh):
        for j in range(kw):
            win = xp[:, :, i * dilation:i * dilation + (oh - 1) * stride + 1:stride,
                     j * dilation:j * dilation + (ow - 1) * stride + 1:stride]
            y += torch.matmul(wg[:, :, :, i, j], win.reshape(n, group, cg, oh * ow))
    y = y.view(n, cout, oh, ow)
    if residual is not None:
        y += residual.double()
    return y.clamp_(min=0) if relu else y


def _exact_forward(c, seed):
    """ResNet-50 on the parameters of `_resnet50`, as the case's type holds them."""
    t = _TYPES[c["dtype"]]
    graph = _resnet50(c["batch"], c["size"], seed)
    par = {v.name: torch.from_numpy(v.initializer).cuda().to(t).double() for v in graph.inputs if v.has_initializer()}

    def conv(x, name, stride, pad, residual=None, relu=True):
        return _conv64(x, par[name + ".W"], par[name + ".B"], stride, pad, 1, 1, residual, relu)

    images = _randn(seed + 1000, (c["batch"], 3, c["size"], c["size"]), c["dtype"])
    logits = []
    for part in images.split(16):
        x = conv(part.double(), "conv1", 2, 3)
        x = torch.nn.functional.max_pool2d(x, 3, 2, 1)
        for stage, (blocks, _, stride) in enumerate(_STAGES):
            for b in range(blocks):
                nm, st = "s%db%d" % (stage + 1, b), stride if b == 0 else 1
                a = conv(conv(x, nm + ".c1", st, 0), nm + ".c2", 1, 1)
                x = conv(a, nm + ".c3", 1, 0, conv(x, nm + ".down", st, 0, relu=False) if b == 0 else x)
        logits.append(x.mean((2, 3)) @ par["fc.W"].t() + par["fc.B"])
    return torch.cat(logits)
