"""Performance cases of the framework: the work a program built on `torch.GPUTensor` and the `nn` modules has it do, called
through the public entry points.

    listed()            the cases timed by name
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call
    run(state)          one pass and its outputs
    work(case)          bytes and floating-point operations the pass cannot do without
    tolerance(case)     how far another correct implementation may be off

Six kinds of work (`case["kind"]`):

    train     a whole SGD step of one of the two classifiers: zero the gradients, forward, criterion, backward, momentum update
    classify  a host batch in, the network's log-probabilities out on the host
    block     convolution -> ReLU -> max-pooling, forward and backward with all three convolution passes
    addmm     the matrix product behind `nn.Linear`, in the four transpose layouts, overwriting or accumulating
    math      the elementwise functions and reductions of `torch.GPUTensor` on matrices, transposed operands among them
    linear    a fully connected layer, forward and backward, over rows of features

`mode` is the math mode: "fp32x3" (FP32-accurate, the default) or "bf16" (opt-in)."""
import math

import numpy as np
import torch

import mcw_cppamp_torch_b200 as gt
from mcw_cppamp_torch_b200 import configs, nn

CLASSES = 1000
IMAGE = 224
LR, MOMENTUM = 0.01, 0.9


def listed():
    return [
        # the data-parallel configuration's global batch on one GPU: the throughput end of training
        {"name": "train_alexnet_1024", "kind": "train", "net": "alexnet", "batch": 1024, "mode": "fp32x3"},
        # the rows one of eight ranks gets of that batch
        {"name": "train_alexnet_128", "kind": "train", "net": "alexnet", "batch": 128, "mode": "fp32x3"},
        # the opt-in BF16 mode on an ordinary batch
        {"name": "train_alexnet_256_bf16", "kind": "train", "net": "alexnet", "batch": 256, "mode": "bf16"},
        # the deeper configuration: 3x3 layers on large planes, 2x2 pooling, a first layer over three planes at stride 1
        {"name": "train_vgg_a_64", "kind": "train", "net": "vgg_a", "batch": 64, "mode": "fp32x3"},
        # serving one image: latency and the weights' traffic count
        {"name": "classify_alexnet_1", "kind": "classify", "net": "alexnet", "batch": 1, "mode": "fp32x3"},
        # the last, partly filled batch of an evaluation run
        {"name": "classify_vgg_a_13", "kind": "classify", "net": "vgg_a", "batch": 13, "mode": "fp32x3"},
        # the single-block configuration: 11x11 stride 4 over three planes, gradInput included
        {"name": "block_3x64_k11s4", "kind": "block", "N": 16, "C": 3, "H": 224, "W": 224, "K": 64, "k": 11, "stride": 4, "pad": 2,
         "pool": 3, "pool_stride": 2, "mode": "fp32x3"},
        # a small layer whose sizes are multiples of nothing, as the module's own tests draw them
        {"name": "block_ragged", "kind": "block", "N": 6, "C": 17, "H": 45, "W": 37, "K": 29, "k": 5, "stride": 1, "pad": 1,
         "pool": 2, "pool_stride": 2, "mode": "fp32x3"},
        # the tensor-math configuration's matrix product
        {"name": "addmm_4096", "kind": "addmm", "m": 4096, "n": 4096, "k": 4096, "t1": False, "t2": False, "beta": 0.0,
         "mode": "fp32x3"},
        # rows, columns and pitch that no tile or 16-byte access divides, a transposed operand, accumulation
        {"name": "addmm_ragged", "kind": "addmm", "m": 1000, "n": 777, "k": 1531, "t1": True, "t2": False, "beta": 1.0,
         "mode": "fp32x3"},
        # the tensor-math configuration's elementwise and reduction work: HBM bandwidth
        {"name": "math_8192", "kind": "math", "rows": 8192, "cols": 8192},
        # the same calls on a matrix of a few kilobytes: what a call costs by itself
        {"name": "math_small", "kind": "math", "rows": 40, "cols": 101},
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        kind = rng.choice(["train", "train", "classify", "block", "block", "addmm", "addmm", "linear", "math", "math"])
        mode = "bf16" if rng.random() < 0.25 else "fp32x3"
        if kind == "train":
            net = rng.choice(["alexnet", "alexnet", "vgg_a"])
            case = {"kind": kind, "net": net, "batch": _log(rng, 2, 900 if net == "alexnet" else 56), "mode": mode}
        elif kind == "classify":
            net = rng.choice(["alexnet", "vgg_a"])
            case = {"kind": kind, "net": net, "batch": _log(rng, 1, 128 if net == "alexnet" else 24), "mode": mode}
        elif kind == "block":
            side = _log(rng, 9, 128)
            k = rng.choice([3, 3, 5, 7, 11])
            case = {"kind": kind, "N": _log(rng, 1, 128), "C": _log(rng, 1, 256), "H": side, "W": max(9, side + rng.randint(-4, 4)),
                    "K": _log(rng, 8, 256), "k": k, "stride": rng.choice([1, 1, 1, 2, 4]) if k > 3 else 1, "pad": rng.choice([0, 1, k // 2]),
                    "pool": rng.choice([2, 3]), "pool_stride": 2, "mode": mode}
            oh, ow = _conv_out(case)
            if case["stride"] > 1 and work(case)["flops"] > 2e10:      # strided layers are first layers: few planes, or small images
                continue
            if min(oh, ow) < 3 or case["N"] * (case["C"] * case["H"] * case["W"] + case["K"] * oh * ow) > 1 << 27:
                continue
        elif kind == "addmm":
            case = {"kind": kind, "m": _log(rng, 8, 4096), "n": _log(rng, 8, 4096), "k": _log(rng, 8, 4096), "t1": rng.random() < 0.5,
                    "t2": rng.random() < 0.5, "beta": rng.choice([0.0, 1.0]), "mode": mode}
        elif kind == "linear":
            case = {"kind": kind, "rows": _log(rng, 1, 1024), "inputs": _log(rng, 64, 9216), "outputs": _log(rng, 10, 4096), "mode": mode}
        else:
            case = {"kind": kind, "rows": _log(rng, 16, 8192), "cols": _log(rng, 16, 8192)}
        if work(case)["flops"] <= 2.5e12:
            return case


# ------------------------------------------------------------------ inputs
class _Zeros:
    """Stands in for the host generator while a module is built: its parameters are drawn on the device afterwards."""

    def uniform(self, shape, a, b):
        return np.zeros(shape, np.float32)


def _wrap(t):
    """A torch.GPUTensor over a (contiguous) torch tensor's memory."""
    L = gt.lib()
    s = L.THGPUStorage_newWithData(t.data_ptr(), t.numel())
    g = gt.GPUTensor(_ptr=L.THGPUTensor_newWithStorage1d(s, 0, t.numel(), 1)).view(*t.shape)
    L.THGPUStorage_free(s)
    return g


class _State:
    """Device tensors of one case, each as a torch tensor (kept alive, and what run() returns) and as a torch.GPUTensor."""

    def __init__(self, case, seed):
        self.case = case
        self.rand = torch.Generator(device="cuda")
        self.rand.manual_seed(seed)
        self.torch, self.gpu = {}, {}

    def put(self, name, t):
        self.torch[name] = t
        self.gpu[name] = _wrap(t)
        return self.gpu[name]

    def empty(self, name, *shape):
        return self.put(name, torch.zeros(shape, device="cuda"))

    def normal(self, name, *shape):
        return self.put(name, torch.randn(shape, device="cuda", generator=self.rand))

    def uniform(self, name, *shape):
        return self.put(name, torch.rand(shape, device="cuda", generator=self.rand).mul_(2).sub_(1))


def _flatten(s, net):
    """The parameters of `net` in one buffer and their gradients in another, drawn as the modules' reset() does."""
    n = sum(t.nElement() for m in net.modules_list() if m.parameters() for t in m.parameters()[0])
    w, g = torch.empty(n, device="cuda"), torch.zeros(n, device="cuda")
    s.torch["weights"], s.torch["gradient"] = w, g
    s.gpu["weights"], s.gpu["gradient"] = net.getParameters(flat=(w.data_ptr(), g.data_ptr(), n))
    gt.synchronize()
    off = 0
    for m in net.modules_list():
        p = m.parameters()
        if p:
            stdv = 1.0 / math.sqrt(m.weight.size(2))
            for t in p[0]:
                w[off:off + t.nElement()].uniform_(-stdv, stdv, generator=s.rand)
                off += t.nElement()
    return n


def prepare(case, seed):
    gt.set_math_mode(case.get("mode", "fp32x3"))
    s = _State(case, seed)
    kind = case["kind"]
    if kind in ("train", "classify"):
        s.net = getattr(configs, case["net"])(rng=_Zeros()).gpu()
        n = _flatten(s, s.net)
        b = case["batch"]
        s.net.modules[-1].output = s.empty("logprob", b, CLASSES)
        if kind == "train":
            s.crit = nn.ClassNLLCriterion()
            s.crit.outputTensor = s.empty("loss", 1)
            s.empty("velocity", n)
            s.uniform("images", b, 3, IMAGE, IMAGE)
            s.put("labels", torch.randint(1, CLASSES + 1, (b,), device="cuda", generator=s.rand).float())
        else:
            s.images = np.random.default_rng(seed).random((b, 3, IMAGE, IMAGE), dtype=np.float32) * 2 - 1
            s.answer = np.zeros((b, CLASSES), np.float32)
            s.empty("images", b, 3, IMAGE, IMAGE)
    elif kind == "block":
        c = case
        conv = nn.SpatialConvolutionMM(c["C"], c["K"], c["k"], c["k"], c["stride"], c["stride"], c["pad"], rng=_Zeros())
        pool = nn.SpatialMaxPooling(c["pool"], c["pool"], c["pool_stride"], c["pool_stride"])
        s.net = nn.Sequential().add(conv).add(nn.ReLU()).add(pool).gpu()
        _flatten(s, s.net)
        oh, ow = _conv_out(c)
        ph, pw = ((v - c["pool"]) // c["pool_stride"] + 1 for v in (oh, ow))
        s.uniform("input", c["N"], c["C"], c["H"], c["W"])
        conv.gradInput = s.empty("gradInput", c["N"], c["C"], c["H"], c["W"])
        pool.output = s.empty("output", c["N"], c["K"], ph, pw)
        s.normal("gradOutput", c["N"], c["K"], ph, pw)
    elif kind == "linear":
        c = case
        s.net = nn.Linear(c["inputs"], c["outputs"], rng=_Zeros()).gpu()
        _flatten(s, s.net)
        s.uniform("input", c["rows"], c["inputs"])
        s.normal("gradOutput", c["rows"], c["outputs"])
        s.net.output = s.empty("output", c["rows"], c["outputs"])
        s.net.gradInput = s.empty("gradInput", c["rows"], c["inputs"])
    elif kind == "addmm":
        m, n, k = case["m"], case["n"], case["k"]
        s.normal("m1", *((k, m) if case["t1"] else (m, k)))
        s.normal("m2", *((n, k) if case["t2"] else (k, n)))
        s.normal("result", m, n)
    else:
        r, c = case["rows"], case["cols"]
        s.normal("X", r, c)
        s.normal("Y", r, c)
        s.normal("Z", c, r)
        for name in ("cadd", "cmul", "cadd_transposed", "copy_transposed", "exp", "addcmul"):
            s.empty(name, r, c)
        for name in ("sum1", "max1", "index1"):
            s.empty(name, 1, c)
        for name in ("sum2", "max2", "index2"):
            s.empty(name, r, 1)
    torch.cuda.synchronize()
    gt.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    return _RUN[s.case["kind"]](s)


def _run_train(s):
    t, g = s.torch, s.gpu
    g["gradient"].zero()
    out = s.net.forward(g["images"])
    s.crit.updateOutput(out, g["labels"], read_back=False)
    s.net.backward(g["images"], s.crit.updateGradInput(out, g["labels"]))
    gt.lib().THGPUNN_SGD_update(g["weights"].cdata, g["gradient"].cdata, g["velocity"].cdata, LR, MOMENTUM)
    return {k: t[k] for k in ("loss", "logprob", "gradient", "weights", "velocity")}


def _run_classify(s):
    return s.net.forward(s.gpu["images"].copy(s.images)).float(s.answer)


def _run_block(s):
    s.net.zeroGradParameters()
    s.net.forward(s.gpu["input"])
    s.net.backward(s.gpu["input"], s.gpu["gradOutput"])
    return {k: s.torch[k] for k in ("output", "gradInput", "gradient")}


def _run_linear(s):
    s.net.zeroGradParameters()
    s.net.forward(s.gpu["input"])
    s.net.backward(s.gpu["input"], s.gpu["gradOutput"])
    return {k: s.torch[k] for k in ("output", "gradInput", "gradient")}


def _run_addmm(s):
    m1, m2 = s.gpu["m1"], s.gpu["m2"]
    s.gpu["result"].addmm(s.case["beta"], 1.0, m1.t() if s.case["t1"] else m1, m2.t() if s.case["t2"] else m2)
    return s.torch["result"]


def _run_math(s):
    g = s.gpu
    x, y, zt = g["X"], g["Y"], g["Z"].t()
    g["cadd"].add(x, 0.5, y)
    g["cmul"].cmul(x, y)
    g["cadd_transposed"].add(x, 0.5, zt)
    g["copy_transposed"].copy(zt)
    g["exp"].exp(x)
    g["addcmul"].addcmul(x, 0.5, x, y)
    g["sum1"].sum(x, 1)
    g["sum2"].sum(x, 2)
    L = gt.lib()
    L.THGPUTensor_max(g["max1"].cdata, g["index1"].cdata, x.cdata, 0)
    L.THGPUTensor_max(g["max2"].cdata, g["index2"].cdata, x.cdata, 1)
    out = {k: s.torch[k] for k in ("cadd", "cmul", "cadd_transposed", "copy_transposed", "exp", "addcmul", "sum1", "sum2", "max1", "max2",
                                   "index1", "index2")}
    out["sum"], out["max"], out["norm"] = g["exp"].sum(), x.max(), x.norm()
    return out


_RUN = {"train": _run_train, "classify": _run_classify, "block": _run_block, "linear": _run_linear, "addmm": _run_addmm,
        "math": _run_math}


# ------------------------------------------------------------------ what a pass cannot do without
def _conv_out(c):
    return tuple((c[d] + 2 * c["pad"] - c["k"]) // c["stride"] + 1 for d in ("H", "W"))


def _net_work(net):
    """(parameters, forward FLOPs of an image, FLOPs of an image's training step: no gradInput of the first layer)"""
    convs = configs.ALEXNET_CONVS if net == "alexnet" else [(ci, co, 3, 1, 1, pool) for ci, co, pool in configs.VGG_A_CONVS]
    fcs = configs.ALEXNET_FC if net == "alexnet" else configs.VGG_A_FC
    h, fwd, step, n = IMAGE, 0, 0, 0
    for i, (ci, co, k, st, p, pool) in enumerate(convs):
        h = (h + 2 * p - k) // st + 1
        f = 2 * co * ci * k * k * h * h
        fwd += f
        step += f * (2 if i == 0 else 3)
        n += co * ci * k * k + co
        if pool:
            h = (h - 3) // 2 + 1 if net == "alexnet" else h // 2
    for fi, fo in fcs:
        fwd += 2 * fi * fo
        step += 6 * fi * fo
        n += fi * fo + fo
    return n, fwd, step


def work(case):
    kind = case["kind"]
    if kind in ("train", "classify"):
        n, fwd, step = _net_work(case["net"])
        b = case["batch"]
        io = b * (3 * IMAGE * IMAGE + CLASSES)
        if kind == "classify":
            return {"bytes": 4 * (io + n), "flops": b * fwd}
        return {"bytes": 4 * (io + 5 * n), "flops": b * step}      # weights and velocity read and written, gradient written
    if kind == "block":
        c = case
        oh, ow = _conv_out(c)
        ph, pw = ((v - c["pool"]) // c["pool_stride"] + 1 for v in (oh, ow))
        per = c["C"] * c["k"] * c["k"]
        return {"bytes": 4 * (2 * c["N"] * c["C"] * c["H"] * c["W"] + 2 * c["N"] * c["K"] * ph * pw + 2 * c["K"] * (per + 1)),
                "flops": 6 * c["N"] * c["K"] * per * oh * ow}
    if kind == "linear":
        r, i, o = case["rows"], case["inputs"], case["outputs"]
        return {"bytes": 4 * (2 * r * i + 2 * r * o + 2 * (i + 1) * o), "flops": 6 * r * i * o}
    if kind == "addmm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4 * (m * k + k * n + (2 if case["beta"] else 1) * m * n), "flops": 2 * m * n * k}
    r, c = case["rows"], case["cols"]
    # each call reads its operands and writes its result once: four calls of 12 bytes an element (one of them addcmul, whose
    # first two operands are the same matrix), two of 8, seven reductions of 4
    return {"bytes": 4 * (r * c * (4 * 3 + 2 * 2 + 7) + 3 * (r + c)), "flops": 20 * r * c}


def tolerance(case):
    kind, bf16 = case["kind"], case.get("mode") == "bf16"
    if kind in ("train", "block"):
        # A correct FP32 pass may decide a ReLU or a pooling window the other way where a sum lies within its rounding of a
        # tie.  With rounding near 3e-7 of a layer's spread a share of about 3e-7 of the decisions turns, and a gradient that
        # sums such terms moves by its root, a little under 1e-3; a single element fed by a turned decision moves by a good
        # part of its own size.
        return {"rel": 1e-2 if bf16 else 1e-3, "max": 0.9}
    if kind in ("classify", "addmm", "linear"):
        return {"rel": 1e-2 if bf16 else 1e-5}
    return {"rel": 1e-5}
