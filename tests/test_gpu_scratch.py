"""Device memory behind the products: zeroed words inside recordings, records over many groups of images, scratch that is not to be had,
planes that are kept."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from test_gpu_fp16_pairs import REL, gt, products, randn  # noqa: F401

pytestmark = pytest.mark.gpu


def wrap(gt, t):  # noqa: F811
    """A torch.GPUTensor over a torch tensor's memory."""
    L = gt.lib()
    s = L.THGPUStorage_newWithData(t.data_ptr(), t.numel())
    g = gt.GPUTensor(_ptr=L.THGPUTensor_newWithStorage1d(s, 0, t.numel(), 1)).view(*t.shape)
    L.THGPUStorage_free(s)
    return g


def test_recorded_products(gt):  # noqa: F811
    """Enough products in a recording to use up the zeroed words several times over; launches outside it come before, between and after its runs."""
    n, k = 3072, 2048                     # (more tiles than clusters: items are handed out)
    a, b = [randn(i, n, k) * 2.0 ** (15 * i) for i in range(3)], [randn(i, k, n) * 2.0 ** (-15 * i) for i in range(3)]
    want = [x.double() @ y.double() for x, y in zip(a, b)]
    mass = [x.abs().double() @ y.abs().double() for x, y in zip(a, b)]
    out = [torch.empty(n, n, device="cuda") for _ in a]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    gt.lib().THGPUSetStream(ctypes.c_void_p(stream.cuda_stream))
    try:
        A, B, C = ([wrap(gt, t) for t in ts] for ts in (a, b, out))

        def run(times):
            for _ in range(times):
                for x, y, z in zip(A, B, C):
                    z.addmm(0.0, 1.0, x, y)

        def check():
            gt.synchronize()
            for c, w, m in zip(out, want, mass):
                assert torch.all((c.double() - w).abs() <= REL * m)
                c.fill_(float("nan"))
            torch.cuda.synchronize()

        before = products(gt)
        run(200)                          # every word has been used
        assert products(gt)[1] - before[1] == 600
        check()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run(130)
        torch.cuda.synchronize()
        for _ in range(200):              # each result is looked at: a launch that missed its words leaves tiles out
            run(1)
            check()
        with torch.cuda.stream(stream):
            for _ in range(3):
                graph.replay()
                check()
                run(7)
                check()
        del graph
    finally:
        gt.synchronize()
        gt.lib().THGPUSetStream(None)


def test_hundreds_of_groups(gt):  # noqa: F811
    """A batch whose planes come to 350 groups of one image: an image's gradients are the same, bit for bit, wherever it stands."""
    N, C, H, K, k = 350, 3, 1400, 1, 11
    image, gout, w = randn(0, C, H, H), randn(1, K, H, H), randn(5, K, C, k, k)
    x, go = torch.zeros(N, C, H, H, device="cuda"), torch.zeros(N, K, H, H, device="cuda")
    m = gt.nn.SpatialConvolutionMM(C, K, k, k, 1, 1, k // 2)
    m.weight.reshape(-1)[:] = w.cpu().numpy().reshape(-1)
    m.gpu()
    gi = torch.empty_like(x)
    torch.cuda.synchronize()
    m.gradInput = wrap(gt, gi)
    X, GO = wrap(gt, x), wrap(gt, go)
    got = []
    for i in (0, N - 5):
        x[i], go[i] = image, gout
        torch.cuda.synchronize()
        m.zeroGradParameters()
        before = products(gt)
        m.backward(X, GO)
        gt.synchronize()
        assert products(gt)[1] - before[1] == 2 * N
        got.append((gi[i].clone(), torch.from_numpy(m.gradWeight.float())))
        x[i], go[i] = 0, 0
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])

    def grads(f):
        xi, wi = f(image)[None].double().requires_grad_(), f(w).double().requires_grad_()
        return torch.autograd.grad(torch.nn.functional.conv2d(xi, wi, None, 1, k // 2), (xi, wi), f(gout)[None].double())
    (a, b), (am, bm) = grads(lambda t: t), grads(torch.abs)
    assert torch.all((got[0][0].double() - a[0]).abs() <= REL * am[0])
    assert torch.all((got[0][1].cuda().double().view_as(w) - b).abs() <= (REL + 2.0 ** -24 * (H * H / 32 + 64)) * bm)


FULL_DEVICE = """
import torch, mcw_cppamp_torch_b200 as gt
from test_gpu_fp16_pairs import REL, products, randn
from test_gpu_scratch import wrap
m, n, k = 16384, 8192, 16384
a, b, c = randn(1, m, k), randn(2, k, n), torch.empty(m, n, device="cuda")
rows = torch.arange(0, m, 511, device="cuda")
want, mass = a[rows].double() @ b.double(), a[rows].abs().double() @ b.abs().double()
A, B, C = wrap(gt, a), wrap(gt, b), wrap(gt, c)
s = wrap(gt, torch.ones(256, 256, device="cuda"))
wrap(gt, torch.empty(256, 256, device="cuda")).addmm(0.0, 1.0, s, s)
gt.synchronize()
torch.cuda.synchronize()
torch.cuda.empty_cache()
fill = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")     # the pairs take 1.6 GB
for form in (0, 2):
    before = products(gt)
    C.addmm(0.0, 1.0, A, B)
    gt.synchronize()
    assert [x - y for x, y in zip(products(gt), before)] == [form == 0, form == 2], form
    assert torch.all((c[rows].double() - want).abs() <= REL * mass)
    fill = None
    torch.cuda.empty_cache()
"""


FULL_DEVICE_CONVOLUTION = """
import torch, mcw_cppamp_torch_b200 as gt
from test_gpu_fp16_pairs import REL, products, randn
from test_gpu_scratch import wrap
N, C, H, K = 1024, 96, 56, 96
x, w, go, gi = randn(1, N, C, H, H), randn(2, K, C, 3, 3), randn(3, N, K, H, H), torch.empty(N, C, H, H, device="cuda")
out = torch.empty(N, K, H, H, device="cuda")
m = gt.nn.SpatialConvolutionMM(C, K, 3, 3, 1, 1, 1)
m.weight.reshape(-1)[:] = w.cpu().numpy().reshape(-1)
m.bias[:] = 0
m.gpu()
m.output, m.gradInput = wrap(gt, out), wrap(gt, gi)
X, GO = wrap(gt, x), wrap(gt, go)
image = [0, N - 1]
def grads(f):
    xi, wi = f(x[image]).double().requires_grad_(), f(w).double().requires_grad_()
    o = torch.nn.functional.conv2d(xi, wi, None, 1, 1)
    return (o.detach(),) + torch.autograd.grad(o, xi, f(go[image]).double())
want, mass = grads(lambda t: t), grads(torch.abs)
def fill(room):
    gt.synchronize()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
s = wrap(gt, torch.ones(256, 256, device="cuda"))
wrap(gt, torch.empty(256, 256, device="cuda")).addmm(0.0, 1.0, s, s)
full = fill(1500 << 20)                # planes: 1.23 GB, as pairs 1.64
before = products(gt)
m.forward(X)
del full
full = fill(1500 << 20)                # gradOutput's planes likewise
m.zeroGradParameters()
m.backward(X, GO)
gt.synchronize()
assert [b - a for b, a in zip(products(gt), before)] == [3, 0], products(gt)
for got, a, b in zip((out, gi), want, mass):
    assert torch.all((got[image].double() - a).abs() <= REL * b)
del full
torch.cuda.empty_cache()
before = products(gt)
m.forward(X)
m.backward(X, GO)
gt.synchronize()
assert [b - a for b, a in zip(products(gt), before)] == [0, 3], products(gt)
for got, a, b in zip((out, gi), want, mass):
    assert torch.all((got[image].double() - a).abs() <= REL * b)
"""


# A forward pass that fails leaves no planes: neither one that ends for want of memory (the filter's form comes before the planes are
# made) nor one over new values in the input's memory (the planes of the old ones).
REFUSED_FORWARD = """
import torch, mcw_cppamp_torch_b200 as gt
from test_gpu_fp16_pairs import randn
from test_gpu_scratch import wrap
N, C, H, K, k = 4, 1024, 8, 8192, 3
x, w, go = randn(1, N, C, H, H), randn(2, K, C * k * k), randn(3, N, K, H, H)
small, gs = randn(4, 256, C * k * k), randn(5, N, 256, H, H)
out = [torch.empty(N, p, H, H, device="cuda") for p in (K, 256)]
grad = [[torch.zeros_like(f) for f in (w, small)] for _ in range(2)]
bias = torch.zeros(K, device="cuda")
def layer(filters, output, gradWeight):
    m = gt.nn.SpatialConvolutionMM(1, 1, 1, 1).gpu()
    m.kW, m.kH, m.padding = k, k, 1
    m.weight, m.bias, m.output, m.gradWeight = wrap(gt, filters), wrap(gt, bias[:len(filters)]), wrap(gt, output), wrap(gt, gradWeight)
    m.gradBias = wrap(gt, torch.zeros(len(filters), device="cuda"))
    return m
X = wrap(gt, x)
gt.set_math_mode("bf16")
first, second = layer(w, out[0], grad[0][0]), layer(small, out[1], grad[0][1])
second.forward(X)                      # 4.7 MB of filters, and planes of x
assert second.finput.dim() == 5
gt.synchronize()
x.mul_(-1.5)
torch.cuda.synchronize()
torch.cuda.empty_cache()
full = torch.empty(torch.cuda.mem_get_info()[0] - (96 << 20), dtype=torch.uint8, device="cuda")     # the filter's form: 151 MB
second.bias = first.bias
for m, why in ((first, "no room"), (second, "bias")):
    try:
        m.forward(X)
    except gt.THCError as e:
        assert why in str(e), e
    else:
        raise AssertionError("nothing failed")
del full
torch.cuda.empty_cache()
for m, g in ((first, go), (second, gs)):
    m.accGradParameters(X, wrap(gt, g))
for m, f, g, o in ((layer(w, out[0], grad[1][0]), w, go, 0), (layer(small, out[1], grad[1][1]), small, gs, 1)):
    m.accGradParameters(X, wrap(gt, g))
    gt.synchronize()
    assert grad[1][o].abs().max() > 1 and torch.equal(grad[0][o], grad[1][o]), o
"""


@pytest.mark.parametrize("program", [FULL_DEVICE, FULL_DEVICE_CONVOLUTION, REFUSED_FORWARD])
def test_product_on_a_full_device(gt, program):  # noqa: F811
    """Pairs are copies; where there is no room for them the product runs over the operands as they lie, or planes in FP32 where those are
    smaller.  (A process of its own: this one's workspace has grown already.)"""
    tests = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(tests), tests]))
    r = subprocess.run([sys.executable, "-c", program], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("N,kept", [(64, False), (4, True)])
def test_planes_of_the_bf16_mode(gt, N, kept):  # noqa: F811
    """A layer that the BF16 mode leaves FP32-accurate keeps planes for its weight gradient where that reads them, not where it runs over pairs."""
    C, H, K, k = 64, 56, 32, 3
    x, w, go = randn(1, N, C, H, H), randn(2, K, C, k, k), randn(3, N, K, H, H)
    m = gt.nn.SpatialConvolutionMM(C, K, k, k, 1, 1, 1)
    m.weight.reshape(-1)[:] = w.cpu().numpy().reshape(-1)
    m.gpu()
    gt.set_math_mode("bf16")
    try:
        xg, gog = gt.gpu(x.cpu().numpy()), gt.gpu(go.cpu().numpy())
        m.forward(xg)
        assert (m.finput.dim() > 0) == kept
        m.zeroGradParameters()
        before = products(gt)
        m.accGradParameters(xg, gog)
        assert [a - b for a, b in zip(products(gt), before)] == ([1, 0] if kept else [0, 1])
        gw = torch.from_numpy(m.gradWeight.float()).cuda().double().view_as(w)
    finally:
        gt.set_math_mode("fp32x3")

    def grad(f):
        wi = f(w).double().requires_grad_()
        return torch.autograd.grad(torch.nn.functional.conv2d(f(x).double(), wi, None, 1, 1), wi, f(go).double())[0]
    assert torch.all((gw - grad(lambda t: t)).abs() <= (REL + 2.0 ** -24 * (go.numel() / K / 32 + 64)) * grad(torch.abs))


def test_filter_of_a_billion_weights(gt):  # noqa: F811
    """65 output planes are 96 in spans of 32, for which 31 bits count the repacked weights, and 128 in spans of 64, for which they do not."""
    N, C, H, K, k = 16, 4096, 64, 65, 64
    w, go = randn(1, K, C * k * k), randn(2, N, K, 1, 1)
    x, gi = torch.empty(N, C, H, H, device="cuda"), torch.empty(N, C, H, H, device="cuda")
    m = gt.nn.SpatialConvolutionMM(1, 1, 1, 1)
    m.gpu()
    torch.cuda.synchronize()
    m.kW = m.kH = k
    m.weight, m.gradInput = wrap(gt, w), wrap(gt, gi)
    m.updateGradInput(wrap(gt, x), wrap(gt, go))
    gt.synchronize()
    for at in (slice(0, 5000), slice(C * k * k - 5000, C * k * k)):
        a, b = go.view(N, K).double(), w[:, at].double()
        assert torch.all((gi.view(N, -1)[:, at].double() - a @ b).abs() <= REL * (a.abs() @ b.abs()))
