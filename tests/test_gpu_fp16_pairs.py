"""Products over FP16 pairs: remainders of every layout and form, operands whose range the pairs do not hold (the same launch then
multiplies FP32 values), planes kept from a forward pass that the backward pass needs in FP32.  Reference: torch in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# dropped terms and truncating chains, of the sum of |products|: the bound of the TF32 products, which pairs stay below
REL = 2.0 ** -19


@pytest.fixture(scope="module")
def gt():
    import mcw_cppamp_torch_b200 as gt
    return gt


def products(gt):
    """Products so far over FP32 values and over pairs."""
    return [gt.lib().THGPUProductCount(form) for form in (0, 2)]


def randn(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, device="cuda", generator=g)


def wide_rows(t, dim, span):
    """Slices along `dim` scaled by powers of two from 2^-span to 1, a third of them zero."""
    n = t.size(dim)
    s = torch.exp2(-torch.linspace(0, span, n, device="cuda").round())
    s[torch.arange(n, device="cuda") % 3 == 1] = 0
    shape = [1] * t.dim()
    shape[dim] = n
    return t * s.view(shape)


def addmm(gt, a, b, c, t1, t2, beta, pairs=True):
    A, B, C = (gt.gpu(x.cpu().numpy()) for x in (a.t().contiguous() if t1 else a, b.t().contiguous() if t2 else b, c))
    before = products(gt)
    C.addmm(beta, 1.0, A.t() if t1 else A, B.t() if t2 else B)
    assert [n - b for n, b in zip(products(gt), before)] == ([0, 1] if pairs else [1, 0])
    return torch.from_numpy(C.float()).cuda().double()


def check_addmm(gt, a, b, t1=False, t2=False, beta=0.0, rows=slice(None), cols=slice(None), pairs=True):
    c = randn(9, a.size(0), b.size(1))
    got = addmm(gt, a, b, c, t1, t2, beta, pairs)[rows, cols]
    a, b, c = a[rows].double(), b[:, cols].double(), beta * c[rows, cols].double()
    assert torch.all((got - (a @ b + c)).abs() <= REL * (a.abs() @ b.abs() + c.abs()))


@pytest.mark.parametrize("t1,t2", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k,beta", [(1500, 3001, 2222, 0.0), (2049, 1793, 2047, 1.0), (4097, 129, 4095, 0.0), (130, 4100, 4033, 1.0),
                                        (2048, 2048, 2048, 0.0), (2304, 2304, 2304, 0.0), (2304, 2304, 2304, 1.0), (1500, 3001, 2222, 0.5),
                                        (4097, 1025, 4033, 1.0)])
def test_layouts_and_remainders(gt, m, n, k, beta, t1, t2):
    check_addmm(gt, randn(m, m, k), randn(n, k, n), t1, t2, beta, pairs=(m, n) not in [(2049, 1793), (4097, 129), (130, 4100), (2048, 2048)])


@pytest.mark.parametrize("t1,t2", [(False, False), (True, True)])
@pytest.mark.parametrize("span", [20, 28, 36, 44, 100])
def test_rows_of_unlike_size(gt, span, t1, t2):
    """Every row of the result as accurate as if it stood alone, whichever operand has the small rows."""
    a, b = randn(1, 2000, 2100), randn(2, 2100, 2200)
    check_addmm(gt, wide_rows(a, 0, span), b, t1, t2)
    check_addmm(gt, a, wide_rows(b, 1, span), t1, t2)
    check_addmm(gt, wide_rows(a, 1, span), b / wide_rows(torch.ones_like(b), 0, span).clamp_min(2.0 ** -span), t1, t2)


@pytest.mark.parametrize("value", [float("inf"), float("nan"), -3.4028234e38, 1e-44])
def test_single_values(gt, value):
    """One such value in an operand spoils nothing but its own row or column of the result."""
    a, b = randn(3, 2000, 2100), randn(4, 2100, 2200)
    a[777, 1234] = value
    keep = torch.arange(2000, device="cuda") != 777
    check_addmm(gt, a, b, rows=keep)
    b[:, 5] = 0
    if abs(value) < 1:
        check_addmm(gt, a, b)
    check_addmm(gt, b.t().contiguous(), a.t().contiguous(), cols=keep)


def test_zeros_and_extreme_scales(gt):
    a, b = randn(5, 2000, 2100), randn(6, 2100, 2200)
    assert torch.all(addmm(gt, torch.zeros_like(a), b, torch.ones(2000, 2200), False, False, 0.0) == 0)
    for e in (-120, -62, -58, 50, 58, 62, 100):
        check_addmm(gt, a * 2.0 ** e, b * 2.0 ** -max(min(e, 60), -100))


# N, C, H, W, K, k, stride, pad; how many products of forward, backward and a second accGradParameters run over FP32 values, and over pairs
CONVS = [
    ((32, 64, 56, 55, 64, 3, 1, 1), [0, 4]),       # pixel pairs
    ((20, 100, 41, 37, 130, 3, 1, 1), [0, 4]),     # channels padded to whole spans
    ((64, 3, 99, 101, 64, 11, 4, 2), [4, 0]),      # cells, too small for pairs
    ((64, 3, 224, 224, 64, 11, 4, 2), [0, 4]),     # cells, rows staged in shared memory
    ((21, 4, 211, 1903, 64, 11, 4, 2), [0, 4]),    # cells of rows that shared memory does not hold
    ((64, 12, 131, 133, 64, 8, 4, 2), [0, 4]),     # cells whose chunks do not divide a block
    ((24, 64, 31, 33, 192, 5, 1, 2), [0, 4]),
    ((24, 128, 29, 29, 256, 3, 2, 1), [4, 0]),     # strided windows, folded gradInput
    ((96, 128, 29, 29, 256, 3, 2, 1), [0, 4]),
    ((4, 3, 500, 1000, 8, 11, 1, 5), [0, 4]),      # gradInput as a layer of its own
    ((14, 3001, 28, 29, 1024, 1, 1, 0), [0, 4]),   # kept planes of two pixels a block, brought back next to the transposition of gradOutput
    ((6, 7001, 28, 29, 1024, 1, 1, 0), [0, 4]),    # of more channels than that takes
]


@pytest.mark.parametrize("wide", ["", "input", "weight", "gradOutput", "inf"])
@pytest.mark.parametrize("case", CONVS)
def test_convolution(gt, case, wide):
    (N, C, H, W, K, k, stride, pad), expected = case
    x, w, b = randn(1, N, C, H, W), randn(2, K, C, k, k) / (C * k * k) ** 0.5, randn(3, K)
    go = randn(4, N, K, (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1)
    x, w, go = (wide_rows(t, 0, 45) if wide == name else t for t, name in ((x, "input"), (w, "weight"), (go, "gradOutput")))
    if wide == "inf":
        x[1, C - 1, 3, 3] = float("inf")
    live = torch.arange(N, device="cuda") != 1 if wide == "inf" else slice(None)
    m = gt.nn.SpatialConvolutionMM(C, K, k, k, stride, stride, pad)
    m.weight, m.bias = w.reshape(K, -1).cpu().numpy(), b.cpu().numpy()
    m.gpu()
    xg, gog = gt.gpu(x.cpu().numpy()), gt.gpu(go.cpu().numpy())
    m.zeroGradParameters()
    before = products(gt)
    out = torch.from_numpy(m.forward(xg).float()).cuda().double()
    gi = torch.from_numpy(m.backward(xg, gog).float()).cuda().double()
    gw = torch.from_numpy(m.gradWeight.float()).cuda().double().view_as(w)
    m.accGradParameters(xg, gog)            # the planes once more, whichever form they are in by now
    twice = torch.from_numpy(m.gradWeight.float()).cuda().double().view_as(w)
    assert [n - b for n, b in zip(products(gt), before)] == expected

    def conv(x, w, b, go):
        x, w = x.double().requires_grad_(), w.double().requires_grad_()
        o = torch.nn.functional.conv2d(x, w, b.double(), stride, pad)
        return (o.detach(),) + torch.autograd.grad(o, (x, w), go.double())
    want, mass = conv(x, w, b, go), conv(x.abs(), w.abs(), b.abs(), go.abs())
    long = 2.0 ** -24 * (go.numel() / K / 32 + 64)                                 # one rounding per k tile of the pixel sum
    assert torch.all((out - want[0])[live].abs() <= REL * mass[0][live])
    assert torch.all((gi - want[1]).abs() <= REL * mass[1])
    if wide != "inf":
        assert torch.all((gw - want[2]).abs() <= (REL + long) * mass[2])
        assert torch.all((twice - 2 * want[2]).abs() <= 2 * (REL + long) * mass[2])
