"""Values far below the largest of their operand, one by one: products over FP16 pairs hold a result that rests on such a value alone to the
bound of every other.  Reference: torch in float64."""
import pytest
import torch

from test_gpu_fp16_pairs import REL, check_addmm, gt, products, randn  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t1,t2", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("e", [27, 28, 29, 31, 34, 37, 40, 90])
def test_rows_of_one_value(gt, e, t1, t2):  # noqa: F811
    a, b = randn(1, 2000, 2100), randn(2, 2100, 2200)
    for r, c in ((7, 11), (1999, 2099), (1002, 0)):
        a[r] = 0
        a[r, c] = 1.25 * 2.0 ** -e
    check_addmm(gt, a, b, t1, t2, beta=0.0)
    check_addmm(gt, b.t().contiguous(), a.t().contiguous(), t1, t2, beta=0.0)


@pytest.mark.parametrize("e", [30, 37])
def test_diagonals(gt, e):  # noqa: F811
    """Both operands have one, and theirs meet: the product of two small values is a result of its own."""
    a, b = torch.eye(2304, device="cuda"), torch.eye(2304, device="cuda")
    perm = torch.randperm(2304, generator=torch.Generator().manual_seed(1)).cuda()
    for i in (5, 777, 2303):
        a[i, i] = 1.25 * 2.0 ** -e
        b[i, i] = 1.7 * 2.0 ** -e
    check_addmm(gt, a, b)
    check_addmm(gt, a[:, perm].contiguous(), b[perm].contiguous(), beta=1.0)


@pytest.mark.parametrize("n", [0, 1, 23, 24, 25, 3000])
def test_many(gt, n):  # noqa: F811
    """More of them than are listed, 24 of this operand's, send the product to FP32 values."""
    a, b = randn(3, 2000, 2100), randn(4, 2100, 2200)
    at = torch.randperm(a.numel(), generator=torch.Generator().manual_seed(n))[:n].cuda()
    a.view(-1)[at] = 2.0 ** -(30 + torch.arange(n, device="cuda") % 20).float()
    rows = torch.arange(0, 2000, 5, device="cuda")
    keep = torch.zeros_like(a)
    keep.view(-1)[at] = 1
    a[rows] *= keep[rows]                     # rows of nothing else
    check_addmm(gt, a, b)


CONVS = [
    (32, 64, 56, 55, 64, 3, 1, 1),       # pixel pairs
    (96, 128, 29, 29, 256, 3, 2, 1),     # strided windows, folded gradInput
    (64, 3, 224, 224, 64, 11, 4, 2),     # cells
    (64, 12, 131, 133, 64, 8, 4, 2),
    (4096, 600, 2, 2, 640, 1, 1, 0),     # planes of a few pixels
    (4, 3, 500, 1000, 8, 11, 1, 5),      # gradInput as a layer of its own
]


def conv64(x, w, go, stride, pad):
    x, w = x.double().requires_grad_(), w.double().requires_grad_()
    o = torch.nn.functional.conv2d(x, w, None, stride, pad)
    return (o.detach(),) + torch.autograd.grad(o, (x, w), go.double())


@pytest.mark.parametrize("e", [30, 36])
@pytest.mark.parametrize("which", ["input", "weight", "gradOutput", "all"])
@pytest.mark.parametrize("case", CONVS)
def test_convolution(gt, case, which, e):  # noqa: F811
    """Single small values in an image, a filter and a plane of gradOutput that are zero otherwise."""
    N, C, H, W, K, k, stride, pad = case
    oH, oW = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    x, w, go = randn(1, N, C, H, W), randn(2, K, C, k, k) / (C * k * k) ** 0.5, randn(4, N, K, oH, oW)
    small = 1.25 * 2.0 ** -e
    if which in ("input", "all"):
        x[1] = 0                                             # one image, two values
        x[1, C - 1, H // 2, W // 2] = small
        x[1, 0, 0, 0] = -small
        x[:, 1] = 0                                          # one channel: a slice of gradWeight rests on two values of the batch
        x[2, 1, H - 1, W - 1] = small
        x[N - 1, 1, H // 2, W // 2] = 3 * small
    if which in ("weight", "all"):
        w[3] = 0                                             # one filter
        w[3, C - 1, k // 2, k // 2] = small / (C * k * k) ** 0.5
        w[:, 0] = 0                                          # one input plane
        w[K - 1, 0, k - 1, 0] = small / (C * k * k) ** 0.5
    if which in ("gradOutput", "all"):
        go[3] = 0
        go[3, K - 1, oH // 2, oW // 2] = small
        go[:, 2] = 0
        go[N - 2, 2, 0, oW - 1] = -small
    m = gt.nn.SpatialConvolutionMM(C, K, k, k, stride, stride, pad)
    m.weight.reshape(-1)[:] = w.cpu().numpy().reshape(-1)
    m.bias[:] = 0
    m.gpu()
    xg, gog = gt.gpu(x.cpu().numpy()), gt.gpu(go.cpu().numpy())
    m.zeroGradParameters()
    before = products(gt)
    out = torch.from_numpy(m.forward(xg).float()).cuda().double()
    gi = torch.from_numpy(m.backward(xg, gog).float()).cuda().double()
    gw = torch.from_numpy(m.gradWeight.float()).cuda().double().view_as(w)
    assert [n - b for n, b in zip(products(gt), before)] == [0, 3]
    want, mass = conv64(x, w, go, stride, pad), conv64(x.abs(), w.abs(), go.abs(), stride, pad)
    long = 2.0 ** -24 * (go.numel() / K / 32 + 64)                                 # one rounding per k tile of the pixel sum
    assert torch.all((out - want[0]).abs() <= REL * mass[0])
    assert torch.all((gi - want[1]).abs() <= REL * mass[1])
    assert torch.all((gw - want[2]).abs() <= (REL + long) * mass[2])


def test_input_written_over(gt):  # noqa: F811
    """accGradParameters takes the planes of the forward pass, whatever the input's memory holds by then, also where gradOutput sends the
    product to FP32 values."""
    from test_gpu_fp16_pairs import wide_rows
    N, C, H, W, K, k, stride, pad = 32, 64, 56, 55, 64, 3, 1, 1
    x, w, go = randn(1, N, C, H, W), randn(2, K, C, k, k), randn(4, N, K, H, W)
    x[:, 5] = 0
    x[1, 5, 7, 9] = 2.0 ** -33                # a value that the pairs do not hold
    m = gt.nn.SpatialConvolutionMM(C, K, k, k, stride, stride, pad)
    m.weight.reshape(-1)[:] = w.cpu().numpy().reshape(-1)
    m.gpu()
    xg = gt.gpu(x.cpu().numpy())
    m.forward(xg)
    xg.zero()
    for g in (go, wide_rows(go, 0, 45), go):
        m.zeroGradParameters()
        m.accGradParameters(xg, gt.gpu(g.cpu().numpy()))
        gw = torch.from_numpy(m.gradWeight.float()).cuda().double().view_as(w)
        want, mass = conv64(x, w, g, stride, pad)[2], conv64(x.abs(), w.abs(), g.abs(), stride, pad)[2]
        long = 2.0 ** -24 * (g.numel() / K / 32 + 64)
        assert torch.all((gw - want).abs() <= (REL + long) * mass)


def test_repeats_exactly(gt):  # noqa: F811
    a, b = randn(3, 2000, 2100), randn(4, 2100, 2200)
    at = torch.randperm(a.numel(), generator=torch.Generator().manual_seed(1))[:24].cuda()
    a.view(-1)[at] = 1.1 * 2.0 ** -31
    A, B = gt.gpu(a.cpu().numpy()), gt.gpu(b.cpu().numpy())
    r = [gt.GPUTensor(2000, 2200).addmm(0.0, 1.0, A, B).float() for _ in range(3)]
    assert (r[0] == r[1]).all() and (r[0] == r[2]).all()
