"""The forms in which the tensor-core convolution passes state a layer: planes padded to whole swizzle spans, folded and unfolded
cells, the column matrix with stacked weight-gradient pixels, pixel pairs; both precisions, at remainders and smallest sizes."""
import numpy as np
import pytest

from util import conv_exact, conv_grad_input_exact, conv_grad_weight_exact

pytestmark = pytest.mark.gpu

CASES = [
    # N, C, H, W, K, kH, kW, dH, dW, pad
    (2, 3, 20, 18, 64, 3, 3, 1, 1, 1),     # column matrix, four pixels stacked in the weight gradient
    (1, 3, 19, 17, 64, 3, 3, 1, 1, 1),     # odd pixel count: not stacked
    (3, 1, 11, 13, 40, 5, 5, 1, 1, 2),     # one plane
    (6, 17, 25, 17, 29, 5, 5, 1, 1, 1),    # nothing a multiple of anything
    (2, 35, 14, 15, 18, 11, 11, 1, 1, 5),
    (2, 33, 9, 9, 65, 3, 3, 1, 1, 1),      # one plane more than a span (FP32; BF16 in the next)
    (2, 65, 9, 9, 129, 3, 3, 1, 1, 1),
    (3, 6, 21, 23, 50, 5, 5, 2, 2, 1),     # strided, ragged
    (2, 40, 16, 17, 48, 7, 7, 4, 4, 2),
    (2, 64, 15, 13, 64, 3, 3, 2, 2, 1),    # strided with whole spans: direct windows, folded gradInput
    (2, 64, 16, 16, 64, 1, 1, 2, 2, 0),    # window smaller than the stride: pixels that no window reaches
    (1, 5, 17, 19, 33, 3, 2, 4, 3, 0),
    (2, 8, 6, 5, 40, 2, 3, 1, 1, 3),       # padding not below the window
    (1, 2, 4, 4, 1, 4, 4, 1, 1, 0),        # one output
    (150, 3, 6, 6, 16, 3, 3, 1, 1, 0),
    (2, 32, 32, 48, 40, 16, 16, 16, 16, 0),   # cells of more channels than the table holds
    (1, 44, 37, 29, 140, 14, 13, 13, 12, 2),  # the same, ragged
    (2, 60, 40, 37, 2, 13, 13, 1, 1, 6),      # few output planes: gradInput as a layer over gradOutput
    (3, 33, 31, 30, 1, 9, 9, 1, 1, 0),
    (2, 70, 28, 33, 9, 7, 7, 1, 1, 6),
    (1, 7, 135, 140, 34, 131, 133, 1, 1, 0),  # a window beyond what a window map takes: columns
    (7, 5, 6, 5, 40, 3, 3, 2, 2, 1),          # gradInput from cells: groups of 34 planes, the last of one
    (1, 2, 3, 5000, 33, 2, 4, 2, 4, 0),       # and a plane shared by several blocks
]


@pytest.mark.parametrize("mode", ["fp32x3", "bf16"])
@pytest.mark.parametrize("case", CASES)
def test_conv_forms(mode, case):
    import mcw_cppamp_torch_b200 as gt
    N, C, H, W, K, kH, kW, dH, dW, pad = case
    geo = (kH, kW, dH, dW, pad)
    g = np.random.default_rng(sum(case))
    x = g.uniform(-1, 1, (N, C, H, W)).astype(np.float32)
    s = 1.0 / np.sqrt(C * kH * kW)
    w, b = g.uniform(-s, s, (K, C * kH * kW)).astype(np.float32), g.uniform(-s, s, K).astype(np.float32)
    want = conv_exact(x, w, b, *geo)
    go = g.standard_normal(want.shape).astype(np.float32)
    gw0, gb0 = g.standard_normal(w.shape).astype(np.float32), g.standard_normal(K).astype(np.float32)
    gt.set_math_mode(mode)
    try:
        m = gt.nn.SpatialConvolutionMM(C, K, kW, kH, dW, dH, pad)
        m.weight, m.bias, m.gradWeight, m.gradBias = w.copy(), b.copy(), gw0.copy(), gb0.copy()
        m.gpu()
        xg, gog = gt.gpu(x), gt.gpu(go)
        out = m.forward(xg).float()
        gi = m.backward(xg, gog, 0.5).float()
        gw, gb = m.gradWeight.float(), m.gradBias.float()
        apart = gt.nn.SpatialConvolutionMM(C, K, kW, kH, dW, dH, pad)          # no forward pass, separate calls
        apart.weight, apart.bias, apart.gradWeight, apart.gradBias = w.copy(), b.copy(), gw0.copy(), gb0.copy()
        apart.gpu()
        assert np.array_equal(apart.updateGradInput(xg, gog).float(), gi)
        apart.accGradParameters(xg, gog, 0.5)
        assert np.array_equal(apart.gradWeight.float(), gw) and np.array_equal(apart.gradBias.float(), gb)
    finally:
        gt.set_math_mode("fp32x3")
    a = np.abs
    # 3xTF32: dropped terms and truncating chains are 2^-19 of the sum of |products|; BF16 operands: 2^-8 per product
    rel = 2.0 ** -19 if mode == "fp32x3" else 2.0 ** -7
    gw_e, gb_e = conv_grad_weight_exact(x, go, *geo)
    gw_s, gb_s = conv_grad_weight_exact(a(x), a(go), *geo)
    long = 2.0 ** -24 * (go.size / K / 32 + 64)                                    # one rounding per k tile of the pixel sum
    assert np.all(a(out - want) <= rel * conv_exact(a(x), a(w), a(b), *geo) + 1e-30)
    assert np.all(a(gi - conv_grad_input_exact(go, w, x.shape, *geo)) <= rel * conv_grad_input_exact(a(go), a(w), x.shape, *geo) + 1e-30)
    assert np.all(a(gw - (gw0 + 0.5 * gw_e)) <= (rel + long) * (gw_s + a(gw0)))
    assert np.all(a(gb - (gb0 + 0.5 * gb_e)) <= (2.0 ** -19 + long) * (gb_s + a(gb0)))


@pytest.mark.parametrize("C", [3, 32])
def test_planes_of_a_finput_put_to_another_use_are_not_taken(C):
    """`finput` resized (its memory stays where it is) and written to between the forward pass and accGradParameters."""
    import mcw_cppamp_torch_b200 as gt
    g = np.random.default_rng(C)
    m = gt.nn.SpatialConvolutionMM(C, 40, 3, 3, 1, 1, 1).gpu()
    x, go = (gt.gpu(g.standard_normal((4, c, 16, 16)).astype(np.float32)) for c in (C, 40))

    def weight_gradient(touch):
        m.gradWeight.zero(); m.gradBias.zero()
        m.forward(x)
        if touch:
            at = m.finput.data_ptr()
            m.finput.resize(100, 7).fill(3)
            assert m.finput.data_ptr() == at
        m.accGradParameters(x, go)
        return m.gradWeight.float()
    assert np.array_equal(weight_gradient(False), weight_gradient(True))


def test_planes_no_weight_gradient_reads_are_not_kept():
    """BF16 mode: the first layer's column matrix is not its FP32-accurate weight gradient's input; a wide layer's planes are."""
    import mcw_cppamp_torch_b200 as gt
    gt.set_math_mode("bf16")
    try:
        first, wide = gt.nn.SpatialConvolutionMM(3, 64, 11, 11, 4, 4, 2).gpu(), gt.nn.SpatialConvolutionMM(64, 192, 5, 5, 1, 1, 2).gpu()
        first.forward(gt.gpu(np.ones((4, 3, 63, 63), np.float32)))
        wide.forward(gt.gpu(np.ones((4, 64, 27, 27), np.float32)))
        assert first.finput.dim() == 0 and wide.finput.size() == (1, 4, 27, 27, 32)
    finally:
        gt.set_math_mode("fp32x3")


def test_bf16_columns_in_groups_of_images():
    """400 images of the 11 x 11 / 4 layer are 2.5 GB of columns: two groups.  Each image's result is its own, bit for bit."""
    import mcw_cppamp_torch_b200 as gt
    x = np.random.default_rng(1).standard_normal((400, 3, 224, 224), dtype=np.float32)
    gt.set_math_mode("bf16")
    try:
        m = gt.nn.SpatialConvolutionMM(3, 64, 11, 11, 4, 4, 2).gpu()
        out = m.forward(gt.gpu(x))
        for n in (1, 198, 201, 397):
            assert np.array_equal(out.narrow(1, n, 4).float(), m.clone().forward(gt.gpu(x[n - 1:n + 3])).float())
    finally:
        gt.set_math_mode("fp32x3")


@pytest.mark.parametrize("stride", [1, 2])
def test_planes_that_would_outgrow_the_batch_many_times(stride):
    """125 images of one 1024 x 1024 plane: 0.5 GB, 17 GB as padded planes, which are made in groups and not kept.  Whole numbers,
    whose sums are exact in any order, against the FP32 FMA engine."""
    import mcw_cppamp_torch_b200 as gt
    g = np.random.default_rng(stride)
    N, K, side = 125, 2, 1024
    x = g.integers(-1, 2, (N, 1, side, side), np.int8).astype(np.float32)
    go = g.integers(-1, 2, (N, K, (side - 1) // stride + 1, (side - 1) // stride + 1), np.int8).astype(np.float32)
    got = {}
    try:
        for mode in ("fp32x3", "simt"):
            gt.set_math_mode(mode)
            m = gt.nn.SpatialConvolutionMM(1, K, 3, 3, stride, stride, 1)
            m.weight = g.integers(-2, 3, m.weight.shape).astype(np.float32) if not got else got["weight"]
            m.bias = np.zeros_like(m.bias)
            got["weight"] = m.weight
            m.gpu()
            X = gt.gpu(x)
            out = m.forward(X)
            m.gradWeight.zero(); m.gradBias.zero()
            gi = m.backward(X, gt.gpu(go))
            assert stride > 1 or m.finput.dim() == 0
            now = [out.float(), gi.float(), m.gradWeight.float(), m.gradBias.float()]
            if mode == "simt":
                assert all(np.array_equal(a, b) for a, b in zip(got["planes"], now))
            got["planes"] = now
            del m, X, out, gi
    finally:
        gt.set_math_mode("fp32x3")


def test_grad_input_of_few_output_planes_does_not_pay_for_padding():
    """9 x 9 taps, 32 <- K planes, 46 of 87 x 88: 516 us for 32 planes and as much for two padded to 32; 121 as a layer over two."""
    import torch
    import mcw_cppamp_torch_b200 as gt
    stream = torch.cuda.ExternalStream(gt.lib().THGPUGetStream())

    def us(K):
        m = gt.nn.SpatialConvolutionMM(32, K, 9, 9, 1, 1, 4).gpu()
        x, go, times = gt.GPUTensor(46, 32, 87, 88).fill(1), gt.GPUTensor(46, K, 87, 88).fill(1), []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            m.updateGradInput(x, go)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return sorted(times[2:])[2]
    assert us(2) < us(32) / 2


@pytest.mark.parametrize("case", [(70, 3, 224, 224, 64, 11, 11, 4, 4, 2), (3, 8, 130, 97, 33, 3, 3, 1, 1, 1), (9, 1, 40, 61, 64, 1, 1, 1, 1, 0), (40, 2, 33, 47, 48, 8, 8, 2, 3, 3),
                                  (5, 7, 64, 64, 64, 1, 17, 1, 1, 0), (6, 4, 60, 52, 50, 20, 2, 1, 1, 0), (300, 3, 32, 32, 64, 5, 5, 1, 1, 2), (20, 5, 12, 13, 40, 2, 2, 5, 6, 1)])   # (the mode leaves layers of up to 128 windows in FP32)
def test_bf16_gathered_windows(case):
    """First layers in BF16, whose taps the engine copies to shared memory itself: taps that fill no k tile, filter rows longer and shorter than one,
    windows apart and overlapping, last tiles in part.  Products of BF16 values are exact in FP32; K sums, each rounded or truncated once."""
    import torch
    import mcw_cppamp_torch_b200 as gt
    N, C, H, W, K, kH, kW, dH, dW, pad = case
    g = torch.Generator().manual_seed(sum(case))
    x, w, b = torch.randn(N, C, H, W, generator=g), torch.randn(K, C, kH, kW, generator=g), torch.randn(K, generator=g)
    gt.set_math_mode("bf16")
    try:
        m = gt.nn.SpatialConvolutionMM(C, K, kW, kH, dW, dH, pad)
        m.weight, m.bias = w.reshape(K, -1).numpy().copy(), b.numpy().copy()
        m.gpu()
        out = torch.from_numpy(m.forward(gt.gpu(x.numpy())).float()).cuda()
        assert m.finput.dim() == 0
    finally:
        gt.set_math_mode("fp32x3")

    def conv(f):
        q = lambda t: f(t.bfloat16().double()).cuda()
        return torch.nn.functional.conv2d(q(x), q(w), f(b.double()).cuda(), (dH, dW), pad)
    assert torch.all((out - conv(lambda t: t)).abs() <= (C * kH * kW + 2) * 2.0 ** -23 * conv(torch.abs))


def test_grad_input_from_cells_by_pixels():
    """Four rows of 262144 pixels take what 1024 rows of 1024 do; a lane or a block per row leaves the device idle."""
    import torch
    import mcw_cppamp_torch_b200 as gt

    def us(H, W):
        m = gt.nn.SpatialConvolutionMM(1, 33, 4, 4, 4, 4)
        m.gpu()
        x, go = gt.GPUTensor(1, 1, H, W), gt.GPUTensor(1, 33, H // 4, W // 4).fill(0.5)
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        times = []
        for _ in range(8):
            gt.synchronize()
            a.record()
            m.updateGradInput(x, go)
            gt.synchronize()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return sorted(times[2:])[2]
    assert us(4, 262144) < 4 * us(1024, 1024)


@pytest.mark.parametrize("mode,shape", [("bf16", (4, 64, 20, 18)), ("fp32x3", (4, 64, 20, 18)), ("fp32x3", (64, 512, 13, 13))])
def test_grad_bias_of_4096_planes(mode, shape):
    """Their sums come along with gradOutput's planes, as those of fewer planes do: as many launches."""
    import mcw_cppamp_torch_b200 as gt
    N, C, H, W = shape
    g = np.random.default_rng(7)
    x = gt.gpu(g.standard_normal(shape, dtype=np.float32))
    gt.set_math_mode(mode)
    try:
        counts = []
        for K in (3968, 4096):
            m = gt.nn.SpatialConvolutionMM(C, K, 1, 1).gpu()
            go = g.standard_normal((N, K, H, W), dtype=np.float32)
            gg = gt.gpu(go)
            m.zeroGradParameters()
            n = gt.lib().THGPUKernelLaunchCount()
            m.accGradParameters(x, gg)
            counts.append(gt.lib().THGPUKernelLaunchCount() - n)
            go = go.astype(np.float64)
            # (partial sums of at most 16 pixels a lane, then trees and rows of blocks: far fewer roundings in turn than values)
            assert np.all(np.abs(m.gradBias.float() - go.sum((0, 2, 3))) <= N * H * W * 2.0 ** -24 * np.abs(go).sum((0, 2, 3)))
        assert counts[0] == counts[1]
    finally:
        gt.set_math_mode("fp32x3")


@pytest.mark.parametrize("case", [(300, 3, 64, 64, 64, 11, 11, 4, 4, 2), (40, 2, 33, 47, 48, 8, 8, 2, 3, 3), (9, 1, 40, 61, 64, 1, 1, 1, 1, 0), (5, 7, 64, 64, 64, 1, 17, 1, 1, 0)])
def test_bf16_gathered_windows_and_columns_agree(case):
    """The same bits as over the column matrix, which a layer of 128 planes takes: its first planes have this layer's filters."""
    import mcw_cppamp_torch_b200 as gt
    N, C, H, W, K, kH, kW, dH, dW, pad = case
    g = np.random.default_rng(sum(case))
    x, w, b = (g.standard_normal(s, dtype=np.float32) for s in ((N, C, H, W), (128, C * kH * kW), (128,)))
    xg, out = gt.gpu(x), []
    gt.set_math_mode("bf16")
    try:
        for planes in (K, 128):
            m = gt.nn.SpatialConvolutionMM(C, planes, kW, kH, dW, dH, pad)
            m.weight, m.bias = w[:planes].copy(), b[:planes].copy()
            out.append(m.gpu().forward(xg).float()[:, :K])
    finally:
        gt.set_math_mode("fp32x3")
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
