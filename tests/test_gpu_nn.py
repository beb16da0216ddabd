"""gpunn operators on the device vs the CPU oracle: SpatialConvolutionMM (all three passes, stride,
padding, 3-D inputs), SpatialMaxPooling (values and bit-exact indices, overlapping windows),
Threshold, LogSoftMax, ClassNLLCriterion, SGD; the reference's own golden vectors; and the
single-conv-block configuration at full size."""
import os

import numpy as np
import pytest

from util import close, close_accumulated, close_scaled, conv_exact, conv_grad_input_exact, conv_grad_weight_exact

pytestmark = pytest.mark.gpu
G = np.load(os.path.join(os.path.dirname(__file__), "golden", "reference_cpu.npz"))
MODES = ["fp32x3", "simt"]


@pytest.fixture(scope="module")
def gt():
    import mcw_cppamp_torch_b200 as m
    m.lib().THGPUInit()
    yield m
    m.set_math_mode("fp32x3")


def run_conv(gt, x, w, b, go, k, d, pad, scale=1.0, gw0=None, gb0=None):
    K = w.shape[0]
    C = x.shape[-3]
    m = gt.nn.SpatialConvolutionMM(C, K, k[1], k[0], d[1], d[0], pad)
    m.weight, m.bias = w.copy(), b.copy()
    m.gradWeight = np.zeros_like(w) if gw0 is None else gw0.copy()
    m.gradBias = np.zeros_like(b) if gb0 is None else gb0.copy()
    m.gpu()
    xg = gt.gpu(x)
    out = m.forward(xg).float()
    gi = gw = gb = None
    if go is not None:
        gi = m.backward(xg, gt.gpu(go), scale).float()
        gw, gb = m.gradWeight.float(), m.gradBias.float()
    return out, gi, gw, gb


CONV_CASES = [
    # N, C, H, W, K, kH, kW, dH, dW, pad
    (2, 3, 12, 11, 8, 3, 3, 1, 1, 0),
    (3, 5, 9, 9, 16, 5, 5, 1, 1, 2),
    (2, 3, 23, 23, 8, 11, 11, 4, 4, 2),      # the first AlexNet-style layer, small image
    (2, 4, 12, 15, 6, 3, 3, 2, 2, 1),
    (1, 2, 9, 10, 4, 5, 3, 3, 2, 0),         # non-square kernel and stride
    (2, 16, 13, 13, 24, 3, 3, 1, 1, 1),
    (1, 1, 6, 6, 3, 1, 1, 1, 1, 0),
    (5, 7, 17, 17, 70, 3, 3, 1, 1, 1),       # K_out > 64: wide tile
    (2, 40, 10, 10, 130, 3, 3, 1, 1, 1),     # two N tiles, ragged
    (1, 3, 8, 8, 5, 8, 8, 1, 1, 0),          # kernel covers the image: 1x1 output
    # channel counts that are multiples of 32: the channels-last hi/lo plane passes
    (2, 32, 9, 9, 32, 3, 3, 1, 1, 1),
    (3, 64, 13, 13, 96, 3, 3, 1, 1, 1),
    (2, 64, 14, 11, 192, 5, 5, 1, 1, 2),     # non-square image, two ragged tiles of output planes
    (2, 32, 12, 15, 64, 3, 3, 2, 2, 1),      # strided: planes forward / gradWeight, gathered gradInput
    (1, 96, 7, 7, 160, 3, 5, 1, 1, 0),       # kH != kW, a gradWeight tile that straddles two taps
    (2, 160, 6, 6, 32, 1, 1, 1, 1, 0),       # 1x1 filter
    (4, 32, 10, 10, 32, 3, 3, 1, 1, 2),      # padding = k - 1
    (37, 32, 5, 6, 64, 3, 3, 1, 1, 1),       # pixel count not a multiple of the 32-pixel reduction tile
    # layer shapes of the VGG-A-style configuration (3x3, pad 1) on reduced images
    (1, 3, 32, 32, 64, 3, 3, 1, 1, 1),
    (2, 64, 28, 28, 128, 3, 3, 1, 1, 1),
    (1, 256, 14, 14, 512, 3, 3, 1, 1, 1),
    (3, 64, 27, 27, 192, 5, 5, 1, 1, 2),     # second AlexNet-style layer, full image size
    # strided layers with few input planes: restated as stride-1 layers over folded stride cells
    (3, 3, 47, 51, 64, 11, 11, 4, 4, 2),     # 4 x 4 cells of 3 (+1) planes -> 64 channels, ragged image
    (4, 3, 35, 35, 64, 7, 7, 4, 4, 3),       # filter not a multiple of the stride, padding 3
    (4, 6, 20, 22, 96, 5, 5, 2, 2, 2),       # 2 x 2 cells of 6 (+2) planes -> 32 channels, no pixel pairs
    (5, 3, 40, 38, 64, 11, 10, 4, 4, 0),     # kH != kW, no padding
]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("case", CONV_CASES)
def test_conv_all_passes(gt, oracle_port, mode, case):
    gt.set_math_mode(mode)
    N, C, H, W, K, kH, kW, dH, dW, pad = case
    g = oracle_port.rng(sum(case))
    x = g.uniform((N, C, H, W), -1, 1)
    s = 1.0 / np.sqrt(C * kH * kW)
    w, b = g.uniform((K, C * kH * kW), -s, s), g.uniform((K,), -s, s)
    want = oracle_port.conv_forward(x, w, b, kH, kW, dH, dW, pad)
    go = g.normal(want.shape)
    gw0, gb0 = g.normal(w.shape), g.normal(b.shape)            # accGradParameters accumulates
    out, gi, gw, gb = run_conv(gt, x, w, b, go, (kH, kW), (dH, dW), pad, 0.5, gw0, gb0)
    geo = (kH, kW, dH, dW, pad)
    close_accumulated(out, want, conv_exact(x, w, b, *geo), what="conv output")
    close_accumulated(gi, oracle_port.conv_grad_input(go, w, x.shape, *geo), conv_grad_input_exact(go, w, x.shape, *geo),
                      what="conv gradInput")
    gw_o, gb_o = gw0.copy(), gb0.copy()
    oracle_port.conv_acc_grad(x, go, gw_o, gb_o, 0.5, *geo)
    gw_e, gb_e = conv_grad_weight_exact(x, go, *geo)
    close_accumulated(gw, gw_o, gw0 + 0.5 * gw_e, what="conv gradWeight")
    close_accumulated(gb, gb_o, gb0 + 0.5 * gb_e, what="conv gradBias")


@pytest.mark.parametrize("mode", MODES)
def test_conv_3d_input_and_errors(gt, oracle_port, mode):
    gt.set_math_mode(mode)
    g = oracle_port.rng(9)
    x = g.uniform((3, 10, 12), -1, 1)
    w, b = g.uniform((6, 27), -0.2, 0.2), g.uniform((6,), -0.2, 0.2)
    want = oracle_port.conv_forward(x[None], w, b, 3, 3, 1, 1, 1)[0]
    go = g.normal(want.shape)
    out, gi, gw, gb = run_conv(gt, x, w, b, go, (3, 3), (1, 1), 1)
    assert out.shape == want.shape and gi.shape == x.shape
    close(out, want)
    close(gi, oracle_port.conv_grad_input(go[None], w, (1,) + x.shape, 3, 3, 1, 1, 1)[0])
    m = gt.nn.SpatialConvolutionMM(4, 6, 3, 3).gpu()
    with pytest.raises(gt.THCError, match="input channels"):
        m.forward(gt.gpu(x[None]))
    with pytest.raises(gt.THCError, match="3D or 4D"):
        m.forward(gt.GPUTensor(4, 4))
    with pytest.raises(gt.THCError, match="smaller than kernel"):
        m.forward(gt.GPUTensor(1, 4, 2, 2))


@pytest.mark.parametrize("mode", MODES)
def test_conv_golden_vectors(gt, mode):
    gt.set_math_mode(mode)
    N, C, H, W, K, k, d, pad = G["s1_cfg"]
    out, gi, gw, gb = run_conv(gt, G["s1_x"], G["s1_w"], G["s1_b"], G["s1_g_conv"], (k, k), (d, d), pad)
    close(out, G["s1_conv"]); close(gi, G["s1_gi"]); close(gw, G["s1_gw"]); close(gb, G["s1_gb"])
    N, C, H, W, K, k, d, pad = G["s4_cfg"]
    out, gi, gw, gb = run_conv(gt, G["s4_x"], G["s4_w"], G["s4_b"], G["s4_go"], (k, k), (d, d), pad)
    close(out, G["s4_conv"]); close(gi, G["s4_gi"]); close(gw, G["s4_gw"]); close(gb, G["s4_gb"])


@pytest.mark.parametrize("case", [(3, 32, 9, 9, 64, 3, 3, 1, 1, 1),        # raw-operand layer: finput = one FP32 plane
                                  (2, 5, 9, 9, 16, 3, 3, 1, 1, 1),         # hi / lo planes in finput
                                  (3, 3, 47, 51, 64, 11, 11, 4, 4, 2)])    # folded input in finput
def test_acc_grad_parameters_uses_the_input_it_is_given(gt, oracle_port, case):
    """forward(A) leaves A's planes in finput; accGradParameters(B) on another input of the same shape must
    compute with B (the reference GPU path rebuilds its columns from `input`,
    gputorch/lib/THC/gpunn-impl/SpatialConvolutionMM.cpp:313-429), and so must an accGradParameters after a
    forward pass in another math mode, which does not write finput at all."""
    gt.set_math_mode("fp32x3")
    N, C, H, W, K, kH, kW, dH, dW, pad = case
    g = oracle_port.rng(7 + sum(case))
    A, B = g.uniform((N, C, H, W), -1, 1), g.uniform((N, C, H, W), -1, 1)
    s = 1.0 / np.sqrt(C * kH * kW)
    w, b = g.uniform((K, C * kH * kW), -s, s), g.uniform((K,), -s, s)
    m = gt.nn.SpatialConvolutionMM(C, K, kW, kH, dW, dH, pad)
    m.weight, m.bias = w.copy(), b.copy()
    m.gpu()
    geo = (kH, kW, dH, dW, pad)
    a_gpu, b_gpu = gt.gpu(A), gt.gpu(B)
    go = g.normal(m.forward(a_gpu).size())

    def check(x_np, what):
        gw_o, gb_o = np.zeros_like(w), np.zeros_like(b)
        oracle_port.conv_acc_grad(x_np, go, gw_o, gb_o, 1.0, *geo)
        gw_e, gb_e = conv_grad_weight_exact(x_np, go, *geo)
        close_accumulated(m.gradWeight.float(), gw_o, gw_e, what=what)
        close_accumulated(m.gradBias.float(), gb_o, gb_e, what=what + " (bias)")

    m.zeroGradParameters()
    m.accGradParameters(b_gpu, gt.gpu(go))
    check(B, "gradWeight of B after forward(A)")
    m.zeroGradParameters()
    m.accGradParameters(a_gpu, gt.gpu(go))               # and the planes of A are still good for A
    check(A, "gradWeight of A after forward(A)")
    gt.set_math_mode("simt")
    m.forward(b_gpu)                                     # writes no planes
    gt.set_math_mode("fp32x3")
    m.zeroGradParameters()
    m.accGradParameters(b_gpu, gt.gpu(go))
    check(B, "gradWeight of B after a forward pass in another math mode")


def test_conv_is_deterministic(gt, oracle_port):
    gt.set_math_mode("fp32x3")
    g = oracle_port.rng(2)
    x, w, b = g.uniform((4, 8, 20, 20), -1, 1), g.uniform((32, 72), -0.1, 0.1), g.uniform((32,), -0.1, 0.1)
    go = g.normal((4, 32, 20, 20))
    r1 = run_conv(gt, x, w, b, go, (3, 3), (1, 1), 1)
    r2 = run_conv(gt, x, w, b, go, (3, 3), (1, 1), 1)
    for a, c in zip(r1, r2):
        assert np.array_equal(a, c)


def test_conv_backward_entry_and_finput(gt, oracle_port):
    """backward() (one library call) gives what updateGradInput + accGradParameters give; accGradParameters reads
    the planes the forward pass left in finput, and rebuilds them when finput does not fit the input."""
    gt.set_math_mode("fp32x3")
    g = oracle_port.rng(77)
    N, C, H, W, K, k, pad = 3, 32, 11, 9, 64, 3, 1
    x = g.uniform((N, C, H, W), -1, 1)
    w, b = g.uniform((K, C * k * k), -0.1, 0.1), g.uniform((K,), -0.1, 0.1)
    go = g.normal((N, K, H, W))

    def fresh():
        m = gt.nn.SpatialConvolutionMM(C, K, k, k, 1, 1, pad)
        m.weight, m.bias = w.copy(), b.copy()
        m.gradWeight, m.gradBias = np.zeros_like(w), np.zeros_like(b)
        return m.gpu()
    xg, gog = gt.gpu(x), gt.gpu(go)
    m1 = fresh(); m1.forward(xg)
    gi1 = m1.backward(xg, gog, 0.5).float()
    m2 = fresh(); m2.forward(xg)
    gi2 = m2.updateGradInput(xg, gog).float()
    m2.accGradParameters(xg, gog, 0.5)
    assert np.array_equal(gi1, gi2)
    assert np.array_equal(m1.gradWeight.float(), m2.gradWeight.float())
    assert np.array_equal(m1.gradBias.float(), m2.gradBias.float())
    # one FP32 plane when the layer runs on the raw-operand engine, TF32 hi / lo planes otherwise
    assert m1.finput.size()[0] in (1, 2) and m1.finput.size()[1:] == (N, H, W, C)
    # no forward pass (finput empty) and a forward pass over another shape: planes are rebuilt from the input
    m3 = fresh()
    m3.accGradParameters(xg, gog, 0.5)
    assert np.array_equal(m3.gradWeight.float(), m2.gradWeight.float())
    m4 = fresh(); m4.forward(gt.gpu(x[:2]))
    m4.accGradParameters(xg, gog, 0.5)
    assert np.array_equal(m4.gradWeight.float(), m2.gradWeight.float())
    # first layer of a network: gradInput switched off
    m5 = fresh(); m5.gradInput = None
    m5.forward(xg)
    assert m5.backward(xg, gog, 0.5) is None
    assert np.array_equal(m5.gradWeight.float(), m2.gradWeight.float())


POOL_CASES = [((2, 3, 9, 11), (3, 3), (2, 2)), ((4, 7, 7), (2, 2), (2, 2)), ((1, 2, 13, 13), (3, 2), (1, 3)),
              ((2, 2, 6, 6), (6, 6), (1, 1)), ((3, 5, 55, 55), (3, 3), (2, 2)), ((2, 4, 28, 28), (2, 2), (2, 2)),
              ((2, 3, 10, 10), (4, 4), (3, 3)), ((1, 1, 5, 5), (1, 1), (1, 1)),
              ((2, 2, 160, 150), (2, 2), (2, 2)), ((1, 3, 170, 131), (3, 3), (2, 2)),   # planes cut into row bands
              ((40, 16, 13, 13), (3, 3), (2, 2))]                                        # several planes per block


@pytest.mark.parametrize("shape,k,d", POOL_CASES)
def test_maxpool_bit_exact(gt, oracle_port, shape, k, d):
    g = oracle_port.rng(shape[-1])
    x = g.normal(shape)
    x.reshape(-1)[::5] = 0.25          # ties: the first maximum in row-major window order must win
    m = gt.nn.SpatialMaxPooling(k[1], k[0], d[1], d[0])
    xg = gt.gpu(x)
    out = m.forward(xg).float()
    want, ind = oracle_port.maxpool_forward(x, k[0], k[1], d[0], d[1])
    got_ind = m.indices.float()
    assert got_ind.shape == ind.shape
    assert np.array_equal(out, want)
    assert np.array_equal(got_ind.view(np.uint32), ind.view(np.uint32))     # identical bit patterns
    go = g.normal(want.shape)
    gi = m.backward(xg, gt.gpu(go)).float()
    assert np.array_equal(gi, oracle_port.maxpool_backward(go, ind, x.shape, d[0], d[1]))


def test_maxpool_golden_and_errors(gt):
    for name, k, d in (("p32", 3, 2), ("p22", 2, 2)):
        x = G[name + "_x"]
        m = gt.nn.SpatialMaxPooling(k, k, d, d)
        xg = gt.gpu(x)
        assert np.array_equal(m.forward(xg).float(), G[name + "_out"])
        assert np.array_equal(m.indices.float(), G[name + "_ind"])
        assert np.array_equal(m.backward(xg, gt.gpu(G[name + "_go"])).float(), G[name + "_gi"])
    with pytest.raises(gt.THCError, match="smaller than kernel"):
        gt.nn.SpatialMaxPooling(3, 3).forward(gt.GPUTensor(1, 2, 2))
    # non-contiguous input goes through newContiguous like the reference
    x = G["p32_x"]
    m = gt.nn.SpatialMaxPooling(3, 3, 2, 2)
    xt = gt.gpu(np.ascontiguousarray(x.transpose(0, 1, 3, 2))).transpose(3, 4)
    assert np.array_equal(m.forward(xt).float(), G["p32_out"])


def test_threshold(gt, oracle_port):
    g = oracle_port.rng(5)
    x, go = g.normal((3, 4, 5, 6)), g.normal((3, 4, 5, 6))
    x.reshape(-1)[::9] = 0.0
    for th, val in ((0.0, 0.0), (0.3, -1.5), (1e-6, 0.0)):
        m = gt.nn.Threshold(th, val)
        xg = gt.gpu(x)
        assert np.array_equal(m.forward(xg).float(), oracle_port.threshold_forward(x, th, val))
        assert np.array_equal(m.backward(xg, gt.gpu(go)).float(), oracle_port.threshold_backward(x, go, th))
    r = gt.nn.ReLU()
    xt = gt.gpu(np.ascontiguousarray(x.reshape(12, 30).T)).t()           # strided input
    assert np.array_equal(r.forward(xt).float(), np.maximum(x.reshape(12, 30), 0))


def test_logsoftmax_classnll_sgd(gt, oracle_port):
    g = oracle_port.rng(31)
    z = g.normal((9, 1000), 0, 2)
    m = gt.nn.LogSoftMax()
    zg = gt.gpu(z)
    out = m.forward(zg).float()
    # The CPU kernel sums a polynomial approximation of exp (mcw_torch7_core/lib/TH/THLogAdd.c:56-86); the
    # device evaluates the same polynomial, so it tracks the CPU result at the usual bound and the
    # mathematically exact log-softmax only to about 5e-3.
    close(out, oracle_port.logsoftmax_forward(z), what="logsoftmax vs CPU")
    z64 = z.astype(np.float64)
    exact = z64 - (z64.max(1, keepdims=True) + np.log(np.exp(z64 - z64.max(1, keepdims=True)).sum(1, keepdims=True)))
    close(out, exact.astype(np.float32), rtol=1e-3, atol=5e-3, what="logsoftmax exact")
    go = g.normal(z.shape)
    close(m.backward(zg, gt.gpu(go)).float(), oracle_port.logsoftmax_backward(go, out), what="logsoftmax bwd")
    target = np.floor(g.uniform((9,), 0, 1000)).astype(np.float32) + 1
    crit = gt.nn.ClassNLLCriterion()
    og, tg = gt.gpu(out), gt.gpu(target)
    loss = crit.forward(og, tg)
    assert abs(loss - oracle_port.classnll_forward(out, target)) <= 1e-5 + 1e-4 * abs(loss)
    assert np.array_equal(crit.backward(og, tg).float(), oracle_port.classnll_backward(target, out.shape))
    # golden logsoftmax
    mg = gt.nn.LogSoftMax()
    lz = gt.gpu(G["l_z"])
    close(mg.forward(lz).float(), G["l_out"])
    close(mg.backward(lz, gt.gpu(G["l_go"])).float(), G["l_gi"])
    # SGD: plain (Module:updateParameters) and with momentum
    w, gr, v = g.normal((1003,)), g.normal((1003,)), g.normal((1003,))
    L = gt.lib()
    wg, gg, vg = gt.gpu(w), gt.gpu(gr), gt.gpu(v)
    L.THGPUNN_SGD_update(wg.cdata, gg.cdata, None, 0.01, 0.0)
    close(wg.float(), w - np.float32(0.01) * gr)
    wg = gt.gpu(w)
    L.THGPUNN_SGD_update(wg.cdata, gg.cdata, vg.cdata, 0.01, 0.9)
    v2 = np.float32(0.9) * v + gr
    close(vg.float(), v2)
    close(wg.float(), w - np.float32(0.01) * v2)


def test_linear_module(gt, oracle_port):
    g = oracle_port.rng(12)
    B, I, O = 16, 300, 70
    lin = gt.nn.Linear(I, O, rng=g)
    w, b = lin.weight.copy(), lin.bias.copy()
    lin.gpu()
    x, go = g.normal((B, I)), g.normal((B, O))
    xg = gt.gpu(x)
    want = oracle_port.addmm(1.0, np.tile(b, (B, 1)).astype(np.float32), 1.0, x, w.T)
    close(lin.forward(xg).float(), want, what="Linear output")
    lin.zeroGradParameters()
    gi = lin.backward(xg, gt.gpu(go)).float()
    close(gi, oracle_port.addmm(0.0, np.zeros((B, I), np.float32), 1.0, go, w), what="Linear gradInput")
    close(lin.gradWeight.float(), oracle_port.addmm(0.0, np.zeros((O, I), np.float32), 1.0, go.T, x), what="Linear gradWeight")
    close(lin.gradBias.float(), go.astype(np.float64).sum(0).astype(np.float32), what="Linear gradBias")


def test_conv_block_full_size(gt, oracle_port):
    """The single-conv-block configuration: batch 16 x 3 x 224 x 224 U[-1,1], conv 3->64 k11 s4 p2 with
    U(+-1/sqrt(363)) parameters (weight drawn first), ReLU, max-pool 3/2, gradOutput N(0,1); output, pool
    indices, gradInput, gradWeight and gradBias against the CPU oracle on the same seeded inputs."""
    gt.set_math_mode("fp32x3")
    g = oracle_port.rng(1234)
    x = g.uniform((16, 3, 224, 224), -1, 1)
    conv = gt.nn.SpatialConvolutionMM(3, 64, 11, 11, 4, 4, 2, rng=g)
    w, b = conv.weight.copy(), conv.bias.copy()
    pool = gt.nn.SpatialMaxPooling(3, 3, 2, 2)
    net = gt.nn.Sequential().add(conv).add(gt.nn.ReLU()).add(pool).gpu()
    go = g.normal((16, 64, 27, 27))
    xg = gt.gpu(x)
    out = net.forward(xg).float()
    net.zeroGradParameters()
    gi = net.backward(xg, gt.gpu(go)).float()
    c = oracle_port.conv_forward(x, w, b, 11, 11, 4, 4, 2)
    r = oracle_port.threshold_forward(c)
    p, ind = oracle_port.maxpool_forward(r, 3, 3, 2, 2)
    close(out, p, what="block output")
    got_ind = pool.indices.float()
    # indices must be bit-identical wherever the pooled window has a unique maximum at fp32 resolution
    # of the conv output; ties created by conv rounding differences are counted, not hidden
    same = got_ind.view(np.uint32) == ind.view(np.uint32)
    assert same.mean() > 0.9999, "pool indices differ in %d of %d places" % ((~same).sum(), same.size)
    g_r = oracle_port.maxpool_backward(go, got_ind, r.shape, 2, 2)
    g_c = oracle_port.threshold_backward(c, g_r)
    close(gi, oracle_port.conv_grad_input(g_c, w, x.shape, 11, 11, 4, 4, 2), what="block gradInput")
    gw, gb = np.zeros_like(w), np.zeros_like(b)
    oracle_port.conv_acc_grad(x, g_c, gw, gb, 1.0, 11, 11, 4, 4, 2)
    gw_e, gb_e = conv_grad_weight_exact(x, g_c, 11, 11, 4, 4, 2)      # sums of 48400 terms
    close_accumulated(conv.gradWeight.float(), gw, gw_e, what="block gradWeight")
    close_accumulated(conv.gradBias.float(), gb, gb_e, what="block gradBias")


def test_get_parameters_flattening(gt, oracle_port):
    g = oracle_port.rng(3)
    net = gt.nn.Sequential().add(gt.nn.SpatialConvolutionMM(2, 4, 3, 3, rng=g)).add(gt.nn.ReLU()) \
        .add(gt.nn.View(4 * 4 * 4)).add(gt.nn.Linear(64, 5, rng=g)).gpu()
    w0 = [m.weight.float().copy() for m in (net.modules[0], net.modules[3])]
    fw, fg = net.getParameters()
    assert fw.nElement() == 4 * 18 + 4 + 5 * 64 + 5
    assert np.array_equal(net.modules[0].weight.float(), w0[0]) and np.array_equal(net.modules[3].weight.float(), w0[1])
    fw.fill(0.5)                              # the modules now view the flat storage
    assert np.all(net.modules[3].bias.float() == 0.5)
    x = gt.gpu(g.normal((3, 2, 6, 6)))
    out = net.forward(x)
    net.zeroGradParameters()
    net.backward(x, gt.gpu(np.ones(out.size(), np.float32)))
    assert np.abs(fg.float()).sum() > 0
    before = fw.float().copy()
    gt.lib().THGPUNN_SGD_update(fw.cdata, fg.cdata, None, 0.1, 0.0)
    close(net.modules[0].weight.float().reshape(-1), (before - np.float32(0.1) * fg.float())[:72])


def _device_step(gt, net, params, x, labels):
    """Loads `params` into the net's conv / Linear layers, runs forward + loss + backward on the device."""
    layers = [m for m in net.modules if isinstance(m, (gt.nn.SpatialConvolutionMM, gt.nn.Linear))]
    assert len(layers) == len(params)
    for m, (w, b) in zip(layers, params):
        m.weight, m.bias = w.copy(), b.copy()
        m.gradWeight, m.gradBias = np.zeros_like(w), np.zeros_like(b)
    net.gpu()
    crit = gt.nn.ClassNLLCriterion()
    xg, yg = gt.gpu(x), gt.gpu(labels)
    out = net.forward(xg)
    loss = crit.forward(out, yg)
    net.backward(xg, crit.backward(out, yg))
    return loss, layers


def _turned_relus(net, m, params, inp, pre, x):
    """What the ReLU behind layer `m` lets through on one side only: a pre-activation within rounding of zero may come out
    positive on the device and not on the CPU (`inp`: the layer's input there, `pre`: its output before the ReLU), or the
    other way round.  One side then passes the gradient g there and the other does not, which adds g times the unit's
    window of the input to its row of gradWeight and g to its gradBias.  Returns the sums of |g| max|window| and |g| per
    row, zero for rows without such a unit.  Every such unit must have both values within both sides' rounding: K terms
    of a sequential FP32 sum, and the weights times how far the two inputs are apart."""
    w, b = (p.astype(np.float64) for p in params)
    extra_w, extra_b = np.zeros(len(b)), np.zeros(len(b))
    at = net.modules.index(m)
    if at + 2 >= len(net.modules) or type(net.modules[at + 1]).__name__ != "ReLU":
        return extra_w, extra_b
    out = m.output.float().reshape(pre.shape)
    turned = np.argwhere((out > 0) != (pre > 0))
    if len(turned) == 0:
        return extra_w, extra_b
    g = np.abs(net.modules[at + 2].gradInput.float().reshape(pre.shape))
    inputs = [(net.modules[at - 1].output.float() if at else x).reshape(inp.shape), inp]
    if inp.ndim == 4:
        p = m.padding
        inputs = [np.pad(a, ((0, 0), (0, 0), (p, p), (p, p))) for a in inputs]
    for unit in map(tuple, turned):
        n, k = unit[:2]
        if inp.ndim == 4:
            y, z = unit[2] * m.dH, unit[3] * m.dW
            dev, cpu = (a[n, :, y:y + m.kH, z:z + m.kW].ravel().astype(np.float64) for a in inputs)
        else:
            dev, cpu = (a[n].astype(np.float64) for a in inputs)
        rounding = 2 * len(dev) * 2.0 ** -24 * (np.abs(w[k]) @ np.abs(dev) + abs(b[k])) + np.abs(w[k]) @ np.abs(dev - cpu)
        assert max(abs(out[unit]), abs(pre[unit])) <= rounding, (at, unit, out[unit], pre[unit], rounding)
        extra_w[k] += g[unit] * np.abs(dev).max()
        extra_b[k] += g[unit]
    return extra_w, extra_b


def test_alexnet_step_matches_cpu(gt, oracle_port):
    """One whole SGD step of the AlexNet-style classifier over 8 images: the loss and all 16 gradient tensors
    against the CPU path run on the same parameters, inputs and labels -- the reference's own TH/nn code when it was
    compiled (conv1 through its strided nn.SpatialConvolution), else the plain-C restatement."""
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
    import bench
    import oracle
    from mcw_cppamp_torch_b200 import configs
    gt.set_math_mode("fp32x3")
    cpu = "reference" if oracle.ref.available() else "port"
    _, loss_cpu, d = bench.cpu_alexnet_step(cpu, 8, details=True)
    assert len(d["params"]) == 8
    net = configs.alexnet(rng=oracle_port.rng(1))
    loss, layers = _device_step(gt, net, d["params"], d["x"], d["labels"])
    assert abs(loss - loss_cpu) <= 1e-5 + 1e-4 * abs(loss_cpu)
    for i, (m, (gw, gb)) in enumerate(zip(layers, d["grads"])):
        got, got_b = m.gradWeight.float(), m.gradBias.float()
        gw = gw.reshape(got.shape)
        extra_w, extra_b = _turned_relus(net, m, d["params"][i], *d["layers"][i], x=d["x"])
        for k in np.flatnonzero(extra_b):
            what = "alexnet 8 images vs %s: layer %d %%s, plane %d" % (cpu, i + 1, k)
            close_scaled(got[k], gw[k], what % "gradWeight", atol=1e-5 + extra_w[k])
            close_scaled(got_b[k:k + 1], gb[k:k + 1], what % "gradBias", atol=1e-5 + extra_b[k])
        rest = np.flatnonzero(extra_b == 0)
        close_scaled(got[rest], gw[rest], "alexnet 8 images vs %s: layer %d gradWeight" % (cpu, i + 1))
        close_scaled(got_b[rest], gb[rest], "alexnet 8 images vs %s: layer %d gradBias" % (cpu, i + 1))


def test_vgg_a_step_matches_cpu(gt, oracle_port):
    """The VGG-A-style classifier (8 convs 3x3 pad 1, 5 max-pools 2/2, 3 Linear) over 2 images of 224 x 224: loss
    and all 11 (gradWeight, gradBias) pairs against the plain-C CPU path on the same TH-stream tensors."""
    from mcw_cppamp_torch_b200 import configs
    from mcw_cppamp_torch_b200.random import THGenerator
    from util import cpu_classifier_step
    gt.set_math_mode("fp32x3")
    rs = THGenerator(7)
    n = 2
    x = rs.uniform((n, 3, 224, 224), -1, 1)
    labels = rs.labels(n, 1000)
    convs = [(ci, co, 3, 1, 1, (2, 2) if pool else None) for ci, co, pool in configs.VGG_A_CONVS]
    params = []
    for ci, co, k, s, p, pool in convs:
        sd = 1.0 / np.sqrt(ci * k * k)
        params.append((rs.uniform((co, ci * k * k), -sd, sd), rs.uniform((co,), -sd, sd)))
    for fi, fo in configs.VGG_A_FC:
        sd = 1.0 / np.sqrt(fi)
        params.append((rs.uniform((fo, fi), -sd, sd), rs.uniform((fo,), -sd, sd)))
    loss_cpu, grads = cpu_classifier_step(oracle_port, convs, configs.VGG_A_FC, x, labels, params)
    loss, layers = _device_step(gt, configs.vgg_a(rng=oracle_port.rng(1)), params, x, labels)
    assert len(layers) == len(grads) == 11
    assert abs(loss - loss_cpu) <= 1e-5 + 1e-4 * abs(loss_cpu)
    for i, (m, (gw, gb)) in enumerate(zip(layers, grads)):
        got = m.gradWeight.float()
        close_scaled(got, gw.reshape(got.shape), "vgg-a 2 images vs port: layer %d gradWeight" % (i + 1))
        close_scaled(m.gradBias.float(), gb, "vgg-a 2 images vs port: layer %d gradBias" % (i + 1))


@pytest.mark.parametrize("layer", [(64, 192, 5, 2, 27), (192, 384, 3, 1, 13), (384, 256, 3, 1, 13), (256, 256, 3, 1, 13)])
def test_conv_engines_agree_at_full_size(gt, oracle_port, layer):
    """The AlexNet-style layers at the benchmark's per-image size, batch 32: the tensor-core path (planes, two-SM
    tiles, TMA) against the FP32 FMA engine, which shares none of that code, plus exact linearity in the input."""
    ci, co, k, pad, hw = layer
    g = oracle_port.rng(co)
    N = 32
    x = g.uniform((N, ci, hw, hw), -1, 1)
    s = 1.0 / np.sqrt(ci * k * k)
    w, b = g.uniform((co, ci * k * k), -s, s), g.uniform((co,), -s, s)
    go = g.normal((N, co, hw, hw))
    res = {}
    for mode in MODES:
        gt.set_math_mode(mode)
        res[mode] = run_conv(gt, x, w, b, go, (k, k), (1, 1), pad)
    gt.set_math_mode("fp32x3")
    for a, c, name in zip(res["fp32x3"], res["simt"], ("output", "gradInput", "gradWeight", "gradBias")):
        scale = np.abs(c).max()
        assert np.abs(a - c).max() <= 1e-5 + 1e-4 * scale, (name, np.abs(a - c).max(), scale)
    # scaling the input by a power of two scales (output - bias) exactly
    out2 = run_conv(gt, 2 * x, w, np.zeros_like(b), None, (k, k), (1, 1), pad)[0]
    out1 = run_conv(gt, x, w, np.zeros_like(b), None, (k, k), (1, 1), pad)[0]
    assert np.array_equal(out2, 2 * out1)


BF16_RTOL = 2e-2     # of the tensor's largest magnitude: BF16 carries 8 significant bits


@pytest.mark.parametrize("case", [(4, 64, 13, 13, 128, 3, 3, 1, 1, 1), (3, 64, 27, 27, 192, 5, 5, 1, 1, 2),
                                  (2, 40, 9, 9, 130, 3, 3, 1, 1, 1), (2, 32, 12, 15, 64, 3, 3, 2, 2, 1),
                                  (2, 3, 23, 23, 8, 11, 11, 4, 4, 2)])
def test_conv_bf16_mode(gt, oracle_port, case):
    """The opt-in BF16 math mode: all three passes within BF16 accuracy of the float64 values (products that are
    too small for the BF16 engine, like the last case, run on the FP32-accurate path)."""
    gt.set_math_mode("bf16")
    try:
        N, C, H, W, K, kH, kW, dH, dW, pad = case
        g = oracle_port.rng(sum(case) + 1)
        x = g.uniform((N, C, H, W), -1, 1)
        s = 1.0 / np.sqrt(C * kH * kW)
        w, b = g.uniform((K, C * kH * kW), -s, s), g.uniform((K,), -s, s)
        geo = (kH, kW, dH, dW, pad)
        want = conv_exact(x, w, b, *geo)
        go = g.normal(want.shape)
        out, gi, gw, gb = run_conv(gt, x, w, b, go, (kH, kW), (dH, dW), pad)
        gw_e, gb_e = conv_grad_weight_exact(x, go, *geo)
        for got, ref, name in ((out, want, "output"), (gi, conv_grad_input_exact(go, w, x.shape, *geo), "gradInput"),
                               (gw, gw_e, "gradWeight"), (gb, gb_e, "gradBias")):
            assert np.abs(got - ref).max() <= BF16_RTOL * np.abs(ref).max(), (name, np.abs(got - ref).max(), np.abs(ref).max())
    finally:
        gt.set_math_mode("fp32x3")


def test_vgg_a_steps_engines_agree(gt, oracle_port):
    """The VGG-A-style configuration at full image size (4 images, 3 x 224 x 224): two consecutive steps (forward,
    loss, whole backward pass, nothing synchronising the host between layers) on the tensor-core engines against
    the FP32 FMA engine, which shares none of their code (the CPU oracle needs minutes for one such step).

    Among the 29 M pre-activations of such a pass a handful lie within rounding of the ReLU threshold, or tie with
    a neighbour inside a pooling window, and two correct engines may then take different branches: one gradient
    element of that layer, and everything it feeds further down, legitimately differs.  The test finds those
    decisions (ReLU masks and pooling indices of both runs); layers above the highest one must agree to the
    tolerance everywhere, layers at or below it everywhere except a few elements, which are counted and reported."""
    from mcw_cppamp_torch_b200 import configs
    from util import PARITY_REPORT
    g = oracle_port.rng(5)
    x, labels = g.uniform((4, 3, 224, 224), -1, 1), np.array([3, 999, 42, 500], np.float32)
    res = {}
    for mode in MODES:
        gt.set_math_mode(mode)
        net = configs.vgg_a(rng=oracle_port.rng(6))
        layers = [m for m in net.modules if isinstance(m, (gt.nn.SpatialConvolutionMM, gt.nn.Linear))]
        assert len(layers) == 11
        net.gpu()
        crit = gt.nn.ClassNLLCriterion()
        xg, yg = gt.gpu(x), gt.gpu(labels)
        for _ in range(2):
            for m in layers:
                m.gradWeight.zero(); m.gradBias.zero()
            out = net.forward(xg)
            crit.updateOutput(out, yg, read_back=False)
            net.backward(xg, crit.updateGradInput(out, yg))
        loss = crit.forward(out, yg)
        # the branch decisions of the pass, per parameterised layer: ReLU masks and pooling indices that follow it
        decisions, li = [[] for _ in layers], -1
        for m in net.modules:
            if m in layers:
                li += 1
            elif isinstance(m, gt.nn.ReLU):
                decisions[li].append(np.packbits(m.output.float() > 0))
            elif isinstance(m, gt.nn.SpatialMaxPooling):
                decisions[li].append(m.indices.float().astype(np.int16))
        res[mode] = (loss, out.float(), [(m.gradWeight.float(), m.gradBias.float()) for m in layers], decisions)
        del net
    gt.set_math_mode("fp32x3")
    (la, oa, ga, da), (lb, ob, gb, db) = res["fp32x3"], res["simt"]
    assert abs(la - lb) <= 1e-5 + 1e-4 * abs(lb)
    close(oa, ob, what="log-softmax output")
    differs = [i for i, (p, q) in enumerate(zip(da, db)) if any(not np.array_equal(u, v) for u, v in zip(p, q))]
    highest = max(differs) if differs else -1
    PARITY_REPORT.append("vgg-a 4 images, tensor-core engine vs FP32 FMA engine: ReLU / pooling decisions differ after layers %s"
                         % ([i + 1 for i in differs] or "none"))
    for i, ((wa, ba), (wb, bb)) in enumerate(zip(ga, gb)):
        for got, want, name in ((wa, wb, "gradWeight"), (ba, bb, "gradBias")):
            scale = np.abs(want).max()
            outside = int((np.abs(got - want) > 1e-5 + 1e-4 * scale).sum())
            if i <= highest and outside:
                PARITY_REPORT.append("    layer %d %s: %d of %d elements differ by more than 1e-5 + 1e-4 * max|.| (a decision differs at or above this layer)"
                                     % (i + 1, name, outside, got.size))
            allowed = max(2, got.size // 10000) if i <= highest else 0
            assert outside <= allowed, (i, name, outside, np.abs(got - want).max(), scale, differs)
