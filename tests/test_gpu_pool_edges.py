"""The row-walking pooling kernels at the widths and heights where lanes, tiles, bands and store alignment change, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 3, 3), (2, 3, 4, 15), (3, 2, 5, 16), (2, 5, 17, 17), (1, 2, 9, 31), (1, 3, 10, 32), (2, 1, 33, 33), (1, 2, 8, 62),
          (1, 2, 7, 63), (1, 1, 12, 64), (2, 2, 11, 65), (1, 3, 6, 66), (1, 1, 130, 127), (1, 2, 5, 129), (3, 7, 13, 13), (1, 40, 55, 55),
          (2, 1, 224, 8)]


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("shape", SHAPES)
def test_pooling_edges(oracle_port, shape, k):
    import mcw_cppamp_torch_b200 as gt
    g = np.random.default_rng(sum(shape) + k)
    x = g.standard_normal(shape).astype(np.float32)
    x.reshape(-1)[::3] = 0.5                            # ties: neighbouring windows share maxima
    x.reshape(-1)[1::17] = np.nan
    x[0, 0, :3, :3] = -np.inf                           # a window without a maximum
    m = gt.nn.SpatialMaxPooling(k, k, 2, 2)
    xg = gt.gpu(x)
    out, ind = m.forward(xg).float(), m.indices.float()
    want, wind = oracle_port.maxpool_forward(x, k, k, 2, 2)
    assert np.array_equal(out.view(np.uint32), want.view(np.uint32)) and np.array_equal(ind, wind)
    # gradients: from an input in which every window has a maximum
    x = np.where(np.isfinite(x), x, np.float32(0.25))
    out = m.forward(gt.gpu(x)).float()
    want, wind = oracle_port.maxpool_forward(x, k, k, 2, 2)
    assert np.array_equal(out, want) and np.array_equal(m.indices.float(), wind)
    go = g.standard_normal(want.shape).astype(np.float32)
    gi = m.updateGradInput(gt.gpu(x), gt.gpu(go)).float()
    assert np.array_equal(gi, oracle_port.maxpool_backward(go, wind, x.shape, 2, 2))


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("W", [8, 9])
def test_negative_zero_gradients(k, W):
    """The CPU adds a gradient to a zeroed pixel, which turns -0 into +0; no pixel of the result has a sign bit."""
    import mcw_cppamp_torch_b200 as gt
    x = gt.gpu(np.random.default_rng(W).standard_normal((2, 3, 9, W)).astype(np.float32))
    p = gt.nn.SpatialMaxPooling(k, k, 2, 2)
    out = p.forward(x).size()
    gi = p.updateGradInput(x, gt.gpu(np.full(out, -0.0, np.float32))).float()
    assert np.all(gi == 0) and not np.signbit(gi).any()


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("shape", SHAPES + [(2, 3, 8, 64), (3, 4, 18, 65), (1, 2, 34, 66), (5, 24, 24), (2, 2, 9, 128)])
def test_threshold_and_pooling_in_one_pass(shape, k):
    """A container's pass over both modules leaves in each what their own calls leave, bit for bit (nothing is rounded)."""
    import mcw_cppamp_torch_b200 as gt
    g = np.random.default_rng(sum(shape) * 2 + k)
    x = g.standard_normal(shape).astype(np.float32)
    x.reshape(-1)[::5] = 0.25
    x.reshape(-1)[1::17] = np.nan
    x.reshape(-1)[2::29] = -np.inf
    xg = gt.gpu(x)
    for th, val in ((0.0, 0.0), (0.25, -1.5)):
        one, two = [(gt.nn.Threshold(th, val), gt.nn.SpatialMaxPooling(k, k, 2, 2)) for _ in range(2)]
        net = gt.nn.Sequential().add(one[0]).add(one[1])
        n = gt.lib().THGPUKernelLaunchCount()
        out = net.forward(xg)
        assert gt.lib().THGPUKernelLaunchCount() == n + 1
        want = two[1].forward(two[0].forward(xg))
        go = gt.gpu(g.standard_normal(want.size()).astype(np.float32))
        n = gt.lib().THGPUKernelLaunchCount()
        gi = net.backward(xg, go)
        assert gt.lib().THGPUKernelLaunchCount() == n + 1
        two[0].backward(xg, two[1].backward(two[0].output, go))
        for a, b in ((out, want), (one[0].output, two[0].output), (one[1].indices, two[1].indices), (one[1].gradInput, two[1].gradInput),
                     (gi, two[0].gradInput)):
            assert a.size() == b.size() and np.array_equal(a.float().view(np.uint32), b.float().view(np.uint32))


# Tensors large enough for the kernels that take whole planes: widths on both sides of the rules, planes and groups that do not come out even.
@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("shape", [(67, 401, 13, 13), (23, 257, 27, 29), (31, 1000, 9, 16), (9, 191, 55, 55), (5, 101, 101, 97), (7, 230, 51, 54), (4700, 90, 10, 10),
                                   (331, 170, 29, 27), (90000, 7, 9, 8), (5, 100000, 3, 3), (1501, 3, 31, 32), (3, 100, 60, 62), (2, 99, 84, 66)])
def test_whole_planes(oracle_port, shape, k):
    import mcw_cppamp_torch_b200 as gt
    g = np.random.default_rng(sum(shape) + 3 * k)
    x = g.standard_normal(shape, dtype=np.float32)
    x.reshape(-1)[::7] = 0.5
    relu = np.where(x > 0, x, np.float32(0))
    xg, rg = gt.gpu(x), gt.gpu(relu)
    net = gt.nn.Sequential().add(gt.nn.ReLU()).add(gt.nn.SpatialMaxPooling(k, k, 2, 2))
    m = gt.nn.SpatialMaxPooling(k, k, 2, 2)
    want, wind = oracle_port.maxpool_forward(relu, k, k, 2, 2)
    go = g.standard_normal(want.shape, dtype=np.float32)
    back = oracle_port.maxpool_backward(go, wind, x.shape, 2, 2)
    gg = gt.gpu(go)
    assert np.array_equal(net.forward(xg).float(), want) and np.array_equal(net.modules[1].indices.float(), wind)
    assert np.array_equal(net.modules[0].output.float(), relu)
    assert np.array_equal(net.backward(xg, gg).float(), np.where(x > 0, back, np.float32(0)))
    assert np.array_equal(net.modules[1].gradInput.float(), back)
    assert np.array_equal(m.forward(rg).float(), want) and np.array_equal(m.indices.float(), wind)
    assert np.array_equal(m.updateGradInput(rg, gg).float(), back)
    if shape[1] * shape[2] * shape[3] % 4:   # without the first image: an address that 16-byte pieces do not start on
        tail = xg.narrow(1, 2, shape[0] - 1)
        assert np.array_equal(net.forward(tail).float(), want[1:])


def test_one_pass_only_for_what_it_knows():
    """Other windows, strided inputs, results over their sources, overridden methods: the modules' own calls, same results."""
    import mcw_cppamp_torch_b200 as gt
    g = np.random.default_rng(5)
    x = g.standard_normal((2, 3, 12, 11)).astype(np.float32)
    relu = np.where(x > 0, x, np.float32(0))

    def net(k, d):
        return gt.nn.Sequential().add(gt.nn.ReLU()).add(gt.nn.SpatialMaxPooling(k, k, d, d))

    def alone(k, d, data):
        r, p = gt.nn.ReLU(), gt.nn.SpatialMaxPooling(k, k, d, d)
        return p.forward(r.forward(gt.gpu(data))).float()

    assert np.array_equal(net(3, 1).forward(gt.gpu(x)).float(), alone(3, 1, x))
    t = gt.gpu(np.ascontiguousarray(x.transpose(0, 1, 3, 2))).transpose(3, 4)
    assert np.array_equal(net(2, 2).forward(t).float(), alone(2, 2, x))
    m, xg = net(3, 2), gt.gpu(x)
    m.modules[0].output = xg                                        # in place
    assert np.array_equal(m.forward(xg).float(), alone(3, 2, x)) and np.array_equal(xg.float(), relu)
    m, calls = net(2, 2), []
    m.modules[1].updateOutput = lambda v: calls.append(1) or v
    assert m.forward(gt.gpu(x)) is m.modules[0].output and calls == [1]
    with pytest.raises(gt.THCError):
        net(2, 2).forward(gt.GPUTensor(1, 1, 1))
    m = net(2, 2)
    out = m.forward(gt.gpu(x))
    with pytest.raises(gt.THCError):
        m.backward(gt.gpu(x), gt.GPUTensor(*(v + 1 for v in out.size())))


def test_sources_that_borrow_a_results_memory():
    """A result outgrows memory that a source lies in: what the source holds is read before that memory goes back."""
    import mcw_cppamp_torch_b200 as gt
    L = gt.lib()

    def borrow(t, *shape):
        s = L.THGPUStorage_newWithData(t.data_ptr(), int(np.prod(shape)))
        v = gt.GPUTensor(_ptr=L.THGPUTensor_newWithStorage1d(s, 0, int(np.prod(shape)), 1)).view(*shape)
        L.THGPUStorage_free(s)
        return v

    g = np.random.default_rng(9)
    shape, pooled = (2, 3, 12, 11), (2, 3, 6, 5)
    n, x, go = int(np.prod(shape)), g.standard_normal(shape).astype(np.float32), g.standard_normal(pooled).astype(np.float32)
    r, p = gt.nn.ReLU(), gt.nn.SpatialMaxPooling(2, 2, 2, 2)
    want = p.forward(r.forward(gt.gpu(x))).float()
    back = r.backward(gt.gpu(x), p.backward(r.output, gt.gpu(go))).float()
    for field in ("output", "indices"):
        m = gt.nn.Sequential().add(gt.nn.ReLU()).add(gt.nn.SpatialMaxPooling(2, 2, 2, 2))
        held = gt.GPUTensor(n + 8)
        held.narrow(1, 1, n).copy(x.reshape(-1))
        setattr(m.modules[1], field, held.narrow(1, n + 1, 8))      # its storage has no room for the result behind it
        xg = borrow(held, *shape)
        del held
        assert np.array_equal(m.forward(xg).float(), want)
    m = gt.nn.Sequential().add(gt.nn.ReLU()).add(gt.nn.SpatialMaxPooling(2, 2, 2, 2))
    xg = gt.gpu(x)
    m.forward(xg)
    m.modules[0].gradInput = gt.gpu(go)
    gg = borrow(m.modules[0].gradInput, *pooled)
    assert np.array_equal(m.backward(xg, gg).float(), back)


@pytest.mark.parametrize("k,shape", [(3, (256, 64, 64, 64)), (2, (64, 256, 56, 56))])
def test_pooling_by_itself_goes_by_rows(k, shape):
    """Without a threshold, planes of these widths took a quarter to two fifths longer through shared memory than by rows, which memory off
    a 16-byte boundary is taken by."""
    import torch
    import mcw_cppamp_torch_b200 as gt
    stream = torch.cuda.ExternalStream(gt.lib().THGPUGetStream())
    n = int(np.prod(shape))
    m, held, back = gt.nn.SpatialMaxPooling(k, k, 2, 2).gpu(), gt.GPUTensor(n + 4).fill(0.5), gt.GPUTensor(n + 4)
    at = lambda t, first: t.narrow(1, first, n).view(*shape)
    go = m.forward(at(held, 1)).clone()

    def ms(f):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        f()
        b.record(stream)
        b.synchronize()
        return a.elapsed_time(b)

    times = {}
    for _ in range(7):
        for first in (1, 2):
            x = at(held, first)
            m.gradInput = at(back, first)
            times.setdefault((first, "forward"), []).append(ms(lambda: m.updateOutput(x)))
            times.setdefault((first, "back"), []).append(ms(lambda: m.updateGradInput(x, go)))
    for way in ("forward", "back"):
        assert sorted(times[1, way])[3] < 1.12 * sorted(times[2, way])[3], way


# (2 x 2 windows go back by planes from 40 M pixels on)
@pytest.mark.parametrize("k,shape", [(3, (67, 401, 13, 13)), (3, (23, 257, 27, 29)), (3, (9, 191, 55, 55)), (2, (331, 170, 29, 27)), (3, (20, 64, 35, 33)),
                                     (3, (40, 100, 21, 19)), (2, (60, 64, 20, 38)), (3, (26, 420, 11, 5)),
                                     (2, (90, 45, 9, 9))])
def test_whole_planes_of_special_values(k, shape):
    """NaN, infinities, windows without a maximum, ties, zeros of both signs: the same bits as by rows, which batches of few pixels and memory off
    16-byte boundaries are taken by."""
    import mcw_cppamp_torch_b200 as gt
    g = np.random.default_rng(sum(shape))
    x = g.standard_normal(shape, dtype=np.float32)
    flat = x.reshape(-1)
    for step, v in ((7, 0.5), (11, -np.inf), (13, np.nan), (17, 0.25), (19, -0.0), (1009, np.inf)):
        flat[::step] = v
    x[1, :, :8, :8] = -np.inf
    x[2, :, 3:9, 2:9] = np.nan
    xg, per = gt.gpu(x), (1 << 20 if shape[3] > 9 else 1 << 18) // int(np.prod(shape[1:]))   # (narrow planes: from 2^18 pixels on)
    bits = lambda t: t.float().view(np.uint32)

    def off(t):
        """the same values, 4 bytes off a 16-byte boundary"""
        size, n = t.size(), int(np.prod(t.size()))
        u = gt.GPUTensor(n + 1).narrow(1, 2, n).view(*size)
        return u.copy(t)

    def run(make, outs, xs, go, before=None):
        m = make()
        if before:
            before(m)
        m.forward(xs)
        m.backward(xs, go)
        return [bits(f(m)) for f in outs]

    net = lambda: gt.nn.Sequential().add(gt.nn.Threshold(0.25, -1.5)).add(gt.nn.SpatialMaxPooling(k, k, 2, 2))
    fields = [lambda m: m.output, lambda m: m.modules[0].output, lambda m: m.modules[1].gradInput, lambda m: m.gradInput]
    pool, one = lambda: gt.nn.SpatialMaxPooling(k, k, 2, 2), [lambda m: m.output, lambda m: m.gradInput]
    go = g.standard_normal((*shape[:2], (shape[2] - k) // 2 + 1, (shape[3] - k) // 2 + 1), dtype=np.float32)
    go.reshape(-1)[::5] = -0.0
    gg = gt.gpu(go)
    for make, outs in ((net, fields), (pool, one)):
        whole = run(make, outs, xg, gg)
        for n in range(0, shape[0], per):
            c = min(per, shape[0] - n)
            for a, b in zip(whole, run(make, outs, xg.narrow(1, n + 1, c), gg.narrow(1, n + 1, c))):
                assert np.array_equal(a[n:n + c], b)
    whole = run(net, fields, xg, gg)
    for before in (lambda m: setattr(m.modules[1], "gradInput", off(xg)), lambda m: setattr(m.modules[0], "gradInput", off(xg)),
                   lambda m: setattr(m.modules[0], "output", off(xg))):
        for a, b in zip(whole, run(net, fields, xg, gg, before)):
            assert np.array_equal(a, b)
    for a, b in zip(whole, run(net, fields, off(xg), gg)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("k,shape", [(3, (1, 10909, 11, 5)), (2, (1, 16363, 11, 5)), (3, (1, 11111, 9, 9))])
def test_one_pass_over_narrow_planes(k, shape):
    """Threshold and pooling in one pass take no longer than one after the other; by rows, which planes of so few columns leave idle, they did."""
    import torch
    import mcw_cppamp_torch_b200 as gt
    stream = torch.cuda.ExternalStream(gt.lib().THGPUGetStream())
    x, net = gt.GPUTensor(*shape).fill(0.5), gt.nn.Sequential().add(gt.nn.ReLU()).add(gt.nn.SpatialMaxPooling(k, k, 2, 2)).gpu()
    relu, pool = gt.nn.ReLU().gpu(), gt.nn.SpatialMaxPooling(k, k, 2, 2).gpu()

    def ms(f):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(50):
            f()
        b.record(stream)
        b.synchronize()
        return a.elapsed_time(b)

    one, two = (sorted(ms(f) for _ in range(9))[4] for f in (lambda: net.updateOutput(x), lambda: pool.updateOutput(relu.updateOutput(x))))
    assert one < two
