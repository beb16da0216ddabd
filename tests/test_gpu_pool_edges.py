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
