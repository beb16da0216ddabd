"""The warp-level product engine (small and narrow products, any pitch and alignment) and the packing in front of the
two-SM engine, at tile edges, remainders and slice counts, in the four layouts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gt():
    import mcw_cppamp_torch_b200 as gt
    gt.set_math_mode("fp32x3")
    return gt


def bound(A, B, K):
    """3xTF32 drops terms of 2^-22 |a||b|; a 32-k tile's chains truncate 12 times at 2^-23 of what they have summed and
    every tile (and slice) is added once at 2^-24: all relative to the sum of |a||b|."""
    rel = 2.0 ** -22 + 12 * 2.0 ** -23 + (K / 32 + 34) * 2.0 ** -24
    return rel * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64)) + 1e-30


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 8, 32), (65, 9, 33), (8, 64, 31), (63, 16, 65), (130, 17, 100), (200, 64, 68),
                                   (67, 33, 640), (5, 70, 4099), (129, 40, 2050), (256, 192, 128), (1001, 777, 1531)])
@pytest.mark.parametrize("beta", [0.0, 1.0, 0.5])
def test_products(gt, M, N, K, beta):
    g = np.random.default_rng(M * 7919 + N * 31 + K)
    A, B, C = (g.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (M, N)))
    exact = beta * C.astype(np.float64) + 0.75 * (A.astype(np.float64) @ B.astype(np.float64))
    tol = bound(A, B, K) + 2.0 ** -22 * (np.abs(exact) + np.abs(C))
    wide_a, wide_b = gt.gpu(np.zeros((M, K + 3), np.float32)), gt.gpu(np.zeros((K, N + 1), np.float32))
    va, vb = wide_a.narrow(2, 2, K).copy(A), wide_b.narrow(2, 2, N).copy(B)          # pitch and address off 16 bytes
    for a in (gt.gpu(A), gt.gpu(np.ascontiguousarray(A.T)).t(), va):
        for b in (gt.gpu(B), gt.gpu(np.ascontiguousarray(B.T)).t(), vb):
            r = gt.gpu(C if beta else np.full((M, N), np.nan, np.float32))
            r.addmm(beta, 0.75, a, b)
            got = r.float()
            assert np.all(np.abs(got - exact) <= tol)
            again = gt.gpu(C if beta else np.full((M, N), np.nan, np.float32)).addmm(beta, 0.75, a, b).float()
            assert np.array_equal(got, again)
    rt = gt.gpu(np.ascontiguousarray(C.T)).t()                                       # column-major result
    rt.addmm(beta, 0.75, gt.gpu(A), gt.gpu(B))
    assert np.all(np.abs(rt.float() - exact) <= tol)


@pytest.mark.parametrize("rows,inputs,outputs", [(1, 9216, 300), (13, 1000, 130), (33, 257, 7), (300, 512, 1000), (1, 1, 1)])
@pytest.mark.parametrize("mode", ["fp32x3", "simt", "bf16"])
def test_linear_forward_bias(gt, rows, inputs, outputs, mode):
    gt.set_math_mode(mode)
    try:
        g = np.random.default_rng(rows + inputs)
        x, w, b = (g.standard_normal(s).astype(np.float32) for s in ((rows, inputs), (outputs, inputs), (outputs,)))
        m = gt.nn.Linear(inputs, outputs)
        m.weight, m.bias = w, b
        got = m.gpu().forward(gt.gpu(x)).float()
        exact = x.astype(np.float64) @ w.T + b
        scale = np.abs(x).astype(np.float64) @ np.abs(w.T) + np.abs(b)
        # bf16 operands: 2^-8 on each product; FP32 chains of the FMA engine: at most K roundings
        rel = {"fp32x3": 2.0 ** -19, "simt": inputs * 2.0 ** -24 + 2.0 ** -22, "bf16": 2.0 ** -7}[mode]
        assert np.all(np.abs(got - exact) <= (rel + inputs / 32 * 2.0 ** -24) * scale)
    finally:
        gt.set_math_mode("fp32x3")


def test_nan_and_infinity_reach_the_result(gt):
    A = np.ones((70, 40), np.float32)
    A[3, 5], A[4, 6] = np.nan, np.inf
    A[2, 1:2].view(np.uint32)[:] = 0x7fffffff           # the NaN that device arithmetic makes
    r = gt.GPUTensor(70, 20).zero().addmm(0.0, 1.0, gt.gpu(A), gt.gpu(np.ones((40, 20), np.float32))).float()
    assert np.isnan(r[2:4]).all() and np.all(r[4] == np.inf) and np.all(r[5] == 40)


@pytest.mark.filterwarnings("ignore:invalid value encountered")
@pytest.mark.parametrize("n", [2, 8, 12, 20, 33, 70])
@pytest.mark.parametrize("k", [40, 44, 700])
def test_values_next_to_the_largest(gt, n, k):
    """Operands whose TF32 part would round to infinity, on either side, and infinities: what FP32 arithmetic gives.  (Products of
    the two-SM engine keep the finite ones; an infinity there meets its own NaN low part.)"""
    top = np.finfo(np.float32).max
    g = np.random.default_rng(n + k)
    A, B = (g.standard_normal(s).astype(np.float32) for s in ((70, k), (k, n)))
    A[:4] = 0
    A[0, 5], A[1, 5], A[2, 7], A[3, 9] = top, -3.4028e38, np.inf, -np.inf
    B[5], B[7], B[9] = 0.5, 2, 4096                                                      # exact in TF32: no low part
    exact = A.astype(np.float64) @ B.astype(np.float64)
    for a in (gt.gpu(A), gt.gpu(np.ascontiguousarray(A.T)).t()):
        for b in (gt.gpu(B), gt.gpu(np.ascontiguousarray(B.T)).t()):
            r = gt.GPUTensor(70, n).zero().addmm(0.0, 1.0, a, b).float()
            assert np.all(np.abs(r[:2] / exact[:2] - 1) <= 2.0 ** -21)
            assert np.all(r[2] == np.inf) and np.all(r[3] == -np.inf)
            assert np.all(np.abs(r[4:] - exact[4:]) <= (bound(A, B, k) + 2.0 ** -22 * np.abs(exact))[4:])
            other = gt.GPUTensor(n, 70).zero().addmm(0.0, 1.0, b.t(), a.t()).float()     # the huge ones on the other side
            assert np.array_equal(other.T[2:4], r[2:4]) and np.all(np.abs(other.T[:2] / exact[:2] - 1) <= 2.0 ** -21)


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("inputs,outputs", [(4, 9), (124, 33), (516, 4099), (9216, 260), (4096, 2049)])
def test_few_rows(gt, rows, inputs, outputs):
    """Few rows against a K-major matrix: remainders of rows, outputs and k chunks, both sides of the size rule."""
    g = np.random.default_rng(rows * 31 + inputs)
    x, w, b = (g.standard_normal(s).astype(np.float32) for s in ((rows, inputs), (outputs, inputs), (outputs,)))
    m = gt.nn.Linear(inputs, outputs)
    m.weight, m.bias = w, b
    got = m.gpu().forward(gt.gpu(x)).float()
    exact = x.astype(np.float64) @ w.T.astype(np.float64) + b
    tol = bound(x, w.T, inputs) + 2.0 ** -22 * (np.abs(exact) + np.abs(b))
    assert np.all(np.abs(got - exact) <= tol)
    c = g.standard_normal((rows, outputs)).astype(np.float32)
    r = gt.gpu(c).addmm(0.5, 0.75, gt.gpu(x), gt.gpu(w).t()).float()
    exact = 0.5 * c.astype(np.float64) + 0.75 * (x.astype(np.float64) @ w.T.astype(np.float64))
    assert np.all(np.abs(r - exact) <= bound(x, w.T, inputs) + 2.0 ** -22 * (np.abs(exact) + np.abs(c)))


def test_accumulating_costs_no_round_trip_per_element(gt):
    """1574 x 1276 x 2, bound by its result: 15 us overwriting it, 18 adding to it (53 with a load behind every store)."""
    import torch
    a, b, r = gt.GPUTensor(1574, 2).fill(1), gt.GPUTensor(2, 1276).fill(1), gt.GPUTensor(1574, 1276).fill(0)
    stream = torch.cuda.ExternalStream(gt.lib().THGPUGetStream())

    def us(beta):
        times = []
        for _ in range(7):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record(stream)
            for _ in range(20):
                r.addmm(beta, 1.0, a, b)
            t1.record(stream)
            t1.synchronize()
            times.append(t0.elapsed_time(t1) * 50)
        return sorted(times)[3]
    us(0.0)
    assert us(1.0) < 2 * us(0.0)
