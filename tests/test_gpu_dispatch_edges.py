"""The elementwise, reduction and host-copy kernels at the sizes where their dispatch changes: tile edges and 16-byte
alignment of transposed operands, one block or many and one slice or several in the reductions, the staging limit of
small downloads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gt():
    import mcw_cppamp_torch_b200 as gt
    return gt


def borrowed(gt, ptr, *shape):
    """A tensor over memory that some other storage owns."""
    L = gt.lib()
    n = int(np.prod(shape))
    s = L.THGPUStorage_newWithData(ptr, n)
    t = gt.GPUTensor(_ptr=L.THGPUTensor_newWithStorage1d(s, 0, n, 1))
    L.THGPUStorage_free(s)
    return t.view(*shape)


@pytest.mark.parametrize("r,c", [(64, 64), (4, 8), (63, 65), (128, 68), (130, 3), (3, 130), (200, 516), (577, 129)])
def test_transposed_operands(gt, r, c):
    g = np.random.default_rng(r * 1000 + c)
    x, y, z = (g.standard_normal(s).astype(np.float32) for s in ((r, c), (c, r), (c, r)))
    X, Y, Z, R = gt.gpu(x), gt.gpu(y), gt.gpu(z), gt.GPUTensor(r, c)
    half = np.float32(0.5)
    assert np.array_equal(R.copy(Y.t()).float(), y.T)
    assert np.array_equal(R.add(X, 0.5, Y.t()).float(), x + half * y.T)                  # second operand transposed
    assert np.array_equal(R.add(Y.t(), 0.5, X).float(), y.T + half * x)                  # first
    assert np.array_equal(R.add(Y.t(), 0.5, Z.t()).float(), y.T + half * z.T)            # both
    out = gt.GPUTensor(c, r)
    out.t().cmul(X, Y.t())
    assert np.array_equal(out.float(), (x * y.T).T)                                      # result transposed
    sub = gt.GPUTensor(r, c + 3).zero()
    sub.narrow(2, 2, c).copy(Y.t())                                                      # pitch and address off 16 bytes
    want = np.zeros((r, c + 3), np.float32)
    want[:, 1:1 + c] = y.T
    assert np.array_equal(sub.float(), want)


@pytest.mark.parametrize("r,c", [(64, 64), (4, 8), (63, 65), (128, 68), (130, 3), (200, 516), (577, 129)])
def test_transposed_operands_of_addcmul(gt, r, c):
    """Every set of transposed operands, contiguous and transposed results, in whole 16-byte pieces and off them."""
    g = np.random.default_rng(r * 1000 + c)
    v = [g.standard_normal((r, c)).astype(np.float32) + np.float32(3) for _ in range(3)]
    half = np.float32(0.5)
    mul, div = v[0] + half * v[1] * v[2], v[0] + half * v[1] / v[2]
    for turned in range(8):
        a, b, d = (gt.gpu(np.ascontiguousarray(x.T)).t() if turned >> k & 1 else gt.gpu(x) for k, x in enumerate(v))
        assert np.array_equal(gt.GPUTensor(r, c).addcmul(a, 0.5, b, d).float(), mul)
        assert np.array_equal(gt.GPUTensor(r, c).addcdiv(a, 0.5, b, d).float(), div)
        out = gt.GPUTensor(c, r)
        out.t().addcmul(a, 0.5, b, d)
        assert np.array_equal(out.float(), mul.T)
        a.addcmul(0.5, b, d)
        assert np.array_equal(a.float(), mul)


@pytest.mark.parametrize("few", [2, 4, 7, 8, 11, 12, 13])
@pytest.mark.parametrize("many", [129, 4096])
def test_transposed_operands_of_a_few_rows(gt, few, many):
    for r, c in ((few, many), (many, few)):
        test_transposed_operands(gt, r, c)
        test_transposed_operands_of_addcmul(gt, r, c)


def device_us(gt, f, n=5):
    """Median time of f() on the library's stream."""
    import torch
    s, times = torch.cuda.ExternalStream(gt.lib().THGPUGetStream()), []
    for _ in range(n + 2):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        f()
        b.record(s)
        b.synchronize()
        times.append(a.elapsed_time(b) * 1e3)
    return sorted(times[2:])[n // 2]


def test_addcmul_reads_transposed_operands_by_lines(gt):
    """At 8192 x 8192: 161 us contiguous; one operand (the result) transposed 527 (1346) when elements are fetched one by one a
    row apart, 170 (194) through tiles."""
    n = 8192
    t, a, b, at, tt = (gt.GPUTensor(n, n).fill(1.0) for _ in range(5))
    plain = device_us(gt, lambda: t.addcmul(0.5, a, b))
    assert device_us(gt, lambda: t.addcmul(0.5, at.t(), b)) < 2 * plain
    assert device_us(gt, lambda: tt.t().addcmul(0.5, a, b)) < 2 * plain


@pytest.mark.parametrize("cols", [(1 << 24) + 4, (1 << 24) + 5])
def test_transposed_copy_of_very_long_rows(gt, cols):
    """Rows of 16.8 M floats: 2.0 ms through tiles, 8.7 element by element (1.3 for the contiguous copy)."""
    x, y = gt.GPUTensor(64, cols), gt.GPUTensor(cols, 64)
    for r in range(1, 65):
        x.narrow(1, r, 1).fill(r)
    x.narrow(2, 12345678, 1).fill(77)
    y.copy(x.t())
    want = np.arange(1, 65, dtype=np.float32)
    lo, hi = y.min(1)[0].float().ravel(), y.max(1)[0].float().ravel()
    assert np.array_equal(lo, want) and np.all(hi == 77)
    assert np.all(y.narrow(1, 12345678, 1).float() == 77) and np.array_equal(y.narrow(1, cols, 1).float().ravel(), want)
    flat = y.view(64, cols)
    assert device_us(gt, lambda: y.copy(x.t()), 3) < 3 * device_us(gt, lambda: flat.copy(x), 3)


def test_addcmul_in_place_with_overlapping_operand(gt):
    x = np.random.default_rng(3).standard_normal((96, 96)).astype(np.float32)
    X = gt.gpu(x)
    X.addcmul(0.5, X.t(), X)
    assert np.array_equal(X.float(), x + np.float32(0.5) * x.T * x)


@pytest.mark.parametrize("r", [96, 1031])
def test_addcmul_over_borrowed_memory(gt, r):
    """The result's memory seen through another storage: transposed, and one element further on."""
    x = np.random.default_rng(4).standard_normal((r, r)).astype(np.float32)
    half = np.float32(0.5)
    for _ in range(5):
        X = gt.gpu(x)
        X.addcmul(0.5, borrowed(gt, X.data_ptr(), r, r).t(), X)
        assert np.array_equal(X.float(), x + half * x.T * x)
        buf = gt.gpu(x.ravel())
        a = buf.narrow(1, 2, r * r - 1)
        a.addcdiv(0.5, borrowed(gt, buf.data_ptr(), r * r - 1), a)
        assert np.array_equal(a.float(), x.ravel()[1:] + half * x.ravel()[:-1] / x.ravel()[1:])


@pytest.mark.parametrize("offset", [0, 5, 40])
def test_addcmul_into_a_view_that_grows_over_its_operands(gt, offset):
    x = np.random.default_rng(7).standard_normal(9000).astype(np.float32)
    want = x[2000:5000] + np.float32(0.5) * x[40:3040] * x[offset:offset + 3000]
    buf = gt.gpu(x)
    r = buf.narrow(1, 1, 4)                                                              # the first four, 3000 in a moment
    r.addcmul(buf.narrow(1, 2001, 3000), 0.5, buf.narrow(1, 41, 3000), buf.narrow(1, offset + 1, 3000))
    assert np.array_equal(r.float(), want) and np.array_equal(buf.float()[3000:], x[3000:])


@pytest.mark.parametrize("n", [1, 3, 4096 * 4, 4096 * 4 + 4, 4096 * 4 + 1, 300007])
def test_full_reductions(gt, n):
    x = (np.random.default_rng(n).standard_normal(n) + 0.5).astype(np.float32)
    X = gt.gpu(x)
    # a float32 run of four and the final rounding: 3 roundings of terms bounded by the sum of magnitudes
    bound = 4 * 2.0 ** -24 * np.abs(x.astype(np.float64)).sum() + 1e-12
    assert abs(X.sum() - x.astype(np.float64).sum()) <= bound
    assert X.max() == x.max() and X.min() == x.min()
    exact = np.sqrt((x.astype(np.float64) ** 2).sum())
    assert abs(X.norm() - exact) <= 8 * 2.0 ** -24 * exact
    assert abs(X.dist(gt.gpu(np.zeros_like(x))) - exact) <= 64 * 2.0 ** -24 * exact      # powf: a few ulp a term
    last = gt.lib().THGPUTensor_get1d(X.cdata, n - 1)
    assert last == x[-1]


@pytest.mark.parametrize("shape", [(256, 40), (257, 40), (8200, 33), (700, 128), (5000, 132), (1000, 516), (3, 511), (3, 512),
                                   (9, 31), (7, 4097), (3, 300, 130), (2, 5000, 8)])
def test_dim_reductions(gt, shape):
    g = np.random.default_rng(sum(shape))
    x = g.standard_normal(shape).astype(np.float32)
    x.reshape(-1)[::7] = 5.0            # ties across slices: the first maximum wins
    X = gt.gpu(x)
    for dim in range(x.ndim):
        s, (v, i) = X.sum(dim + 1).float(), X.max(dim + 1)
        x64 = x.astype(np.float64)
        assert np.all(np.abs(s - x64.sum(dim, keepdims=True)) <= 2.0 ** -23 * np.abs(x64).sum(dim, keepdims=True))
        assert np.array_equal(v.float(), x.max(dim, keepdims=True))
        assert np.array_equal(i.float(), np.expand_dims(x.argmax(dim), dim) + 1)
        lo, k = X.min(dim + 1)
        assert np.array_equal(lo.float(), x.min(dim, keepdims=True)) and np.array_equal(k.float(), np.expand_dims(x.argmin(dim), dim) + 1)
    X.sum(X, 1)                          # the result in the source's own storage
    assert X.size() == (1,) + shape[1:]
    assert np.all(np.abs(X.float() - x.astype(np.float64).sum(0, keepdims=True)) <= 2.0 ** -23 * np.abs(x.astype(np.float64)).sum(0, keepdims=True))


def test_dim_reductions_over_more_than_2_31_rows(gt):
    rows = (1 << 31) + 8
    x = gt.GPUTensor(rows, 2).fill(0)
    for first, value in ((5, 1), (1 << 31, 7), (rows, 2)):
        x.narrow(1, first, 1).fill(value)
    x.narrow(1, rows - 6, 1).narrow(2, 2, 1).fill(-3)
    (hi, i), (lo, k) = x.max(1), x.min(1)
    assert hi.float().tolist() == [[7, 7]] and i.float().tolist() == [[float(1 << 31)] * 2]
    assert lo.float().tolist() == [[0, -3]] and k.float().tolist() == [[1, float(np.float32(rows - 6))]]
    assert x.sum(1).float().tolist() == [[10, 7]]


@pytest.mark.parametrize("shape,dim", [((300, 64), 1), ((64, 300), 2), ((700, 64), 1)])
def test_values_and_indices_in_one_storage(gt, shape, dim):
    """Two views of one buffer, both of which have to grow: the values are written, then the indices over what they share."""
    x = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    buf = gt.GPUTensor(8).fill(-1)
    v, i = buf.narrow(1, 1, 4), buf.narrow(1, 5, 4)
    src = gt.gpu(x)
    gt.lib().THGPUTensor_max(v.cdata, i.cdata, src.cdata, dim - 1)
    val, pos = x.max(dim - 1), x.argmax(dim - 1) + 1
    assert np.array_equal(i.float().ravel(), pos)
    assert np.array_equal(v.float().ravel(), np.concatenate([val[:4], pos[:-4]]))


@pytest.mark.parametrize("shape,dim", [((3000, 600), 2), ((1000, 4096), 1), ((5000, 40), 2)])
def test_dim_reductions_into_memory_the_source_borrows(gt, shape, dim):
    """Destination and source over the same memory through storages of their own: the source is read before it is written."""
    x = np.random.default_rng(6).standard_normal(shape).astype(np.float32)
    out = tuple(1 if d == dim - 1 else n for d, n in enumerate(shape))
    for _ in range(5):
        src = gt.gpu(x)
        v, i = borrowed(gt, src.data_ptr(), *out), gt.GPUTensor()
        gt.lib().THGPUTensor_max(v.cdata, i.cdata, src.cdata, dim - 1)
        assert np.array_equal(v.float(), x.max(dim - 1, keepdims=True))
        assert np.array_equal(i.float(), np.expand_dims(x.argmax(dim - 1), dim - 1) + 1)
        src = gt.gpu(x)
        i, v = borrowed(gt, src.data_ptr(), *out), gt.GPUTensor()
        gt.lib().THGPUTensor_max(v.cdata, i.cdata, src.cdata, dim - 1)
        assert np.array_equal(v.float(), x.max(dim - 1, keepdims=True))
        assert np.array_equal(i.float(), np.expand_dims(x.argmax(dim - 1), dim - 1) + 1)


@pytest.mark.parametrize("n", [1, 1023, 16384, 16385])
def test_download_sizes(gt, n):
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    out = np.zeros(n, np.float32)
    assert gt.gpu(x).float(out) is out and np.array_equal(out, x)


@pytest.mark.parametrize("n", [(1 << 21) - 1, 1 << 21, (1 << 21) + 1, 17 << 17, 2500007])
def test_large_uploads_from_several_threads(gt, n):
    """Staged uploads around their smallest size and piece boundaries; a second thread that finds the stager busy."""
    import threading
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    bad = []

    def work(k):
        y = x + np.float32(k)
        for _ in range(4):
            if not np.array_equal(gt.gpu(y).float(), y):
                bad.append(k)
    ts = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    assert np.array_equal(gt.gpu(np.arange(n)).float(), np.arange(n).astype(np.float32))      # another element type


def test_first_products_of_a_process_from_several_threads():
    """What the engines look up once per process is there for every thread that comes while it is being looked up."""
    import subprocess
    import sys
    code = """if True:
        import threading, numpy as np, mcw_cppamp_torch_b200 as gt
        a = np.random.default_rng(1).standard_normal((640, 640)).astype(np.float32)
        start, got = threading.Barrier(8), []
        def work():
            x, r = gt.gpu(a), gt.GPUTensor(640, 640)
            start.wait()
            got.append(r.addmm(0.0, 1.0, x, x).float())
        ts = [threading.Thread(target=work) for _ in range(8)]
        [t.start() for t in ts]; [t.join() for t in ts]
        assert len(got) == 8 and all(np.array_equal(g, got[0]) for g in got)
        """
    subprocess.check_call([sys.executable, "-c", code], timeout=300)
