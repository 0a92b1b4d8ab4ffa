"""Element-wise calls on vectors that are worked on four elements a thread, beside the same vectors one
element past that alignment (the general kernels), and the dense-to-sparse, counting and reducing calls over
lengths around a warp's step and the ranges of the CTAs, against numpy.  Single operations: exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def capi():
    from gb_kun_b200 import capi
    capi.init(0)
    return capi


def dev(a, offset):
    """a on the GPU, `offset` elements past a 16-byte boundary."""
    t = torch.zeros(len(a) + 8, dtype=torch.from_numpy(a).dtype, device="cuda")
    v = t[offset:offset + len(a)]
    v.copy_(torch.from_numpy(a))
    return v


NUMPY = {"plus": np.add, "minus": np.subtract, "times": np.multiply, "min": np.minimum, "max": np.maximum,
         "second": lambda a, b: b, "ne": lambda a, b: (a != b), "lt": lambda a, b: (a < b)}


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4099, 3_000_001])
@pytest.mark.parametrize("dtype", [np.float32, np.int32])
def test_ewise_apply_accum(capi, dtype, n, offset):
    rng = np.random.default_rng(n)
    a, b, c = (rng.integers(-9, 10, n).astype(dtype) for _ in range(3))
    m = rng.random(n) < 0.5
    code = capi.F32 if dtype == np.float32 else capi.I32
    da, db, dm = dev(a, offset), dev(b, offset), dev(m, offset)
    for op, f in NUMPY.items():
        want = f(a, b).astype(dtype)
        w = dev(c, offset)
        capi.ewise(op, code, w, da, db)
        assert np.array_equal(w.cpu().numpy(), want)
        w = dev(c, offset)
        capi.ewise(op, code, w, da, db, mask=capi.dense_mask(dm))
        assert np.array_equal(w.cpu().numpy(), np.where(m, want, c))
        wb = dev(np.zeros(n, bool), offset)
        capi.ewise(op, code, wb, da, db)
        assert np.array_equal(wb.cpu().numpy(), want != 0)
        w = dev(c, offset)
        capi.assign_vector(op, code, w, db)
        assert np.array_equal(w.cpu().numpy(), f(c, b).astype(dtype))
        for kind, g in ((1, lambda x: f(dtype(3), x)), (2, lambda x: f(x, dtype(3)))):
            w = dev(c, offset)
            capi.apply(kind, op, code, w, da, scalar=3)
            assert np.array_equal(w.cpu().numpy(), np.broadcast_to(g(a), n).astype(dtype))
    w = dev(a, offset)
    capi.apply(0, "abs", code, w, w)  # in place
    assert np.array_equal(w.cpu().numpy(), np.abs(a))
    idx = rng.integers(0, n, n).astype(np.int32)
    w = dev(c, offset)
    capi.extract("second", code, w, da, indices=dev(idx, offset))
    assert np.array_equal(w.cpu().numpy(), a[idx])


@pytest.mark.parametrize("share", [0.0, 0.03, 1.0])
@pytest.mark.parametrize("n", [1, 31, 128, 129, 1024, 1025, 148 * 8 * 1024, 148 * 8 * 1024 + 1, 4_000_003])
@pytest.mark.parametrize("dtype", [np.float32, np.int32, np.bool_, np.int64, np.float64])
def test_sparse_count_reduce(capi, dtype, n, share):
    rng = np.random.default_rng(n)
    a = np.where(rng.random(n) < share, rng.integers(1, 9, n), 0).astype(dtype)
    if share == 1.0 and dtype == np.float32 and n > 1:
        a[0], a[-1] = np.nan, -0.0  # NaN is an element, minus zero is not
    d = dev(a, 1)
    ids, vals = capi.to_sparse(d)
    want = np.flatnonzero(a != 0)
    assert np.array_equal(ids.cpu().numpy(), want)
    assert np.array_equal(vals.cpu().numpy(), a[want], equal_nan=a.dtype.kind == "f")
    assert capi.nvals(d) == len(want)
    a = np.nan_to_num(a)
    d = dev(a, 1)
    rt = {np.float32: capi.F64, np.float64: capi.F64}.get(dtype, capi.I64)
    assert capi.reduce("plus", rt, d) == a.astype(np.float64).sum()  # whole numbers below 2^53
    if dtype != np.bool_:
        assert capi.reduce("max", rt, d) == a.max() and capi.reduce("min", rt, d) == a.min()
