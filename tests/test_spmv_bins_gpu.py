"""The degree-binned CSR product at the edges of its bins (2 entries a lane: rows of 2, 3, 4, 5, 8, 9, ... 64,
65, 2048, 2049 entries), with rows in and outside a mask of every type, warps that take several batches of rows,
and accumulators, against numpy; whole numbers, so every order of a sum gives the same value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGES = [0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 2047, 2048, 2049, 4100]


@pytest.fixture(scope="module")
def capi():
    from gb_kun_b200 import capi
    capi.init(0)
    return capi


def matrix(rng, degrees, ncols):
    ptr = np.zeros(len(degrees) + 1, np.int64)
    ptr[1:] = np.cumsum(degrees)
    col = rng.integers(0, ncols, ptr[-1])
    return ptr.astype(np.int32), col.astype(np.int32)


def rowwise(f, ptr, x, ident):
    """f.reduceat over the rows, the identity for empty ones."""
    out = np.full(len(ptr) - 1, ident, np.int64)
    full = np.flatnonzero(np.diff(ptr))
    if len(full):
        out[full] = f.reduceat(x, ptr[full])
    return out


@pytest.mark.parametrize("mask_type", [None, np.bool_, np.int32, np.float32])
@pytest.mark.parametrize("accum", ["second", "plus", "min"])
@pytest.mark.parametrize("shape", ["edges", "many"])
def test_bins(capi, shape, accum, mask_type):
    rng = np.random.default_rng(5)
    if shape == "edges":
        degrees = np.repeat(EDGES, rng.integers(1, 40, len(EDGES)))
        rng.shuffle(degrees)
    else:  # more rows than the warps hold at once: several batches a warp
        degrees = rng.choice([3, 7, 12, 20], 1_300_000, p=[0.1, 0.5, 0.2, 0.2])
    n, m = len(degrees), 5000
    ptr, col = matrix(rng, degrees, m)
    x, y0 = rng.integers(-4, 5, m), rng.integers(-50, 50, n)
    mask = None if mask_type is None else (rng.random(n) < 0.4)
    for dtype in (np.int32, np.float32):
        val = rng.integers(-3, 4, len(col)).astype(dtype)
        A = capi.Matrix(ptr, col, val, ncols=m)
        A.set_format("CSR", csr_kernel=2)
        dx = torch.from_numpy(x.astype(dtype)).cuda()
        dm = None if mask is None else torch.from_numpy(mask.astype(mask_type)).cuda()
        v64, big = val.astype(np.int64), np.iinfo(np.int32).max
        for sr, ident, want in (("plus_times", 0, rowwise(np.add, ptr, v64 * x[col], 0)),
                                ("plus_second", 0, rowwise(np.add, ptr, x[col], 0)),
                                ("min_plus", big, rowwise(np.minimum, ptr, v64 + x[col], big))):
            if sr == "min_plus" and (dtype == np.float32 or accum == "plus"):
                continue  # a largest value of its own; saturates
            want = {"second": want, "plus": y0 + want, "min": np.minimum(y0, want)}[accum]
            if mask is not None:
                want = np.where(mask, want, 0)
            dy = torch.from_numpy(y0.astype(dtype)).cuda()
            A.mxv(dx, dy, semiring=sr, accum=accum, mask=dm)
            assert np.array_equal(dy.cpu().numpy().astype(np.int64), want), sr
