"""gbk_mxm at the edges of its column windows (1,280 columns for float sums, otherwise 2,048; 131,072 in all)
and for the operands that the windows refuse (repeated or unsorted columns, too many columns, too few products
a window), against sums in numpy: whole numbers, so every order of the sums gives the same value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

COLS = [1, 31, 1279, 1280, 1281, 2047, 2048, 2049, 4097, 64 * 2048 - 1, 64 * 2048, 64 * 2048 + 1]


@pytest.fixture(scope="module")
def capi():
    from gb_kun_b200 import capi
    capi.init(0)
    return capi


def csr(rows, cols, n):
    ptr = np.zeros(n + 1, np.int64)
    np.add.at(ptr, rows + 1, 1)
    return np.cumsum(ptr).astype(np.int32), cols.astype(np.int32)


def pattern(rng, n, m, count):
    """Distinct (row, column) pairs, half of them in the first rows and all columns at both ends."""
    r = np.minimum(rng.integers(0, n, count), rng.integers(0, n, count) * 4)
    c = rng.integers(0, m, count)
    c[:8] = [0, m - 1] * 4
    key = np.unique(r.astype(np.int64) * m + c)
    return key // m, key % m


def product(ar, ac, av, br, bc, bv, m, sr):
    """Entries (key, value) of the product from all its terms, zeros dropped."""
    nb = int(br.max()) + 1
    order = np.argsort(br, kind="stable")
    br, bc, bv = br[order], bc[order], bv[order]
    start = np.searchsorted(br, np.arange(max(nb, int(ac.max()) + 1) + 1))
    cnt = start[ac + 1] - start[ac]
    e = np.repeat(np.arange(len(ac)), cnt)
    f = np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt) + start[ac[e]]
    key = ar[e].astype(np.int64) * m + bc[f]
    a, b = av[e].astype(np.int64), bv[f].astype(np.int64)
    x = {"plus_times": a * b, "plus_second": b, "plus_one": np.ones_like(a), "min_second": b,
         "min_plus": np.minimum(a + b, np.iinfo(np.int32).max), "lor_land": ((a != 0) & (b != 0)).astype(np.int64)}[sr]
    keys, inv = np.unique(key, return_inverse=True)
    if sr.startswith("min"):
        out = np.full(len(keys), np.iinfo(np.int64).max)
        np.minimum.at(out, inv, x)
    else:
        out = np.zeros(len(keys), np.int64)
        np.add.at(out, inv, x)
        if sr == "lor_land":
            out = np.minimum(out, 1)
    keep = out != 0
    return keys[keep], out[keep]


def room(ar, ac, br, bc, n, m, cols):
    """Entries of room that the product asks for: per row and window of `cols` columns its products, at most the
    window's columns."""
    nw = (m + cols - 1) // cols
    parts = np.zeros((max(int(ac.max()), int(br.max())) + 1, nw), np.int64)
    np.add.at(parts, (br, bc // cols), 1)
    tasks = np.zeros((n, nw), np.int64)
    np.add.at(tasks, ar, parts[ac])
    return np.minimum(tasks, np.minimum(cols, m - cols * np.arange(nw))).sum(axis=1)


def set_blocks(monkeypatch, rows_room, blocks):
    """Has a product with this room per row work in one block, in a block per row, or in a few of several rows
    (a block has room for three entries per product allowed)."""
    if blocks == "one":
        monkeypatch.delenv("GBK_MXM_BLOCK_PRODUCTS", raising=False)
        return
    products = 1 if blocks == "rows" else max(1, int(rows_room.sum()) // 12)
    monkeypatch.setenv("GBK_MXM_BLOCK_PRODUCTS", str(products))
    if blocks == "few":
        assert rows_room.sum() > 3 * products  # two blocks at least,
        assert np.sort(rows_room)[:2].sum() <= 3 * products  # and some hold several rows


def check(capi, A, B, want, m):
    C = A.mxm(B, semiring=want[0])
    rp, col, v = C.download_csr()
    assert (C.n, C.ncols) == (A.n, m)
    key = np.repeat(np.arange(A.n, dtype=np.int64), np.diff(rp)) * m + col
    assert np.array_equal(key, want[1])
    assert np.array_equal(v, want[2].astype(v.dtype))


@pytest.mark.parametrize("blocks", ["one", "rows", "few"])
@pytest.mark.parametrize("sr", ["plus_times", "plus_second", "plus_one", "min_plus", "min_second", "lor_land"])
@pytest.mark.parametrize("m", COLS)
def test_windows(capi, monkeypatch, m, sr, blocks):
    rng = np.random.default_rng(m)
    n, k = 61, 47
    ar, ac = pattern(rng, n, k, 900)
    br, bc = pattern(rng, k, m, 6000)
    for dtype in (np.int32, np.float32):
        cols = 1280 if dtype == np.float32 and sr.startswith("plus") else 2048
        set_blocks(monkeypatch, room(ar, ac, br, bc, n, m, cols), blocks)
        av = rng.integers(-3, 4, len(ar)).astype(dtype)
        bv = rng.integers(-3, 4, len(br)).astype(dtype)
        if dtype == np.int32 and sr.startswith("min"):
            av[ar == 5] = 1
            bv[:] = np.where(rng.random(len(bv)) < 0.3, np.iinfo(np.int32).max, bv)  # reached, and the identity
        A = capi.Matrix(*csr(ar, ac, n), av, ncols=k)
        B = capi.Matrix(*csr(br, bc, k), bv, ncols=m)
        check(capi, A, B, (sr, *product(ar, ac, av, br, bc, bv, m, sr)), m)


@pytest.mark.parametrize("sr", ["plus_times", "plus_second", "plus_one", "min_plus", "min_second", "lor_land"])
@pytest.mark.parametrize("length", [511, 512, 513, 3000])
@pytest.mark.parametrize("blocks", ["one", "rows", "few"])
def test_hub_rows(capi, monkeypatch, length, sr, blocks):
    # a row whose windows a CTA works on, beside short ones
    rng = np.random.default_rng(length)
    n, k, m = 20, 3000, 2100
    ar, ac = pattern(rng, n, k, 300)
    hub = np.sort(rng.permutation(k)[:length])
    key = np.unique(np.concatenate([ar * k + ac, 7 * k + hub]))
    ar, ac = key // k, key % k
    br, bc = pattern(rng, k, m, 200_000)
    for dtype in (np.int32, np.float32):
        cols = 1280 if dtype == np.float32 and sr.startswith("plus") else 2048
        set_blocks(monkeypatch, room(ar, ac, br, bc, n, m, cols), blocks)
        av, bv = rng.integers(-3, 4, len(ar)).astype(dtype), rng.integers(-3, 4, len(br)).astype(dtype)
        A = capi.Matrix(*csr(ar, ac, n), av, ncols=k)
        B = capi.Matrix(*csr(br, bc, k), bv, ncols=m)
        check(capi, A, B, (sr, *product(ar, ac, av, br, bc, bv, m, sr)), m)


@pytest.mark.parametrize("form", ["repeated", "unsorted", "empty", "tall"])
def test_refused_operands(capi, form):
    rng = np.random.default_rng(3)
    n, k, m = (40, 200_000, 64 * 2048) if form == "tall" else (40, 30, 5000)  # tall: far more rows than products
    ar, ac = pattern(rng, n, k, 400)
    br, bc = pattern(rng, k, m, 3000)
    if form == "repeated":
        br, bc = np.concatenate([br, br[::7]]), np.concatenate([bc, bc[::7]])
        order = np.lexsort((bc, br))
        br, bc = br[order], bc[order]
    elif form == "unsorted":
        order = np.lexsort((-bc, br))
        br, bc = br[order], bc[order]
    av = rng.integers(1, 4, len(ar)).astype(np.int32)
    bv = rng.integers(1, 4, len(br)).astype(np.int32)
    A = capi.Matrix(*csr(ar, ac, n), av, ncols=k)
    B = capi.Matrix(*csr(br, bc, k), bv, ncols=m)
    if form == "empty":
        E = capi.Matrix(np.zeros(k + 1, np.int32), np.zeros(0, np.int32), np.zeros(0, np.int32), ncols=m)
        C = A.mxm(E)
        assert C.nnz == 0 and (C.n, C.ncols) == (n, m)
        return
    check(capi, A, B, ("plus_times", *product(ar, ac, av, br, bc, bv, m, "plus_times")), m)


def test_infinities_and_nan(capi):
    # row 0: inf * 0 (NaN, kept) and inf; row 1: 1 * 0 (dropped) and inf - inf; row 2: -inf + inf
    A = capi.Matrix(np.array([0, 1, 3, 5], np.int32), np.array([0, 0, 1, 1, 2], np.int32),
                    np.array([np.inf, 1, 1, 1, 1], np.float32), ncols=3)
    B = capi.Matrix(np.array([0, 2, 3, 4], np.int32), np.array([0, 2500, 2500, 2500], np.int32),
                    np.array([0, np.inf, -np.inf, np.inf], np.float32), ncols=3000)
    rp, col, v = A.mxm(B).download_csr()
    assert rp.tolist() == [0, 2, 3, 4] and col.tolist() == [0, 2500, 2500, 2500]
    assert np.isnan(v[0]) and v[1] == np.inf and np.isnan(v[2]) and np.isnan(v[3])


def dense_rows(rng, rows, length, m):
    """A with `length` entries in every row, B with all of `m` columns, of random floats in [0, 1)."""
    ptr = np.arange(0, (rows + 1) * length, length).astype(np.int32)
    col = np.tile(np.arange(length), rows).astype(np.int32)
    bptr = np.arange(0, (length + 1) * m, m).astype(np.int32)
    bcol = np.tile(np.arange(m), length).astype(np.int32)
    return (ptr, col, rng.random(rows * length).astype(np.float32)), (bptr, bcol, rng.random(length * m).astype(np.float32))


@pytest.mark.parametrize("blocks", [1, 5])
@pytest.mark.parametrize("m,length", [(300, 4000), (2100, 700), (1, 500), (1, 4000), (1, 16000), (8, 300), (1281, 200)])
def test_float_sums(capi, monkeypatch, m, length, blocks):
    # Products rounded to 32 bits, their sums in 64: each product of non-negative terms and the final rounding
    # add at most 2^-24 of the sum.  32-bit sums of 500 terms in order: 3.0e-7, of 4,000: 7.9e-7.
    rows = 20
    rng = np.random.default_rng(m)
    (ap, ac, av), (bp, bc, bv) = dense_rows(rng, rows, length, m)
    monkeypatch.delenv("GBK_MXM_BLOCK_PRODUCTS", raising=False)
    if blocks > 1:  # a block has room for three entries per product allowed
        monkeypatch.setenv("GBK_MXM_BLOCK_PRODUCTS", str(rows * m // (3 * blocks)))
    C = capi.Matrix(ap, ac, av, ncols=length).mxm(capi.Matrix(bp, bc, bv, ncols=m))
    rp, col, v = C.download_csr()
    assert rp.tolist() == list(range(0, (rows + 1) * m, m)) and np.array_equal(col, np.tile(np.arange(m), rows))
    want = av.reshape(rows, length).astype(np.float64) @ bv.reshape(length, m).astype(np.float64)
    err = np.linalg.norm(v.reshape(rows, m) - want) / np.linalg.norm(want)
    assert err <= 2.0 ** -23


@pytest.mark.parametrize("graph,scale,factor,windows", [
    ("uniform", 16, 16, False), ("uniform", 15, 2, False), ("uniform", 15, 32, True), ("uniform", 14, 4, True),
    ("rmat", 14, 8, True)])
def test_route(capi, graph, scale, factor, windows):
    # A product with far fewer products than (row, window) tasks is expanded, as it was before the windows (uniform
    # 2^16, 16 entries a row: 2.6 ms, 6.8 by windows).  The same product with B's rows unsorted is always expanded:
    # the number of launches tells the routes apart.
    from gb_kun_b200 import graphgen as gg
    g = getattr(gg, graph)(scale, factor, seed=3, undirected=graph == "rmat")
    ptr, col = np.asarray(g.row_ptr).astype(np.int32), np.asarray(g.col).astype(np.int32)
    val = np.random.default_rng(4).integers(1, 5, len(col)).astype(np.float32)  # whole sums: every order alike
    rows = np.repeat(np.arange(g.n), np.diff(ptr))
    o = np.lexsort((-col, rows))
    A, U = capi.Matrix(ptr, col, val), capi.Matrix(ptr, col[o], val[o])
    out, launches = [], []
    for B in (A, U):
        before = capi.launch_count()
        C = A.mxm(B)
        launches.append(capi.launch_count() - before)
        out.append(C.download_csr())
    for x, y in zip(*out):
        assert np.array_equal(x, y)
    assert (launches[0] != launches[1]) == windows
