"""Triangle counting on the device at the edges of its size classes (the length of a vertex's
oriented list decides whether a warp, a block with a small or a large table, or a search counts it),
at the edges of its 256-entry tiles, and on patterns that are not simple undirected graphs."""
import numpy as np
import pytest

from gb_kun_b200 import graphgen as gg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def capi():
    from gb_kun_b200 import capi
    capi.init(0)
    return capi


def csr(n, src, dst):
    order = np.lexsort((dst, src))
    rp = np.zeros(n + 1, np.int64)
    np.add.at(rp, np.asarray(src) + 1, 1)
    return np.cumsum(rp).astype(np.int32), np.asarray(dst)[order].astype(np.int32)


def count(capi, rp, col):
    return capi.Matrix(rp, col, np.ones(len(col), np.float32)).triangle_count()


# A complete graph on n vertices has one vertex of every oriented length 0 .. n - 1; its vertices lie
# among `total` ids (up to 262,144 of them and more take different sets).
@pytest.mark.parametrize("n,total", [(2, 2), (3, 3), (16, 16), (17, 17), (23, 23), (33, 33), (34, 34), (35, 35),
                                     (1027, 1027), (2600, 2600), (36, 262144), (70, 262145), (2100, 262144),
                                     (1025, 300000), (1026, 300000), (1027, 1700000), (2600, 1700000),
                                     (8300, 1700000)])
def test_complete_graphs(capi, n, total):
    ids = np.arange(n, dtype=np.int64) * (total // n)
    deg = np.zeros(total, np.int64)
    deg[ids] = n - 1
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    col = np.empty((n, n - 1), np.int32)
    for v in range(n):
        col[v, :v] = ids[:v]
        col[v, v:] = ids[v + 1:]
    assert count(capi, rp, col.reshape(-1)) == n * (n - 1) * (n - 2) // 6


@pytest.mark.parametrize("gap", [1, 40])
@pytest.mark.parametrize("n,ef", [(60, 4), (700, 3), (1500, 40)])
def test_random_graphs_with_isolated_vertices(capi, n, ef, gap):
    """Vertex ids spread `gap` apart: runs of empty rows longer and shorter than a warp."""
    rng = np.random.default_rng(n + gap)
    g = gg.from_edges(n, rng.integers(0, n, n * ef), (rng.pareto(1.2, n * ef) * 3).astype(np.int64) % n,
                      undirected=True)
    D = np.zeros((n, n), np.int64)
    D[np.repeat(np.arange(n), g.degrees()), g.col] = 1
    np.fill_diagonal(D, 0)
    want = int(np.trace(D @ D @ D)) // 6
    src, dst = np.nonzero(D)
    rp, col = csr(n * gap, src * gap, dst * gap)
    assert count(capi, rp, col) == want


def test_star_and_empty(capi):
    n = 5000  # a hub row over many tiles, no triangle
    leaves = np.arange(1, n)
    rp, col = csr(n, np.concatenate([np.zeros(n - 1, int), leaves]), np.concatenate([leaves, np.zeros(n - 1, int)]))
    assert count(capi, rp, col) == 0
    assert count(capi, np.zeros(8, np.int32), np.zeros(0, np.int32)) == 0


def masked_count(D):
    """sum((A A) .* A) / 6 with A's multiplicities as a pattern product over sorted lists."""
    return int(((D @ D) * (D > 0)).sum()) // 6


def test_patterns_that_are_not_simple(capi):
    rng = np.random.default_rng(3)
    n = 80
    D = (rng.random((n, n)) < 0.2).astype(np.int64)   # directed
    np.fill_diagonal(D, 0)
    rp, col = csr(n, *np.nonzero(D))
    assert count(capi, rp, col) == masked_count(D)
    D = D | D.T
    np.fill_diagonal(D, rng.integers(0, 2, n))          # self loops
    rp, col = csr(n, *np.nonzero(D))
    assert count(capi, rp, col) == masked_count(D)


def test_repeated_entries(capi):
    """Repeated entries of a symmetric pattern: every listed entry of an edge's shorter oriented list counts."""
    rng = np.random.default_rng(5)
    n = 90
    M = np.triu((rng.random((n, n)) < 0.25) * rng.integers(1, 3, (n, n)), 1)
    M = M + M.T
    src, dst = np.nonzero(M)
    mult = M[src, dst]
    rp, col = csr(n, np.repeat(src, mult), np.repeat(dst, mult))
    deg = np.diff(rp)
    out = [[v for v in col[rp[u]:rp[u + 1]] if (deg[u], u) < (deg[v], v)] for u in range(n)]
    want = 0
    for u in range(n):
        for v in out[u]:
            short, long_ = (out[u], out[v]) if len(out[u]) <= len(out[v]) else (out[v], out[u])
            want += sum(w in set(long_) for w in short)
    assert count(capi, rp, col) == want
