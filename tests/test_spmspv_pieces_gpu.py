"""The frontier push at the edges of its split (rows of 31, 32, 33 and 127 .. 129 entries, frontiers on both
sides of the 32-entry rule, more pieces than have room when a hub is listed again and again) and its masks
with and without an accumulator, against numpy; whole numbers, so every order gives the same value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def capi():
    from gb_kun_b200 import capi
    capi.init(0)
    return capi


def push(ptr, col, val, ids, xv, n, sr):
    cnt = ptr[ids + 1] - ptr[ids]
    k = np.repeat(np.arange(len(ids)), cnt)
    e = np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt) + ptr[ids][k]
    if sr == "plus_times":
        y = np.zeros(n, np.int64)
        np.add.at(y, col[e], val[e].astype(np.int64) * xv[k])
    elif sr == "min_plus":
        y = np.full(n, np.iinfo(np.int32).max, np.int64)
        np.minimum.at(y, col[e], val[e].astype(np.int64) + xv[k])
    else:
        y = np.zeros(n, np.int64)
        y[col[e]] = 1
    return y


def graph(shape, rng):
    if shape == "repeats":
        degrees = np.array([3000, 40, 5, 0] + [2] * 996)
        ids = np.concatenate([np.zeros(200, np.int64), np.arange(1000), np.ones(50, np.int64)])
    elif shape == "edges":
        degrees = np.tile([0, 1, 31, 32, 33, 127, 128, 129, 300], 60)
        ids = np.flatnonzero(rng.random(len(degrees)) < 0.7)
    else:
        degrees = rng.choice([0, 2, 5, 40], 320_000)
        ids = np.arange(320_000)
    ptr = np.zeros(len(degrees) + 1, np.int64)
    ptr[1:] = np.cumsum(degrees)
    return ptr, rng.integers(0, len(degrees), ptr[-1]), ids


@pytest.mark.parametrize("sr", ["plus_times", "min_plus", "lor_land"])
@pytest.mark.parametrize("shape", ["repeats", "edges", "many"])
def test_push(capi, shape, sr):
    rng = np.random.default_rng(11)
    ptr, col, ids = graph(shape, rng)
    n = len(ptr) - 1
    val, xv = rng.integers(1, 5, len(col)).astype(np.int32), rng.integers(1, 5, len(ids)).astype(np.int32)
    A = capi.Matrix(ptr.astype(np.int32), col.astype(np.int32), val)
    want = push(ptr, col, val, ids, xv, n, sr)
    dids, dx = torch.from_numpy(ids.astype(np.int32)).cuda(), torch.from_numpy(xv).cuda()
    y0 = rng.integers(-9, 10, n).astype(np.int32)
    m = rng.random(n) < 0.3
    dm, sel = torch.from_numpy(m).cuda(), torch.from_numpy(np.flatnonzero(m).astype(np.int32)).cuda()
    saturate = lambda a: np.minimum(a, np.iinfo(np.int32).max)  # noqa: E731
    for accum in ("second", "plus"):
        merged = want if accum == "second" else saturate(y0 + want)
        # (mask, expected): a list of ids that is not complemented touches the listed elements alone
        for mask, expect in ((None, want), (capi.dense_mask(dm), np.where(m, merged, 0)),
                             (capi.dense_mask(dm, "str_comp"), np.where(m, 0, merged)),
                             (capi.sparse_mask(sel), np.where(m, merged, want)),
                             (capi.sparse_mask(sel, "str_comp"), np.where(m, 0, merged))):
            y = torch.from_numpy(y0.copy()).cuda()
            A.spmspv(dids, dx, y, semiring=sr, accum=accum, mask=mask, transpose=True)
            assert np.array_equal(y.cpu().numpy().astype(np.int64), expect)


def test_mask_is_the_output(capi):
    # the mask is applied to the new values, which it then holds
    rng = np.random.default_rng(2)
    ptr, col, ids = graph("edges", rng)
    A = capi.Matrix(ptr.astype(np.int32), col.astype(np.int32), np.ones(len(col), np.int32))
    dids = torch.from_numpy(ids.astype(np.int32)).cuda()
    dx = torch.ones(len(ids), dtype=torch.int32, device="cuda")
    y = torch.zeros(len(ptr) - 1, dtype=torch.int32, device="cuda")
    A.spmspv(dids, dx, y, semiring="plus_times", mask=capi.dense_mask(y), transpose=True)
    want = push(ptr, col, np.ones(len(col), np.int32), ids, np.ones(len(ids), np.int32), len(ptr) - 1, "plus_times")
    assert np.array_equal(y.cpu().numpy(), want)
