"""Products whose arrays come from the stream-ordered pool: dropping one waits for work that still reads it, on any
stream, and disturbs neither a capture nor a first call in another thread."""
import ctypes
import threading

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


@pytest.fixture(scope="module")
def graph():
    return gg.rmat(11, 8, seed=7, undirected=True)


def square(capi, g):
    A = capi.Matrix.from_graph(g)
    return A.mxm(A)


def test_destroy_waits_for_other_streams(capi, graph):
    C = square(capi, graph)
    ref = torch.zeros(graph.n, device="cuda")
    x = torch.ones(graph.n, device="cuda")
    C.mxv(x, ref)
    y = torch.zeros(graph.n, device="cuda")
    torch.cuda.synchronize()
    side, done = torch.cuda.Stream(), torch.cuda.Event()  # torch's streams do not block the legacy one
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)  # some 50 ms
        C.mxv(x, y)
        done.record()
    assert not done.query()
    C.close()
    assert done.query()
    square(capi, graph)  # takes the same memory
    assert torch.equal(y, ref)


@pytest.mark.parametrize("where", ["other thread", "this thread"])
def test_destroy_during_a_capture(capi, graph, where):
    x = torch.arange(1024, dtype=torch.float32, device="cuda")
    y = torch.zeros_like(x)
    C = square(capi, graph)
    rows = C.download_csr()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    if where == "other thread":
        with torch.cuda.graph(g, capture_error_mode="thread_local"):
            y += x
            t = threading.Thread(target=C.close)
            t.start()
            t.join()
            y *= 2
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, 2 * x)
    else:  # the capture is the caller's to keep; the arrays are freed later
        with torch.cuda.graph(g, capture_error_mode="relaxed"):
            y += x
            C.close()
    # the memory is in order: the next product is right
    for a, b in zip(square(capi, graph).download_csr(), rows):
        assert np.array_equal(a, b)


def test_destroy_beside_first_calls(capi, graph, oracle):
    """One thread drops products while another makes first calls, which capture their loops."""
    want = oracle.bfs(graph, 1)
    A = capi.Matrix.from_graph(graph)
    rows, errors, stop = A.mxm(A).download_csr(), [], threading.Event()

    def products():
        try:
            torch.cuda.set_device(0)
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                while not stop.is_set():
                    C = A.mxm(A, stream=s)
                    got = C.download_csr(stream=s)
                    C.close()
                    assert all(np.array_equal(a, b) for a, b in zip(got, rows))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    t = threading.Thread(target=products)
    t.start()
    try:
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(15):
                B = capi.Matrix.from_graph(graph, stream=s)  # new: its loops are captured by these calls
                levels = torch.zeros(graph.n, dtype=torch.int32, device="cuda")
                B.bfs(1, levels, stream=s)
                many = torch.zeros((4, graph.n), dtype=torch.int32, device="cuda")
                B.msbfs(np.array([1, 1, 1, 1], np.int32), many, stream=s)
                s.synchronize()
                assert np.array_equal(levels.cpu().numpy(), want)
                assert all(np.array_equal(r, want) for r in many.cpu().numpy())
                B.close()
    finally:
        stop.set()
        t.join()
    assert not errors, errors


def default_pool():
    rt = ctypes.CDLL("libcudart.so.12")
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    return rt, pool


def test_what_dropped_products_leave(capi):
    """The device's default pool, which others share, keeps what it had; a server counts what products left as free."""
    from gb_kun_b200.serve import Server
    rt, pool = default_pool()
    reserved = ctypes.c_uint64()

    def now():
        torch.cuda.synchronize()
        assert rt.cudaMemPoolGetAttribute(pool, 5, ctypes.byref(reserved)) == 0  # cudaMemPoolAttrReservedMemCurrent
        return reserved.value

    p = ctypes.c_void_p()  # another user of the default pool, with 5 GiB that it will want again
    assert rt.cudaMallocAsync(ctypes.byref(p), ctypes.c_size_t(5 << 30), None) == 0
    assert rt.cudaFreeAsync(p, None) == 0
    g = gg.rmat(14, 16, seed=9, undirected=True)
    A = capi.Matrix.from_graph(g)
    A.mxm(A).close()
    before = now()
    assert before >= 5 << 30
    C = A.mxm(A)  # 40 M entries
    with_c = Server(A).memory()[1]
    size = 8 * C.nnz
    C.close()
    assert now() == before
    assert Server(A).memory()[1] >= with_c + 0.75 * size  # a server's budget is 80 % of the free memory
    assert rt.cudaMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0
