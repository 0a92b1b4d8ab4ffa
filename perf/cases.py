"""Performance cases of the framework: the calls a user's program makes, at the sizes it makes them.

Every case goes through the public Python entry points (`gb_kun_b200.capi`): semiring products over
the storage formats, the frontier push, the element-wise vector calls, the single-query algorithms,
triangle counting, sparse products and the batched traversals.  Graphs are seeded R-MAT (a/b/c/d =
.57/.19/.19/.05, the benchmark's parameters) or uniform random graphs, de-duplicated, without self
loops, generated on the GPU; sizes are those of the benchmark and the tests or lie between them.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gb_kun_b200 import capi

DAMPING = 0.85

# The largest size of each kind is the listed case's; draw() goes down from there.
LISTED = [
    # a product on a small graph, where launches and latency are the cost (an inner step of an
    # iterative solver on a small network); odd size
    {"name": "mxv_small", "kind": "mxv", "graph": "rmat", "n": 5003, "ef": 16, "undirected": False,
     "semiring": "plus_times", "dtype": "f32", "format": "csr", "transpose": False, "masked": False},
    # the benchmark's CSR product: R-MAT scale 18, FP32 plus-times
    {"name": "mxv_csr", "kind": "mxv", "graph": "rmat", "n": 1 << 18, "ef": 16, "undirected": False,
     "semiring": "plus_times", "dtype": "f32", "format": "csr", "transpose": False, "masked": False},
    # the benchmark's headline product: R-MAT scale 22 in the format its autotuner picks there
    {"name": "mxv_staged", "kind": "mxv", "graph": "rmat", "n": 1 << 22, "ef": 16, "undirected": False,
     "semiring": "plus_times", "dtype": "f32", "format": "sell_staged", "transpose": False, "masked": False},
    # a masked relaxation step along in-edges with integer weights on a graph without hubs (vxm,
    # min-plus, min accumulator, a third of the vertices selected); ragged size
    {"name": "vxm_masked", "kind": "mxv", "graph": "uniform", "n": 1_000_003, "ef": 16, "undirected": False,
     "semiring": "min_plus", "dtype": "i32", "format": "csr", "transpose": True, "masked": True},
    # one frontier expansion of a BFS written as GraphBLAS calls: or-and push from a sparse frontier
    # of 3 % of the vertices, the visited vertices masked out
    {"name": "spmspv", "kind": "spmspv", "graph": "rmat", "n": 1 << 20, "ef": 16, "undirected": False,
     "semiring": "lor_land", "dtype": "f32", "fraction": 0.03, "masked": True},
    # the element-wise calls of one PageRank / FastSV iteration written as GraphBLAS calls; odd size
    {"name": "vector_step", "kind": "vector", "n": (1 << 22) + 5, "fraction": 0.1},
    # single-source BFS on an undirected social-network-like graph
    {"name": "bfs", "kind": "bfs", "graph": "rmat", "n": 1 << 21, "ef": 16, "undirected": True, "levels": "i32"},
    # single-source shortest paths, integer weights in a float matrix as the reference stores them
    {"name": "sssp", "kind": "sssp", "graph": "rmat", "n": 1 << 20, "ef": 16, "undirected": True, "dtype": "f32",
     "whole": True},
    # PageRank, 20 iterations, on the matrix as it was loaded (CSR)
    {"name": "pagerank", "kind": "pagerank", "graph": "rmat", "n": 1 << 20, "ef": 16, "undirected": True,
     "format": "csr", "itermax": 20},
    # triangle counting, the benchmark's checked size: R-MAT scale 17
    {"name": "triangles", "kind": "triangles", "graph": "rmat", "n": 1 << 17, "ef": 16, "undirected": True},
    # a sparse product A A (two-hop neighbourhoods), one scale below the benchmark's
    {"name": "mxm", "kind": "mxm", "graph": "rmat", "n": 1 << 14, "ef": 16, "undirected": True,
     "semiring": "plus_times", "dtype": "f32"},
    # one full admission of the query mix a server packs: 64 BFS, 32 personalised PageRank and 32
    # shortest-path queries over one resident graph
    {"name": "batch", "kind": "batch", "graph": "rmat", "n": 1 << 20, "ef": 16, "undirected": False,
     "bfs": 64, "ppr": 32, "sssp": 32, "itermax": 20},
]


def listed():
    return [dict(c) for c in LISTED]


def _size(rng, lo, hi):
    """Log-uniform over [lo, hi]; powers of two only by chance."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mxv", "mxv", "mxv", "spmspv", "vector", "bfs", "sssp", "pagerank", "triangles", "mxm",
                       "batch"])
    graph = {"graph": rng.choice(["rmat", "rmat", "uniform"]), "ef": rng.choice([4, 8, 16])}
    if kind == "mxv":
        semiring, dtype = rng.choice([("plus_times", "f32"), ("plus_times", "f32"), ("plus_second", "f32"),
                                      ("min_plus", "i32"), ("lor_land", "i32")])
        return {"kind": kind, **graph, "n": _size(rng, 1 << 10, 1 << 21), "undirected": rng.random() < 0.5,
                "semiring": semiring, "dtype": dtype,
                "format": rng.choice(["csr", "csr", "sell", "sell_staged", "csr_seg", "lav"]),
                "transpose": rng.random() < 0.5, "masked": rng.random() < 0.3}
    if kind == "spmspv":
        semiring, dtype = rng.choice([("lor_land", "f32"), ("lor_land", "i32"), ("plus_times", "f32"),
                                      ("min_plus", "i32")])
        return {"kind": kind, **graph, "n": _size(rng, 1 << 11, 1 << 20), "undirected": rng.random() < 0.5,
                "semiring": semiring, "dtype": dtype, "fraction": round(10.0 ** rng.uniform(-3, -0.7), 5),
                "masked": rng.random() < 0.5}
    if kind == "vector":
        return {"kind": kind, "n": _size(rng, 1 << 10, 1 << 22), "fraction": round(10.0 ** rng.uniform(-3, -0.05), 5)}
    if kind == "bfs":
        return {"kind": kind, **graph, "n": _size(rng, 1 << 11, 1 << 21), "undirected": rng.random() < 0.7,
                "levels": rng.choice(["i32", "f32"])}
    if kind == "sssp":
        dtype = rng.choice(["f32", "i32"])
        return {"kind": kind, **graph, "n": _size(rng, 1 << 11, 1 << 20), "undirected": rng.random() < 0.7,
                "dtype": dtype, "whole": dtype == "i32" or rng.random() < 0.5}
    if kind == "pagerank":
        return {"kind": kind, **graph, "n": _size(rng, 1 << 11, 1 << 20), "undirected": rng.random() < 0.5,
                "format": rng.choice(["csr", "csr_seg", "sell_staged"]), "itermax": rng.choice([10, 20])}
    if kind == "triangles":
        return {"kind": kind, **graph, "n": _size(rng, 1 << 10, 1 << 17), "undirected": True}
    if kind == "mxm":
        semiring, dtype = rng.choice([("plus_times", "f32"), ("plus_one", "i32"), ("min_plus", "i32"),
                                      ("lor_land", "f32")])
        return {"kind": kind, **graph, "n": _size(rng, 1 << 8, 1 << 14), "undirected": rng.random() < 0.5,
                "semiring": semiring, "dtype": dtype}
    return {"kind": kind, **graph, "n": _size(rng, 1 << 11, 1 << 19), "undirected": rng.random() < 0.5,
            "bfs": rng.randint(1, 64), "ppr": rng.randint(1, 32), "sssp": rng.randint(1, 32), "itermax": 20}


# ---- inputs ------------------------------------------------------------------

@functools.lru_cache(None)
def _init():
    capi.init(0)


def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _edges(case, seed):
    """(row pointers, rows, columns) of the case's graph: int64, sorted by row, then column."""
    # the entries of a sparse product are counted by its inputs: those are one graph under the seed's
    # own vertex numbering, so that results of all seeds have the same number of entries
    label = seed if case.get("kind") == "mxm" else None
    seed = 0 if label is not None else seed
    n, m, g = case["n"], case["n"] * case["ef"], _gen(seed, 1)
    if case["graph"] == "uniform":
        src = torch.randint(n, (m,), generator=g, device="cuda")
        dst = torch.randint(n, (m,), generator=g, device="cuda")
    else:
        src = torch.zeros(m, dtype=torch.int64, device="cuda")
        dst = torch.zeros(m, dtype=torch.int64, device="cuda")
        for _ in range(max(1, (n - 1).bit_length())):
            r = torch.rand(m, generator=g, device="cuda")
            src.mul_(2).add_(r >= 0.76)
            dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        src.remainder_(n)
        dst.remainder_(n)
    if case["undirected"]:
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    if label is not None:
        new = torch.randperm(n, generator=_gen(label, 9), device="cuda")
        src, dst = new[src], new[dst]
    key = torch.unique(src * n + dst)
    rows = torch.div(key, n, rounding_mode="floor")
    cols = key - rows * n
    keep = rows != cols
    rows, cols = rows[keep], cols[keep]
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.bincount(rows, minlength=n).cumsum(0)
    return ptr, rows, cols


@functools.lru_cache(64)
def _counts(graph, n, ef, undirected, fraction):
    """(stored entries, entries of a frontier of that fraction) of the graph of seed 0: what work() counts with."""
    case = {"graph": graph, "n": n, "ef": ef, "undirected": undirected, "fraction": fraction}
    ptr, rows, _ = _edges(case, 0)
    ids = _frontier(case, 0)
    return int(rows.numel()), int((ptr[ids + 1] - ptr[ids]).sum())


def _frontier(case, seed):
    n = case["n"]
    keep = torch.rand(n, generator=_gen(seed, 2), device="cuda") < case.get("fraction", 0.0)
    keep[int(seed) % n] = True
    return torch.nonzero(keep).flatten()


def _values(case, nnz, seed):
    """Entry values: (0, 1] in floats, whole weights 1..255 for integers and for whole float weights."""
    g = _gen(seed, 3)
    if case.get("dtype", "f32") == "i32":
        return torch.randint(1, 256, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    if case.get("whole"):
        return torch.randint(1, 256, (nnz,), generator=g, device="cuda").float()
    return 1.0 - torch.rand(nnz, generator=g, device="cuda")


def _dense(case, seed, salt):
    g, n = _gen(seed, salt), case["n"]
    if case.get("dtype", "f32") == "i32":
        if case.get("semiring") == "lor_land":
            return (torch.rand(n, generator=g, device="cuda") < 0.3).int()
        return torch.randint(0, 100000, (n,), generator=g, device="cuda", dtype=torch.int32)
    return 1.0 - torch.rand(n, generator=g, device="cuda")


def _mask(case, seed, share):
    return torch.rand(case["n"], generator=_gen(seed, 5), device="cuda") < share


def _matrix(ptr, cols, vals):
    return capi.Matrix(ptr.int().cpu().numpy(), cols.int().cpu().numpy(), vals.cpu().numpy())


def _sources(ptr, count, seed):
    """Distinct vertices with out-edges, as the benchmark draws its queries."""
    live = torch.nonzero(ptr[1:] > ptr[:-1]).flatten()
    pick = torch.randperm(live.numel(), generator=_gen(seed, 6), device="cuda")[:count]
    return live[pick].cpu().numpy().astype(np.int32)


_FORMATS = {
    "sell": ("SELL_C", {"sigma": 4096, "reorder_cols": 1}),
    "sell_staged": ("SELL_C", {"seg_staged": 1, "reorder_cols": 1}),
    "csr_seg": ("CSR_SEG", {}),
    "lav": ("LAV", {}),
}


def _set_format(A, case):
    if case["format"] != "csr":
        name, params = _FORMATS[case["format"]]
        A.set_format(name, **params)


def _vector_inputs(case, seed):
    n, g = case["n"], _gen(seed, 7)
    r = torch.rand(n, generator=g, device="cuda")
    y = torch.rand(n, generator=g, device="cuda")
    d = 1.0 + 30.0 * torch.rand(n, generator=g, device="cuda")
    m = torch.rand(n, generator=g, device="cuda") < 0.5
    f = torch.randint(0, n, (n,), generator=g, device="cuda", dtype=torch.int32)
    front = torch.zeros(n, device="cuda")
    set_ = torch.randperm(n, generator=g, device="cuda")[:max(1, int(n * case["fraction"]))]
    front[set_] = 1.0 - torch.rand(set_.numel(), generator=g, device="cuda")
    return r, y, d, m, f, front


def prepare(case, seed):
    _init()
    kind, n = case["kind"], case["n"]
    s = {"case": case}
    if kind == "vector":
        s["r"], s["y"], s["d"], s["m"], s["f"], s["front"] = _vector_inputs(case, seed)
        s["w"], s["diff"], s["z"] = (torch.zeros(n, device="cuda") for _ in range(3))
        s["gp"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        s["changed"] = torch.zeros(n, dtype=torch.bool, device="cuda")
        return s
    ptr, rows, cols = _edges(case, seed)
    s["A"] = A = _matrix(ptr, cols, _values(case, rows.numel(), seed))
    if kind == "mxv":
        _set_format(A, case)
        s["x"] = _dense(case, seed, 4)
        s["y"] = _dense(case, seed, 8)
        s["mask"] = _mask(case, seed, 0.33) if case["masked"] else None
    elif kind == "spmspv":
        ids = _frontier(case, seed)
        s["ids"] = ids.int()
        s["vals"] = torch.ones(ids.numel(), device="cuda", dtype=torch.float32 if case["dtype"] == "f32" else torch.int32)
        s["y"] = torch.zeros(n, device="cuda", dtype=s["vals"].dtype)
        s["mask"] = _mask(case, seed, 0.2) if case["masked"] else None
    elif kind == "bfs":
        s["source"] = int(_sources(ptr, 1, seed)[0])
        s["levels"] = torch.zeros(n, device="cuda", dtype=torch.int32 if case["levels"] == "i32" else torch.float32)
    elif kind == "sssp":
        s["source"] = int(_sources(ptr, 1, seed)[0])
        s["dist"] = torch.zeros(n, device="cuda", dtype=torch.float32 if case["dtype"] == "f32" else torch.int32)
    elif kind == "pagerank":
        _set_format(A, case)
        s["ranks"] = torch.zeros(n, device="cuda")
    elif kind == "batch":
        src = _sources(ptr, case["bfs"] + case["ppr"] + case["sssp"], seed)
        nb, nbp = case["bfs"], case["bfs"] + case["ppr"]
        s["sources"] = [q if len(q) else src[:1] for q in (src[:nb], src[nb:nbp], src[nbp:])]
        s["levels"] = torch.zeros((len(s["sources"][0]), n), dtype=torch.int32, device="cuda")
        s["ranks"] = torch.zeros((len(s["sources"][1]), n), device="cuda")
        s["dist"] = torch.zeros((len(s["sources"][2]), n), dtype=torch.int32, device="cuda")
    return s


# ---- the calls -----------------------------------------------------------------

class _DeviceArray:
    """A device array of a matrix, for torch to view; holds the matrix as long as the view lives."""

    def __init__(self, owner, ptr, count, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (ptr, False), "version": 3}


def _views(M):
    p, i, v = M.arrays()
    if M.nnz == 0:
        return torch.as_tensor(_DeviceArray(M, p, M.n + 1, "<i4"), device="cuda"), None, None
    return (torch.as_tensor(_DeviceArray(M, p, M.n + 1, "<i4"), device="cuda"),
            torch.as_tensor(_DeviceArray(M, i, M.nnz, "<i4"), device="cuda"),
            torch.as_tensor(_DeviceArray(M, v, M.nnz, "<f4" if M.vtype == capi.F32 else "<i4"), device="cuda"))


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "mxv":
        # a masked step accumulates as a relaxation does (idempotent, so a pass can be repeated)
        accum = "min" if case["semiring"] == "min_plus" and case["masked"] else "second"
        return s["A"].mxv(s["x"], s["y"], semiring=case["semiring"], accum=accum, mask=s["mask"],
                          transpose=case["transpose"])
    if kind == "spmspv":
        mask = capi.dense_mask(s["mask"], "str_comp") if case["masked"] else None
        return s["A"].spmspv(s["ids"], s["vals"], s["y"], semiring=case["semiring"], mask=mask, transpose=True)
    if kind == "vector":
        n = case["n"]
        capi.assign_scalar(s["w"], 0.15 / n)
        capi.assign_vector("plus", capi.F32, s["w"], s["y"])
        capi.ewise("minus", capi.F32, s["diff"], s["r"], s["w"])
        capi.apply(0, "abs", capi.F32, s["diff"], s["diff"])
        change = capi.reduce("plus", capi.F32, s["diff"])
        capi.ewise("div", capi.F32, s["z"], s["w"], s["d"], mask=capi.dense_mask(s["m"]))
        capi.extract("second", capi.I32, s["gp"], s["f"], indices=s["f"])
        capi.ewise("ne", capi.I32, s["changed"], s["f"], s["gp"])
        moved = capi.nvals(s["changed"])
        ids, vals = capi.to_sparse(s["front"])
        return {"w": s["w"], "diff": s["diff"], "change": change, "z": s["z"], "gp": s["gp"], "changed": s["changed"],
                "moved": moved, "ids": ids, "vals": vals, "back": capi.to_dense(ids, vals, n)}
    if kind == "bfs":
        depth = s["A"].bfs(s["source"], s["levels"])
        return {"levels": s["levels"], "depth": depth}
    if kind == "sssp":
        s["A"].sssp(s["source"], s["dist"])
        return s["dist"]
    if kind == "pagerank":
        # a fixed number of iterations, as benchmarks run it: stopping on a float threshold could
        # take one iteration more or fewer for another correct rounding
        iters, _ = s["A"].pagerank(s["ranks"], itermax=case["itermax"], damping=DAMPING, tol=0.0)
        return {"ranks": s["ranks"], "iters": iters}
    if kind == "triangles":
        return s["A"].triangle_count()
    if kind == "mxm":
        return dict(zip(("ptr", "col", "val"), _views(s["A"].mxm(s["A"], semiring=case["semiring"]))))
    depths = s["A"].msbfs(s["sources"][0], s["levels"])
    s["A"].ppr(s["sources"][1], s["ranks"], damping=DAMPING, tol=0.0, itermax=case["itermax"])
    s["A"].sssp_multi(s["sources"][2], s["dist"])
    return {"depths": depths, "levels": s["levels"], "ranks": s["ranks"], "dist": s["dist"]}


# ---- what a pass cannot do without ----------------------------------------------

@functools.lru_cache(64)
def _mxm_counts(graph, n, ef, undirected):
    """(entries of A A, products) for the graph of seed 0."""
    ptr, rows, cols = _edges({"graph": graph, "n": n, "ef": ef, "undirected": undirected}, 0)
    a = torch.zeros((n, n), dtype=torch.bfloat16, device="cuda")
    a[rows, cols] = 1
    deg = ptr[1:] - ptr[:-1]
    return int(torch.count_nonzero(a @ a)), int(deg[cols].sum())


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "vector":
        k = int(n * case["fraction"])
        # per call: assign 4, += 12, minus 12, abs 8, reduce 4, masked divide 1 + half of 12, gather 12,
        # ne 9, count 1, to sparse 4, to dense 4 bytes an element; ids and values of the sparse form
        return {"bytes": 77 * n + 8 * k + 8 * k, "flops": 6 * n}
    nnz, fedges = _counts(case["graph"], n, case["ef"], case["undirected"], case.get("fraction", 0.0))
    csr = 4 * (n + 1) + 8 * nnz       # with values
    pattern = 4 * (n + 1) + 4 * nnz   # without
    if kind == "mxv":
        share = 0.33 if case["masked"] else 1.0  # rows outside the mask are not read
        matrix = pattern if case["semiring"] == "plus_second" else csr
        return {"bytes": share * matrix + 8 * n + (n if case["masked"] else 0), "flops": 2 * share * nnz}
    if kind == "spmspv":
        return {"bytes": 8 * fedges + 16 * int(n * case["fraction"]) + 4 * n + (5 * n if case["masked"] else 0),
                "flops": 2 * fedges}
    if kind == "bfs":
        return {"bytes": pattern + 4 * n, "flops": nnz}
    if kind == "sssp":
        return {"bytes": csr + 4 * n, "flops": 2 * nnz}
    if kind == "pagerank":
        return {"bytes": case["itermax"] * (pattern + 8 * n), "flops": 2 * case["itermax"] * nnz}
    if kind == "triangles":
        return {"bytes": pattern + 8, "flops": nnz}
    if kind == "mxm":
        out, products = _mxm_counts(case["graph"], n, case["ef"], case["undirected"])
        return {"bytes": csr + 4 * (n + 1) + 8 * out, "flops": 2 * products}
    lanes = case["ppr"]
    return {"bytes": pattern + 4 * n * case["bfs"] + case["itermax"] * (pattern + 8 * n * lanes) +
            csr + 4 * n * case["sssp"], "flops": 2 * case["itermax"] * nnz * lanes}


def tolerance(case):
    kind = case["kind"]
    if kind in ("bfs", "sssp", "triangles"):
        return "exact"  # levels, fixpoints of rounded sums (order-independent) and counts
    if case.get("dtype", "f32") == "i32" or case.get("semiring") in ("lor_land", "min_plus"):
        return "exact"  # whole numbers
    if kind == "vector":
        return {"rel": 1e-6, "max": 1e-5}  # single float operations; the sum is folded in double
    # 32-bit sums of up to some 10^5 positive terms; the staged formats fold a row's pieces in any
    # order: 3.3e-7 from the 64-bit sums, 4.2e-7 between two runs (R-MAT scale 22)
    return {"rel": 2e-6, "max": 4e-5}


# ---- 64-bit values ---------------------------------------------------------------

def _product(rows, cols, vals, x, n):
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, vals * x[cols])


def _exact_ppr(case, seed):
    n = case["n"]
    ptr, rows, cols = _edges(case, seed)
    src = _sources(ptr, case["bfs"] + case["ppr"] + case["sssp"], seed)
    seeds = src[case["bfs"]:case["bfs"] + case["ppr"]]
    seeds = torch.from_numpy((seeds if len(seeds) else src[:1]).astype(np.int64)).cuda()
    k = seeds.numel()
    coldeg = torch.bincount(cols, minlength=n)
    d = (coldeg.clamp(min=1).double() / DAMPING)[:, None]
    sinks = coldeg == 0
    lanes = torch.arange(k, device="cuda")
    r = torch.zeros((n, k), dtype=torch.float64, device="cuda")
    r[seeds, lanes] = 1.0
    step = 1 << 22
    for _ in range(case["itermax"]):
        w = r / d
        new = torch.zeros_like(r)
        for e in range(0, rows.numel(), step):
            new.index_add_(0, rows[e:e + step], w[cols[e:e + step]])
        new[seeds, lanes] += (1.0 - DAMPING) + DAMPING * r[sinks].sum(0)
        r = new
    return r.t().contiguous()


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("bfs", "sssp", "triangles") or case.get("dtype", "f32") == "i32" or case.get("semiring") == "lor_land":
        return None
    if kind == "vector":
        r, y, d, m, f, front = _vector_inputs(case, seed)
        w = float(np.float32(0.15 / n)) + y.double()
        w32 = w.float().double()  # each call stores its result in the vector's type
        diff = (r.double() - w32).abs()
        z = torch.where(m, w32 / d.double(), torch.zeros_like(w32))
        return {"w": w, "diff": diff, "change": float(diff.float().double().sum()), "z": z, "gp": None,
                "changed": None, "moved": None, "ids": None, "vals": front[front != 0].double(),
                "back": front.double()}
    if kind == "batch":
        return {"depths": None, "levels": None, "ranks": _exact_ppr(case, seed), "dist": None}
    ptr, rows, cols = _edges(case, seed)
    vals = _values(case, rows.numel(), seed).double()
    if kind == "mxv":
        if case["semiring"] == "plus_second":
            vals = torch.ones_like(vals)
        if case["transpose"]:
            rows, cols = cols, rows
        y = _product(rows, cols, vals, _dense(case, seed, 4).double(), n)
        return torch.where(_mask(case, seed, 0.33), y, torch.zeros_like(y)) if case["masked"] else y
    if kind == "spmspv":
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        x[_frontier(case, seed)] = 1.0
        y = _product(cols, rows, vals, x, n)
        return torch.where(_mask(case, seed, 0.2), torch.zeros_like(y), y) if case["masked"] else y
    if kind == "pagerank":
        coldeg = torch.bincount(cols, minlength=n)
        d = coldeg.double().clamp(min=1.0) / DAMPING
        sinks = coldeg == 0
        nsinks = int(sinks.sum())
        if nsinks <= int(0.3 * n):  # the reference reads a sparse sink vector at its list positions
            sinks = torch.arange(n, device="cuda") < nsinks
        r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        one = torch.ones(rows.numel(), dtype=torch.float64, device="cuda")
        for _ in range(case["itermax"]):
            r = (1.0 - DAMPING) / n + DAMPING / n * float(r[sinks].sum()) + _product(rows, cols, one, r / d, n)
        return {"ranks": r, "iters": None}
    # mxm, plus-times over positive values: every reached entry is kept
    a = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    a[rows, cols] = vals
    c = a @ a
    return {"ptr": None, "col": None, "val": c[c != 0]}
