"""The workloads whose speed this repository watches.

Every case is work that a program gives the library through its public entry
points: SpMV in CSR and SELL-C-sigma, the differentiable SpMV step, batched
and single SpMM, building a matrix from triplets, the clustered SpGEMM and
the top-k row similarities.  `listed()` names them with the sizes of the
benchmark configurations (bench.py) and the tests; `draw()` gives further
sizes, types and options of the same ranges.

A case is a dict of plain values.  `prepare(case, seed)` makes the inputs and
what a program keeps between calls (handles, plans, vectors).  Where the
pattern of the input sets the size of the result, the seed draws an order of
the rows and the values of one pattern per case.  `run(state)` is one pass, `work(case)` its least traffic and arithmetic, and
`exact(case, seed)` the same result from plain torch in 64 bits.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from sparseops_b200 import (Batch, COO_Matrix, CSR_Matrix, SpMM_csr, SpOps_csr, SpOps_sell_c_sigma, coo_to_csr,
                            convert_to, csr_to_sell_c_sigma, synth)
from sparseops_b200._lib import call
from sparseops_b200.autograd import SparsePattern, spmv
from sparseops_b200.spgemm import HashSpGEMMTopK, LeSpGEMM_lsh

DEV = "cuda"
FLOAT = {"f64": torch.float64, "f32": torch.float32}
INT = {"i32": torch.int32, "i64": torch.int64}
COL_MAJOR = 1


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one call of a small solver step, y = 0.8 A x + 0.7 y on a 20,000-row
        # matrix: launches and host work count, not bandwidth
        dict(name="csr_small_20k", kind="csr", matrix="powerlaw", n=20000, value="f64", index="i32", alpha=0.8,
             beta=0.7),
        # the 512 x 512 grid's 5-point Laplacian, repeated as an iterative
        # solver does: resident in L2, short equal rows
        dict(name="csr_laplacian_512", kind="csr", matrix="laplacian", n=512 * 512, value="f64", index="i32",
             alpha=1.0, beta=0.0),
        # the full power-law benchmark matrix (103.5M entries, 1.26 GB)
        dict(name="csr_powerlaw_4m", kind="csr", matrix="powerlaw", n=4194304, value="f64", index="i32", alpha=1.0,
             beta=0.0),
        # single precision with 64-bit indices and a ragged row count
        dict(name="csr_f32_i64_1m", kind="csr", matrix="powerlaw", n=1000003, value="f32", index="i64", alpha=1.0,
             beta=1.0),
        # SELL-C-sigma (C = 32, sigma = 512), the format benchmark's parameters
        dict(name="sell_c_sigma_1m", kind="sell", matrix="powerlaw", n=1048576, value="f64", index="i32",
             chunk=32, sigma=512),
        # a training step of the sparse layer: y = A(v) x, then the gradients
        # of v and x, on the 1M-node graph (33.5M entries)
        dict(name="adjoint_graph_1m", kind="adjoint", n=1048576, degree=32.0, value="f64"),
        # 256 matrices of 1k to 200k rows with 32 right-hand sides in one launch
        dict(name="batch_256_k32", kind="batch", count=256, nmin=1000, nmax=200000, k=32, value="f64"),
        # one matrix times a block of 12 vectors (a block solver's odd width)
        dict(name="spmm_k12_300k", kind="spmm", matrix="powerlaw", n=300007, k=12, value="f64", index="i32"),
        # triplets in arrival order with repeated entries to a summed CSR and
        # its SELL-C-sigma form: what comes before the first SpMV
        dict(name="assemble_400k", kind="assemble", n=400000, mean=16.0, value="f64", index="i32", chunk=32,
             sigma=512),
        # MinHash-LSH clustering and the clustered SpGEMM A A^T on the planted
        # communities (C has 1.2e8 entries)
        dict(name="lsh_planted_512k", kind="lsh", matrix="planted", n=524288, value="f64"),
        # the same pipeline on near-duplicate rows: multi-row dense clusters,
        # and clustering itself the longest stage
        dict(name="lsh_grouped_512k", kind="lsh", matrix="grouped", n=524288, value="f64"),
        # the 16 most similar rows of every row
        dict(name="topk_planted_128k", kind="topk", n=131072, k=16, value="f64"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["csr", "csr", "sell", "adjoint", "batch", "spmm", "assemble", "lsh", "lsh", "topk"])
    value = rng.choice(["f64", "f64", "f32"])
    index = rng.choice(["i32", "i32", "i64"])
    if kind == "csr":
        matrix = rng.choice(["powerlaw", "laplacian", "banded"])
        n = _log_uniform(rng, 1000, 3000000)
        if matrix == "laplacian":
            n = max(16, math.isqrt(n)) ** 2
        return dict(kind=kind, matrix=matrix, n=n, value=value, index=index, alpha=rng.choice([1.0, 0.8]),
                    beta=rng.choice([0.0, 1.0, 0.7]))
    if kind == "sell":
        return dict(kind=kind, matrix=rng.choice(["powerlaw", "banded"]), n=_log_uniform(rng, 5000, 2000000),
                    value=value, index="i32", chunk=32, sigma=rng.choice([256, 512, 4096, 16384]))
    if kind == "adjoint":
        return dict(kind=kind, n=_log_uniform(rng, 20000, 1048576), degree=round(rng.uniform(8.0, 32.0), 1),
                    value=value)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(24, 160), nmin=1000, nmax=_log_uniform(rng, 20000, 200000),
                    k=rng.choice([1, 1, 8, 8, 16, 32]), value="f64")
    if kind == "spmm":
        return dict(kind=kind, matrix=rng.choice(["powerlaw", "banded"]), n=_log_uniform(rng, 10000, 1000000),
                    k=rng.choice([2, 4, 5, 8, 12, 16, 24, 32]), value=value, index=index)
    if kind == "assemble":
        return dict(kind=kind, n=_log_uniform(rng, 10000, 800000), mean=round(rng.uniform(5.0, 20.0), 1),
                    value=value, index=index, chunk=32, sigma=rng.choice([256, 512, 4096]))
    if kind == "lsh":
        return dict(kind=kind, matrix=rng.choice(["planted", "grouped"]),
                    n=256 * _log_uniform(rng, 32, 1500) + rng.choice([0, 0, 1, 77]), value="f64")
    return dict(kind=kind, n=256 * _log_uniform(rng, 16, 800) + rng.choice([0, 0, 3, 91]),
                k=rng.choice([4, 8, 10, 16, 20, 32]), value="f64")


# ------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 11)


def _uniform(shape, seed, dtype):
    return (torch.rand(shape, generator=_gen(seed), device=DEV, dtype=torch.float64) * 2 - 1).to(dtype)


def _rows_in_order(rp, ci, v, order):
    """The rows of a CSR matrix listed in another order."""
    lens = torch.diff(rp)[order]
    out = torch.zeros_like(rp)
    out[1:] = torch.cumsum(lens, 0)
    at = torch.arange(len(ci), device=DEV) + torch.repeat_interleave(rp[:-1][order] - out[:-1], lens)
    return out, ci[at], v[at]


def _csr_arrays(case, seed):
    """(row_offset, col_index, values) on the device and the column count."""
    kind, n = case["matrix"], case["n"]
    ncols = n
    if kind == "powerlaw":
        rp, ci, v = synth.powerlaw(n, hi=min(20000, n // 4), seed=seed + 1)
    elif kind == "laplacian":
        rp, ci, v = synth.laplacian_2d(math.isqrt(n))
        v = v * (1.0 + 0.125 * synth.uniform(len(v), seed + 1))  # a variable coefficient
    elif kind == "banded":
        rp, ci, v = synth.banded_random(n, 16.0, 64, seed=seed + 1)
    elif kind == "planted":
        rp, ci, v = synth.planted_communities(n, ncomm=max(1, n // 256), mean=20.0, seed=5)
    else:
        rp, ci, v, ncols = synth.grouped_rows(n - n % 32, seed=8)
    if kind in ("planted", "grouped"):  # whole groups of near-duplicate rows stay together
        rp, ci, g = torch.from_numpy(rp).to(DEV), torch.from_numpy(ci).to(DEV), _gen(seed)
        size = 32 if kind == "grouped" else 1
        blocks = torch.randperm((len(rp) - 1) // size, generator=g, device=DEV)
        order = (blocks[:, None] * size + torch.arange(size, device=DEV)).reshape(-1)
        v = torch.randn(len(ci), generator=g, device=DEV, dtype=torch.float64)
        return _rows_in_order(rp, ci, v.to(FLOAT[case["value"]]), order) + (ncols,)
    it = INT[case.get("index", "i64")]
    return (torch.from_numpy(rp).to(DEV).to(it), torch.from_numpy(ci).to(DEV).to(it),
            torch.from_numpy(v).to(DEV).to(FLOAT[case["value"]]), ncols)


def _transposed(rp, ci, v, ncols):
    """CSR of the transpose, each row's columns ascending."""
    rows = torch.repeat_interleave(torch.arange(len(rp) - 1, device=DEV, dtype=ci.dtype), torch.diff(rp))
    order = torch.sort(ci, stable=True)[1]
    trp = torch.zeros(ncols + 1, dtype=rp.dtype, device=DEV)
    trp[1:] = torch.cumsum(torch.bincount(ci, minlength=ncols), 0)
    return trp, rows[order], v[order]


def _graph(case, seed):
    """Random graph with a symmetric pattern, degree lognormal (sigma = 1)
    with the given mean, values U[0.1, 1]."""
    n, g = case["n"], _gen(4)
    mu = math.log(case["degree"]) - 0.5
    half = torch.exp(torch.randn(n, generator=g, device=DEV, dtype=torch.float64) + mu) / 2
    cnt = torch.clamp(torch.round(half), 1, n // 4).long()
    src = torch.repeat_interleave(torch.arange(n, device=DEV), cnt)
    dst = torch.randint(n, (len(src),), generator=g, device=DEV)
    g = _gen(seed)
    name = torch.randperm(n, generator=g, device=DEV)
    src, dst = name[src], name[dst]
    key = torch.unique(torch.cat([src * n + dst, dst * n + src]))
    rows, cols = key // n, key % n
    rp = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    v = torch.rand(len(cols), generator=g, device=DEV, dtype=torch.float64) * 0.9 + 0.1
    return rp, cols.to(torch.int32), v.to(FLOAT[case["value"]])


def _batch_arrays(case, seed):
    """[(row_offset, col_index, values)] of banded-plus-random matrices, sizes
    log-uniform in [nmin, nmax].  The sizes are the case's, the patterns and
    values the seed's."""
    r = np.random.default_rng(case["count"])
    ns = np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["count"])).astype(np.int64)
    out = []
    for m, n in enumerate(ns):
        rp, ci, v = synth.banded_random(int(n), 16.0, 64, seed=seed * 1000 + m)
        out.append(tuple(torch.from_numpy(a).to(DEV) for a in (rp, ci, v)))
    return ns, out


def _triplets(case, seed):
    """Entries of a banded-plus-random matrix in arrival order, an eighth of
    them given twice."""
    n, g = case["n"], _gen(seed)
    rp, ci, v = synth.banded_random(n, case["mean"], 64, seed=3)
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), torch.diff(torch.from_numpy(rp).to(DEV).long()))
    cols = torch.from_numpy(ci).to(DEV).long()
    vals = torch.randn(len(cols), generator=g, device=DEV, dtype=torch.float64)
    twice = torch.randperm(len(cols), generator=g, device=DEV)[:len(cols) // 8]
    more = torch.randn(len(twice), generator=g, device=DEV, dtype=torch.float64)
    rows, cols, vals = torch.cat([rows, rows[twice]]), torch.cat([cols, cols[twice]]), torch.cat([vals, more])
    order = torch.randperm(len(cols), generator=g, device=DEV)
    it = INT[case["index"]]
    return rows[order].to(it), cols[order].to(it), vals[order].to(FLOAT[case["value"]])


def _csr(arrays, n, ncols):
    return CSR_Matrix(n, ncols, *arrays[:3])


def prepare(case, seed):
    kind, dt = case["kind"], FLOAT[case["value"]]
    s = dict(case=case)
    if kind in ("csr", "sell", "spmm"):
        rp, ci, v, ncols = _csr_arrays(case, seed)
        n, k = len(rp) - 1, case.get("k", 0)
        A = _csr((rp, ci, v), n, ncols)
        A.device()
        s["x"] = _uniform((ncols, k) if k else ncols, seed + 2, dt)
        s["y"] = _uniform((n, k) if k else n, seed + 3, dt)
        s["A"] = csr_to_sell_c_sigma(A, slicewidth=case["sigma"], chunkwidth=case["chunk"],
                                     layout=COL_MAJOR) if kind == "sell" else A
    elif kind == "adjoint":
        rp, ci, v = _graph(case, seed)
        n = case["n"]
        s["pattern"] = SparsePattern(n, n, rp, ci, v)
        s["v"] = v.clone().requires_grad_(True)
        s["x"] = _uniform(n, seed + 2, dt).requires_grad_(True)
        s["g"] = torch.randn(n, generator=_gen(seed + 3), device=DEV, dtype=torch.float64).to(dt)
    elif kind == "batch":
        ns, arrays = _batch_arrays(case, seed)
        k, total = case["k"], int(ns.sum())
        s["X"] = _uniform((total, k), seed + 2, dt)
        s["Y"] = torch.zeros((total, k), dtype=dt, device=DEV)
        at = np.concatenate([[0], np.cumsum(ns)])
        part = [slice(int(a), int(b)) for a, b in zip(at[:-1], at[1:])]
        s["batch"] = Batch([_csr(a, int(n), int(n)) for a, n in zip(arrays, ns)], k=k)
        one = (lambda t: t.reshape(-1)) if k == 1 else (lambda t: t)
        s["batch"].set_vectors([one(s["X"][p]) for p in part], [one(s["Y"][p]) for p in part])
        s["batch"].tune()
        s["batch"].capture(1.0, 0.0)
    elif kind == "assemble":
        s["coo"] = _triplets(case, seed)
    else:
        c = dict(case, matrix=case.get("matrix", "planted"), index="i64")
        rp, ci, v, ncols = _csr_arrays(c, seed)
        s["A"] = _csr((rp, ci, v), len(rp) - 1, ncols)
        s["A"].device()
        if kind == "lsh":
            s["B"] = _csr(_transposed(rp, ci, v, ncols), ncols, len(rp) - 1)
            s["B"].device()
    return s


# --------------------------------------------------------------------- runs
class _DeviceArray:
    """One array of a matrix handle as torch sees it (no copy); keeps its
    owner alive."""

    _TYPES = {(4, "i"): "<i4", (8, "i"): "<i8", (4, "f"): "<f4", (8, "f"): "<f8"}

    def __init__(self, owner, which, kind):
        p, n, eb = ctypes.c_void_p(), ctypes.c_int64(), ctypes.c_int32()
        call("spops_matrix_array", owner.device().handle, which, ctypes.byref(p), ctypes.byref(n), ctypes.byref(eb))
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n.value,), "typestr": self._TYPES[(eb.value, kind)],
                                         "data": (p.value or 0, False), "version": 2}


def _array(owner, which, kind):
    return torch.as_tensor(_DeviceArray(owner, which, kind), device=DEV)


def _csr_out(C):
    return {"row_offset": _array(C, 0, "i"), "col_index": _array(C, 1, "i"), "values": _array(C, 2, "f")}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "csr":  # with beta, y goes on from the last pass as a solver's does
        return SpOps_csr(case["alpha"], s["A"], s["x"], case["beta"], s["y"])
    if kind == "sell":
        return SpOps_sell_c_sigma(1.0, s["A"], s["x"], 0.0, s["y"])
    if kind == "spmm":
        return SpMM_csr(1.0, s["A"], s["x"], 0.0, s["y"])
    if kind == "adjoint":
        y = spmv(s["v"], s["x"], s["pattern"])
        grad_v, grad_x = torch.autograd.grad(y, (s["v"], s["x"]), s["g"])
        return {"y": y.detach(), "grad_v": grad_v, "grad_x": grad_x}
    if kind == "batch":
        s["batch"].run()
        return s["Y"]
    if kind == "assemble":
        coo = COO_Matrix(case["n"], case["n"], *s["coo"])
        A = coo_to_csr(coo, compact=True)
        S = convert_to(A, "sell_c_sigma", sigma=case["sigma"], chunk=case["chunk"], layout=COL_MAJOR)
        out = _csr_out(A)
        out["sell"] = {"reorder": _array(S, 3, "i"), "chunk_len": _array(S, 4, "i"), "col": _array(S, 1, "i"),
                       "val": _array(S, 2, "f")}
        return out
    if kind == "lsh":
        return _csr_out(LeSpGEMM_lsh(s["A"], s["B"], 64, 16, 7, 8))
    return _csr_out(HashSpGEMMTopK(s["A"], case["k"]))


# --------------------------------------------------------------------- work
def _per_row(case):
    """Entries per row, as the generators give them."""
    m = case.get("matrix", {"adjoint": "graph", "assemble": "triplets"}.get(case["kind"], "planted"))
    return {"powerlaw": 24.69, "laplacian": 4.99, "banded": 16.0, "planted": 19.03, "grouped": 6.2,
            "graph": case.get("degree", 32.0), "triplets": case.get("mean", 16.0)}[m]


def work(case):
    kind = case["kind"]
    vs = 8 if case["value"] == "f64" else 4
    isz = 4 if case.get("index", "i32") == "i32" else 8
    if kind == "batch":
        r = np.random.default_rng(case["count"])
        ns = np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["count"])).astype(np.int64)
        n, k, nnz = int(ns.sum()), case["k"], 16.0 * int(ns.sum())
        return {"bytes": 4 * n + (4 + vs) * nnz + 2 * vs * k * n, "flops": 2 * k * nnz}
    n = case["n"]
    nnz = n * _per_row(case)
    if kind in ("csr", "sell", "spmm"):
        k = case.get("k", 1)
        ys = 2 if case.get("beta") else 1
        return {"bytes": isz * (n + 1) + (isz + vs) * nnz + vs * k * n * (1 + ys), "flops": 2 * k * nnz}
    if kind == "adjoint":
        # the pattern read once a direction, the values twice, grad_v written
        return {"bytes": 2 * 4 * (n + 1) + 2 * (4 + vs) * nnz + vs * nnz + 5 * vs * n, "flops": 5 * nnz}
    if kind == "assemble":
        # triplets in, CSR and SELL out
        return {"bytes": nnz * (1.125 * (2 * isz + vs) + 2 * (isz + vs)) + 2 * isz * n, "flops": nnz / 8}
    # 64-bit indices; products and entries of A A^T per row, as measured on
    # the benchmark sizes
    products, entries = {"planted": (381.0, 230.0), "grouped": (105.7, 32.6)}[case.get("matrix", "planted")]
    if kind == "lsh":
        return {"bytes": 2 * (8 + vs) * nnz + 3 * 8 * n + (8 + vs) * entries * n, "flops": 2 * products * n}
    return {"bytes": 8 * nnz + 8 * n + n * (8 + (8 + vs) * case["k"]), "flops": 2 * products * n}


# -------------------------------------------------------------------- exact
def _times(rp, ci, v, X):
    """A X in 64 bits; X [cols] or [cols x k]."""
    X = X.double()
    A = torch.sparse_csr_tensor(rp.long(), ci.long(), v.double(), (len(rp) - 1, X.shape[0]))
    return (A @ X.reshape(X.shape[0], -1)).reshape((len(rp) - 1,) + X.shape[1:])


def _products(rp, ci, v, trp, tci, tv, lo, hi, ncols):
    """Rows lo..hi of A B: (keys row * ncols + col ascending, sums)."""
    a, b = int(rp[lo]), int(rp[hi])
    rows = torch.repeat_interleave(torch.arange(lo, hi, device=DEV), torch.diff(rp[lo:hi + 1]))
    c = ci[a:b]
    cnt = trp[c + 1] - trp[c]
    first = torch.cumsum(cnt, 0) - cnt
    src = torch.repeat_interleave(torch.arange(b - a, device=DEV), cnt)
    at = trp[c][src] + torch.arange(len(src), device=DEV) - first[src]
    key, order = torch.sort(rows[src] * ncols + tci[at], stable=True)
    key, where = torch.unique_consecutive(key, return_inverse=True)
    prod = (v[a:b][src] * tv[at])[order]
    return key, torch.zeros(len(key), dtype=torch.float64, device=DEV).index_add_(0, where, prod)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("csr", "sell", "spmm"):
        rp, ci, v, ncols = _csr_arrays(case, seed)
        n, k, dt = len(rp) - 1, case.get("k", 0), FLOAT[case["value"]]
        y = case.get("alpha", 1.0) * _times(rp, ci, v, _uniform((ncols, k) if k else ncols, seed + 2, dt))
        if case.get("beta"):
            y += case["beta"] * _uniform(n, seed + 3, dt).double()
        return y
    if kind == "adjoint":
        rp, ci, v = _graph(case, seed)
        n, dt = case["n"], FLOAT[case["value"]]
        x = _uniform(n, seed + 2, dt).double()
        g = torch.randn(n, generator=_gen(seed + 3), device=DEV, dtype=torch.float64).to(dt).double()
        rows = torch.repeat_interleave(torch.arange(n, device=DEV), torch.diff(rp.long()))
        gx = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, ci.long(), v.double() * g[rows])
        return {"y": _times(rp, ci, v, x), "grad_v": g[rows] * x[ci.long()], "grad_x": gx}
    if kind == "batch":
        ns, arrays = _batch_arrays(case, seed)
        X = _uniform((int(ns.sum()), case["k"]), seed + 2, FLOAT[case["value"]])
        return torch.cat([_times(*a, x) for a, x in zip(arrays, torch.split(X, [int(n) for n in ns]))])
    if kind == "assemble":
        r, c, v = _triplets(case, seed)
        key, order = torch.sort(r.long() * case["n"] + c.long(), stable=True)
        key, where, cnt = torch.unique_consecutive(key, return_inverse=True, return_counts=True)
        sums = torch.zeros(len(key), dtype=torch.float64, device=DEV).index_add_(0, where, v.double()[order])
        first = order[torch.cumsum(cnt, 0) - cnt]  # stable: the earliest of each entry
        by = torch.sort(first, descending=True)[1]
        by = by[torch.sort(key[by] // case["n"], stable=True)[1]]
        return {"row_offset": None, "col_index": None, "values": sums[by],
                "sell": {"reorder": None, "chunk_len": None, "col": None, "val": None}}
    c = dict(case, matrix=case.get("matrix", "planted"), index="i64")
    rp, ci, v, ncols = _csr_arrays(c, seed)
    n = len(rp) - 1
    v = v.double() if kind == "lsh" else torch.ones(len(ci), dtype=torch.float64, device=DEV)
    trp, tci, tv = _transposed(rp, ci, v, ncols)
    step, values, lens = 65536, [], torch.diff(rp).double()
    for lo in range(0, n, step):
        key, sums = _products(rp, ci, v, trp, tci, tv, lo, min(n, lo + step), n)
        if kind == "topk":  # Jaccard similarity of two rows' patterns, the row itself left out
            i, j = key // n, key % n
            i, j, sums = i[i != j], j[i != j], sums[i != j]
            sim = sums / (lens[i] + lens[j] - sums)
            by = torch.sort(sim, descending=True, stable=True)[1]
            by = by[torch.sort(i[by], stable=True)[1]]
            i = i[by]
            rank = torch.arange(len(i), device=DEV) - torch.searchsorted(i, i)
            sums = sim[by][rank < case["k"]]
        values.append(sums)
    return {"row_offset": None, "col_index": None, "values": torch.cat(values)}
