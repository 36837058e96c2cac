"""The measured workloads of the framework, each through its public entry points.

A case is a dict of plain values; ``kind`` says which entry point it goes
through and the other fields give sizes, method and k:

* ``dense_query`` / ``dense_self``: new query embeddings against a resident
  dense reference (``sdg_dense_knn_query``), or a block of query columns of
  the reference's own self-search (``sdg_dense_knn_block``).
* ``resident_block``: a block of query columns of the self-search of a
  resident single-cell log-count matrix (``sdg_knn_block``).
* ``knn``: ``sparseKNN`` on a host matrix, result on the host.
* ``cross``: ``sparseKNNCross`` on two host matrices, both directions.
* ``batch``: several uneven independent ``sparseKNNCross`` problems in one
  call (``knn_cross_batch``).
* ``snn``: ``sparseSNN`` of a kNN index matrix, the graph on the host.
* ``dist``: ``sparseDist`` of one host matrix (both triangles).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import sparsedist_gb300 as sdg
from sparsedist_gb300 import _lib, synth

CODES = {"binary": 0, "cosine": 1, "euclidean": 2, "manhattan": 3, "pearson": 4, "js": 5}
ROWS = 30000            # genes of the log-count matrices
MEAN_NNZ = 1800.0       # stored entries drawn per log-count column (about 1,540 stay after zero counts drop)
MATCH = 700.0           # rows two log-count columns share, on average


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one interactive lookup in a large embedding index: latency
        {"name": "dense-1x2000000", "kind": "dense_query", "d": 256, "n": 2000000, "nq": 1, "k": 10,
         "method": "cosine"},
        # a ragged group of requests, rows not a multiple of 64, euclidean
        {"name": "dense-777x150001", "kind": "dense_query", "d": 100, "n": 150001, "nq": 777, "k": 15,
         "method": "euclidean"},
        # the neighbour graph of a mid-sized embedding, one block of its columns
        {"name": "dense-self-3000x60000", "kind": "dense_self", "d": 64, "n": 60000, "nq": 3000, "k": 30,
         "method": "cosine"},
        # the benchmark's own step: a full block against two million columns
        {"name": "dense-4096x2000000", "kind": "dense_query", "d": 256, "n": 2000000, "nq": 4096, "k": 20,
         "method": "cosine"},
        # one block of a single-cell kNN graph, cosine on log counts
        {"name": "logcount-cosine-4096", "kind": "resident_block", "n": 30000, "nq": 4096, "k": 20,
         "method": "cosine"},
        # one plate of cells looked up in an atlas
        {"name": "logcount-euclidean-128", "kind": "resident_block", "n": 30000, "nq": 128, "k": 10,
         "method": "euclidean"},
        # a method without an inner product form, on the same kind of data
        {"name": "logcount-manhattan-1000", "kind": "resident_block", "n": 20000, "nq": 1000, "k": 15,
         "method": "manhattan"},
        # the reference's own bench shape: a small matrix, everything from and to the host
        {"name": "knn-binary-2000x10000", "kind": "knn", "rows": 2000, "n": 10000, "density": 0.02, "k": 15,
         "method": "binary"},
        # the smallest call: a toy matrix, where launches and copies count
        {"name": "knn-cosine-1000x301", "kind": "knn", "rows": 1000, "n": 301, "density": 0.05, "k": 10,
         "method": "cosine"},
        # label transfer between two data sets, both directions
        {"name": "cross-manhattan", "kind": "cross", "rows": 12000, "nq": 1500, "nr": 12001, "density": 0.01, "k": 20,
         "method": "manhattan"},
        # many uneven problems in one call, binary / cosine / manhattan in turn
        {"name": "batch-8", "kind": "batch", "problems": 8, "mix": 4, "scale": 0.05},
        # the graph step that follows a kNN search
        {"name": "snn-200000x20", "kind": "snn", "n": 200000, "k": 20, "prune": 1.0 / 15.0},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "dense", "resident_block", "resident_block", "knn", "knn", "cross", "cross",
                       "batch", "snn", "dist"])
    k = rng.choice([5, 10, 15, 20, 30, 50])
    if kind == "dense":
        n = _logint(rng, 10000, 2000000)
        return {"kind": rng.choice(["dense_query", "dense_self"]), "d": _logint(rng, 32, 256), "n": n,
                "nq": _logint(rng, 1, 4096), "k": k, "method": rng.choice(["cosine", "euclidean"])}
    if kind == "resident_block":
        method = rng.choice(["binary", "cosine", "euclidean", "manhattan", "pearson", "js"])
        inner = method in ("binary", "cosine", "euclidean")
        return {"kind": kind, "n": _logint(rng, 5000, 30000 if inner else 20000),
                "nq": _logint(rng, 16, 4096 if inner else 1000), "k": k, "method": method}
    if kind == "knn":
        return {"kind": kind, "rows": _logint(rng, 500, 5000), "n": _logint(rng, 200, 12000),
                "density": round(math.exp(rng.uniform(math.log(0.005), math.log(0.05))), 5), "k": k,
                "method": rng.choice(["binary", "cosine", "euclidean", "manhattan"])}
    if kind == "cross":
        return {"kind": kind, "rows": _logint(rng, 5000, 20000), "nq": _logint(rng, 200, 1500),
                "nr": _logint(rng, 2000, 12000),
                "density": round(math.exp(rng.uniform(math.log(0.003), math.log(0.02))), 5), "k": k,
                "method": rng.choice(["binary", "cosine", "manhattan", "js"])}
    if kind == "batch":
        return {"kind": kind, "problems": rng.randint(3, 8), "mix": rng.randrange(1000),
                "scale": round(rng.uniform(0.02, 0.05), 4)}
    if kind == "snn":
        return {"kind": kind, "n": _logint(rng, 5000, 200000), "k": rng.randint(10, 20),
                "prune": rng.choice([0.0, 1.0 / 15.0, 0.1])}
    return {"kind": "dist", "rows": _logint(rng, 1000, 4000), "n": _logint(rng, 200, 3000),
            "density": round(math.exp(rng.uniform(math.log(0.01), math.log(0.05))), 5),
            "method": rng.choice(["binary", "cosine", "euclidean", "manhattan"])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
class _Dense:
    """A resident dense reference (sdg_dense_upload), freed with its state."""

    def __init__(self, ctx, X):
        self.ctx = ctx
        self.h = C.c_void_p()
        _lib.check(ctx.lib.sdg_dense_upload(ctx.handle, X.data_ptr(), X.shape[1], X.shape[0], C.byref(self.h)))

    def __del__(self):
        try:
            self.ctx.lib.sdg_dense_free(self.h)
        except Exception:
            pass


def _embeddings(case, seed):
    """(reference n x d, queries nq x d or None): half of the columns around
    cluster centres, 1 % near duplicates; queries from the same clusters."""
    self_search = case["kind"] == "dense_self"
    n, nq = case["n"], 0 if self_search else case["nq"]
    X = synth.dense_embeddings(d=case["d"], n=n + nq, centres=max(16, n // 2000), seed=seed)
    return (X, None) if self_search else (X[:n], X[n:].contiguous())


def _matrix(case, n, seed, other=1):
    """(X, Y): host CSC matrices of n and `other` columns, a uniform pattern, |N(0, 1)| values (js: columns sum to 1)."""
    return synth.cross_problem({"nq": n, "nr": other, "rows": case["rows"], "density": case["density"],
                                "method": case["method"], "seed": seed})


def _specs(case, seed):
    # js is left to the other kinds: its values agree between engines to rounding only, and a batched call picks
    # the engine from measured times
    out = [sp for sp in synth.cross_draw(n=2 * case["problems"], seed=case["mix"], scale=case["scale"])
           if sp["method"] != "js"][:case["problems"]]
    for j, sp in enumerate(out):
        sp["k"] = max(1, min(sp["k"], sp["nq"] // 2, sp["nr"] // 2))
        sp["seed"] = int(seed) * 1009 + j
    return out


def _neighbours(case, seed):
    """n x k 1-based kNN indices: k distinct members of a window of 3 k columns around each column, the same graph for
    every seed up to the numbering of its nodes (so that the SNN graph has as many entries)."""
    n, k = case["n"], case["k"]
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    off = torch.rand(n, 3 * k, generator=g, device="cuda").argsort(dim=1)[:, :k]
    off = torch.where(off >= (3 * k) // 2, off + 1, off) - (3 * k) // 2
    idx = (torch.arange(n, device="cuda")[:, None] + off) % n
    g.manual_seed(int(seed))
    number = torch.randperm(n, generator=g, device="cuda")
    out = torch.empty_like(idx)
    out[number] = number[idx]
    return (out + 1).to(torch.int32)


def _logcounts(case, seed):
    return synth.logcount_csc(ROWS, case["n"], mean_nnz=MEAN_NNZ, seed=seed, keep_on_device=True)


def _nq(case):
    return min(case["nq"], case["n"])


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("dense_query", "dense_self", "resident_block"):
        st["ctx"] = _lib.default_context()
        if kind == "resident_block":
            p, i, x = _logcounts(case, seed)
            torch.cuda.synchronize()
            st["ref"] = _lib.Resident.from_device(st["ctx"], ROWS, case["n"], p, i, x)
        else:
            X, st["q"] = _embeddings(case, seed)
            torch.cuda.synchronize()
            st["ref"] = _Dense(st["ctx"], X)
        nq = _nq(case)
        st["idx"] = torch.empty(case["k"], nq, dtype=torch.int32, device="cuda")
        st["dist"] = torch.empty(case["k"], nq, dtype=torch.float64, device="cuda")
    elif kind in ("knn", "dist"):
        st["X"] = _matrix(case, case["n"], seed)[0]
    elif kind == "cross":
        st["X"], st["Y"] = _matrix(case, case["nq"], seed, case["nr"])
    elif kind == "batch":
        st["ctx"] = _lib.default_context()
        st["problems"] = []
        for sp in _specs(case, seed):
            X, Y = synth.cross_problem(sp)
            st["problems"].append((X, Y, CODES[sp["method"]], True, sp["k"]))
    else:
        st["idx"] = np.asfortranarray(_neighbours(case, seed).cpu().numpy())
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("dense_query", "dense_self", "resident_block"):
        ctx, k, nq, m = st["ctx"], case["k"], _nq(case), CODES[case["method"]]
        ke, fl = C.c_int(), C.c_int()
        oi, od = st["idx"].data_ptr(), st["dist"].data_ptr()
        if kind == "dense_query":
            rc = ctx.lib.sdg_dense_knn_query(ctx.handle, st["ref"].h, st["q"].data_ptr(), case["d"], nq, m, k, 0, oi,
                                             od, 1, C.byref(ke), C.byref(fl))
        elif kind == "dense_self":
            rc = ctx.lib.sdg_dense_knn_block(ctx.handle, st["ref"].h, (case["n"] - nq) // 3, nq, m, k, 0, oi, od, 1,
                                             C.byref(ke), C.byref(fl))
        else:
            rc = ctx.lib.sdg_knn_block(ctx.handle, st["ref"].handle, None, (case["n"] - nq) // 3, nq, m, 1, k, 0, 1,
                                       oi, od, 1, C.byref(ke), C.byref(fl))
        _lib.check(rc)
        return {"idx": st["idx"], "dist": st["dist"]}
    if kind == "knn":
        r = sdg.sparseKNN(st["X"], k=case["k"], method=case["method"], verbose=False)
        return {"idx": r.idx, "dist": r.dist}
    if kind == "cross":
        r = sdg.sparseKNNCross(st["X"], st["Y"], k=case["k"], method=case["method"], verbose=False)
        return {s: {"idx": r[s].idx, "dist": r[s].dist} for s in ("forward", "reverse")}
    if kind == "batch":
        rc, res = _lib.knn_cross_batch(st["ctx"], st["problems"])
        _lib.check(rc)
        return [{s: {"idx": r[s][0], "dist": r[s][1]} for s in ("forward", "reverse")} for r in res]
    if kind == "dist":
        return sdg.sparseDist(st["X"], method=case["method"], full=True, verbose=False)
    g = sdg.sparseSNN(st["idx"], prune=case["prune"], verbose=False)
    return {"p": g.indptr, "i": g.indices, "x": g.data}


# ---------------------------------------------------------------------------
# what a pass cannot do without: inputs read once and results written once;
# a multiply and an add for every row that two columns share
# ---------------------------------------------------------------------------
def _cross_work(rows, density, nq, nr, k):
    """One host sparseKNNCross / self-search: CSC in, idx and distances out."""
    nnz = density * rows
    return 12.0 * nnz * (nq + nr) + 12.0 * k * (nq + nr), 2.0 * density * nnz * nq * nr


def work(case):
    kind = case["kind"]
    if kind in ("dense_query", "dense_self"):
        # the reference at the screen's 16 bits a value
        nq = _nq(case)
        return {"bytes": 2.0 * case["d"] * (case["n"] + nq) + 12.0 * nq * case["k"],
                "flops": 2.0 * case["d"] * case["n"] * nq}
    if kind == "resident_block":
        nq = _nq(case)
        return {"bytes": 8.0 * 0.85 * MEAN_NNZ * case["n"] + 12.0 * nq * case["k"],
                "flops": 2.0 * MATCH * case["n"] * nq}
    if kind == "knn":
        b, f = _cross_work(case["rows"], case["density"], case["n"], 0, case["k"])
        return {"bytes": b, "flops": 2.0 * case["density"] ** 2 * case["rows"] * case["n"] ** 2}
    if kind == "cross":
        b, f = _cross_work(case["rows"], case["density"], case["nq"], case["nr"], case["k"])
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0.0
        for sp in _specs(case, 0):
            x, y = _cross_work(sp["rows"], sp["density"], sp["nq"], sp["nr"], sp["k"])
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if kind == "dist":
        n = case["n"]
        return {"bytes": 12.0 * case["density"] * case["rows"] * n + 8.0 * n * n,
                "flops": case["density"] ** 2 * case["rows"] * n * n}
    # the index matrix in, about 1.4 n k graph entries of 12 bytes out
    n, k = case["n"], case["k"]
    return {"bytes": 4.0 * n * k + 12.0 * 1.4 * n * k, "flops": 2.0 * n * k * (k + 1)}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _columns(M):
    """A scipy CSC matrix as a dense (ncol, nrow) float64 tensor."""
    return torch.from_numpy(np.ascontiguousarray(M.toarray().T)).to("cuda")


def _distances(method, X, Y):
    """All distances between the rows of X (nq x rows) and of Y (nr x rows)."""
    if method == "binary":
        A, B = (X != 0).double(), (Y != 0).double()
        both = A @ B.T
        return 1.0 - both / (A.sum(1)[:, None] + B.sum(1)[None, :] - both)
    if method == "cosine":
        return 1.0 - ((X / X.norm(dim=1, keepdim=True)) @ (Y / Y.norm(dim=1, keepdim=True)).T).clamp(-1.0, 1.0)
    if method == "pearson":
        A, B = X - X.mean(1, keepdim=True), Y - Y.mean(1, keepdim=True)
        return 1.0 - ((A / A.norm(dim=1, keepdim=True)) @ (B / B.norm(dim=1, keepdim=True)).T).clamp(-1.0, 1.0)
    if method == "euclidean":
        return (X.square().sum(1)[:, None] + Y.square().sum(1)[None, :] - 2.0 * (X @ Y.T)).clamp(min=0.0).sqrt()
    out = torch.empty(X.shape[0], Y.shape[0], dtype=torch.float64, device=X.device)
    Yt, sx, sy = Y.T.contiguous(), X.sum(1), Y.sum(1)
    for i in range(X.shape[0]):           # rows that the query does not store add the reference's own value
        at = X[i].nonzero()[:, 0]
        p, q = X[i, at][:, None], Yt[at]
        if method == "manhattan":
            out[i] = sx[i] + sy + ((p - q).abs() - p - q).sum(0)
        else:
            s = p + q
            shared = (torch.xlogy(s, s) - torch.xlogy(p, p) - torch.xlogy(q, q)).sum(0)
            out[i] = (0.5 * ((sx[i] + sy) * math.log(2.0) - shared)).clamp(min=0.0).sqrt()
    return out


def _smallest(D, k):
    """The k smallest of each row, ascending, as NaN where a row has no value (an empty column)."""
    v = torch.topk(D, k, dim=1, largest=False, sorted=True).values
    return torch.where(torch.isinf(v), torch.full_like(v, math.nan), v)


def _both_ways(method, X, Y, kf, kr):
    D = _distances(method, X, Y)
    D[(X != 0).sum(1) == 0, :] = math.inf
    D[:, (Y != 0).sum(1) == 0] = math.inf
    return {"forward": {"idx": None, "dist": _smallest(D, kf)},
            "reverse": {"idx": None, "dist": _smallest(D.T.contiguous(), kr)}}


def _exact_dense(case, seed):
    X, Q = _embeddings(case, seed)
    k, nq, n = case["k"], _nq(case), case["n"]
    q0 = -1
    if Q is None:
        q0 = (n - nq) // 3
        Q = X[q0:q0 + nq]
    Q = Q.double()
    cosine = case["method"] == "cosine"
    if cosine:
        Q = Q / Q.norm(dim=1, keepdim=True)
    best_v = best_i = None
    step = 1 << 16
    for r0 in range(0, n, step):
        R = X[r0:r0 + step].double()
        if cosine:
            D = 1.0 - (Q @ (R / R.norm(dim=1, keepdim=True)).T)
        else:
            D = Q.square().sum(1)[:, None] + R.square().sum(1)[None, :] - 2.0 * (Q @ R.T)
        if q0 >= 0:
            own = torch.arange(q0, q0 + nq, device="cuda") - r0
            at = ((own >= 0) & (own < R.shape[0])).nonzero()[:, 0]
            D[at, own[at]] = math.inf
        v, i = torch.topk(D, min(2 * k, D.shape[1]), dim=1, largest=False)
        i = i + r0
        if best_v is not None:
            v, i = torch.cat([best_v, v], 1), torch.cat([best_i, i], 1)
            v, at = torch.topk(v, 2 * k, dim=1, largest=False)
            i = i.gather(1, at)
        best_v, best_i = v, i
    if not cosine:       # differences, not norms: near duplicates cancel
        parts = [(X[best_i[a:a + 256]].double() - Q[a:a + 256, None, :]).square().sum(2).sqrt()
                 for a in range(0, nq, 256)]
        best_v = torch.cat(parts)
    return {"idx": None, "dist": torch.topk(best_v, k, dim=1, largest=False, sorted=True).values.T.contiguous()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dense_query", "dense_self"):
        return _exact_dense(case, seed)
    if kind == "resident_block":
        p, i, x = _logcounts(case, seed)
        n, nq = case["n"], _nq(case)
        col = torch.repeat_interleave(torch.arange(n, device="cuda"), (p[1:] - p[:-1]).long())
        Y = torch.zeros(n, ROWS, dtype=torch.float64, device="cuda")
        Y[col, i.long()] = x
        q0 = (n - nq) // 3
        D = _distances(case["method"], Y[q0:q0 + nq], Y)
        at = torch.arange(nq, device="cuda")
        D[at, at + q0] = math.inf
        return {"idx": None, "dist": _smallest(D, case["k"]).T.contiguous()}
    if kind in ("knn", "dist"):
        X = _columns(_matrix(case, case["n"], seed)[0])
        D = _distances(case["method"], X, X)
        at = torch.arange(case["n"], device="cuda")
        if kind == "dist":
            D[at, at] = 0.0
            return D.cpu().numpy()
        gone = (X != 0).sum(1) == 0
        D[gone, :] = math.inf
        D[:, gone] = math.inf
        D[at, at] = math.inf
        return {"idx": None, "dist": _smallest(D, min(case["k"], int((~gone).sum()) - 1))}
    if kind == "cross":
        X, Y = (_columns(M) for M in _matrix(case, case["nq"], seed, case["nr"]))
        return _both_ways(case["method"], X, Y, case["k"], case["k"])
    if kind == "batch":
        out = []
        for sp in _specs(case, seed):
            X, Y = (_columns(M) for M in synth.cross_problem(sp))
            kf, kr = (min(sp["k"], int(((M != 0).sum(1) > 0).sum())) for M in (Y, X))
            out.append(_both_ways(sp["method"], X, Y, kf, kr))
        return out
    idx = _neighbours(case, seed).long() - 1
    n, k = idx.shape
    sets = torch.cat([idx, torch.arange(n, device="cuda")[:, None]], 1).sort(dim=1).values
    w = torch.empty(n, k, dtype=torch.float64, device="cuda")
    for t in range(k):
        other = sets[idx[:, t]].contiguous()
        at = torch.searchsorted(other, sets).clamp(max=k)
        u = (other.gather(1, at) == sets).sum(1).double()
        w[:, t] = u / (2 * (k + 1) - u)
    keep = w > case["prune"]
    i = torch.arange(n, device="cuda")[:, None].expand(n, k)[keep]
    j, v = idx[keep], w[keep]
    key = torch.cat([j * n + i, i * n + j])
    order = key.argsort()
    key, v = key[order], torch.cat([v, v])[order]
    first = torch.ones_like(key, dtype=torch.bool)
    first[1:] = key[1:] != key[:-1]
    return {"p": None, "i": None, "x": v[first].cpu().numpy()}
