"""The calls a user of this package makes, as cases that can be timed.

Every case is one public entry point on seeded synthetic pedigrees (``redblackgraph_gb300.synth``:
row = child, column = parent, diagonal -1 / 1, father edges 2 and mother edges 3).  ``listed()``
names one case per entry point and size class, ``draw(rng)`` gives another case of the same
ranges.  Sizes are those of the benchmark and the tests: single closures up to 8192 vertices,
batches of pedigrees log-uniform in [16, 4096], forests of up to 2,000,000 vertices.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from redblackgraph_gb300 import _lib, synth
from redblackgraph_gb300.core import array as rb_array
from redblackgraph_gb300.core.avos import matmul_device
from redblackgraph_gb300.dag import dag_closure_device
from redblackgraph_gb300.dense import fw_batch, fw_dense
from redblackgraph_gb300.gpu import CSRMatrixGPU, matmul_gpu
from redblackgraph_gb300.relationship import lookup_many
from redblackgraph_gb300.sparse import component_wise_closure
from redblackgraph_gb300.spgemm import DeviceCSR, squaring_closure


def listed():
    return [
        # one family as a host array: rb.array(...).transitive_closure(), the reference's first
        # example; copies, launches and latency are all of it
        {"name": "array_closure_24", "kind": "array", "n": 24, "dtype": "int32"},
        # the plain dense closure of the benchmark's smallest configuration, resident on the GPU
        {"name": "closure_512", "kind": "closure", "n": 512, "generations": 12, "dtype": "int32",
         "renumbered": False},
        # the largest single dense closure: 30 generations, 64-bit values
        {"name": "closure_8192_int64", "kind": "closure", "n": 8192, "generations": 30, "dtype": "int64",
         "renumbered": False},
        # a pedigree as people enter it: vertices in no particular order
        {"name": "closure_renumbered_3001", "kind": "closure", "n": 3001, "generations": 17, "dtype": "int32",
         "renumbered": True},
        # a dense layered DAG, rows of hundreds of entries (what the blocked kernels are for)
        {"name": "closure_dense_dag_2048", "kind": "dense_dag", "n": 2048, "layers": 24, "dtype": "int32"},
        # many pedigrees of uneven sizes, resident, closed in one call
        {"name": "batch_closure_512", "kind": "batch", "count": 512, "lo": 16, "hi": 4096},
        # a forest on the host, in and out as scipy matrices, split into its components
        {"name": "component_closure_1024", "kind": "components", "count": 1024, "lo": 16, "hi": 4096},
        # rb.array @ on resident operands: a closure times its pedigree extends every path by one
        {"name": "product_2048", "kind": "product", "m": 2048, "q": 2048, "p": 2048, "dtype": "int32"},
        # closure of a sparse forest by repeated squaring, 64-bit values
        {"name": "squaring_1000000", "kind": "squaring", "n": 1_000_000, "dtype": "int64"},
        # one sparse product (redblackgraph.gpu): a forest with itself
        {"name": "sparse_product_300007", "kind": "sparse_product", "n": 300_007},
        # closure of a sparse forest by topological levels
        {"name": "dag_closure_2000000", "kind": "dag", "n": 2_000_000},
        # a serving loop's batch of relationship queries on resident closures
        {"name": "lookup_256", "kind": "lookup", "queries": 256, "graphs": 8, "n": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["array", "closure", "closure", "dense_dag", "batch", "components", "product", "product",
                       "squaring", "sparse_product", "dag", "lookup"])
    if kind == "array":
        return {"kind": kind, "n": _log_int(rng, 4, 64), "dtype": rng.choice(["int32", "int64"])}
    if kind == "closure":
        renumbered = rng.random() < 0.4
        n = _log_int(rng, 64, 3000 if renumbered else 8191)
        return {"kind": kind, "n": n, "generations": rng.randint(8, 18), "dtype": rng.choice(["int32", "int64"]),
                "renumbered": renumbered}
    if kind == "dense_dag":
        return {"kind": kind, "n": _log_int(rng, 130, 2047), "layers": rng.randint(12, 24), "dtype": "int32"}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 4, 300), "lo": 16, "hi": 4096}
    if kind == "components":
        return {"kind": kind, "count": _log_int(rng, 8, 1000), "lo": 16, "hi": 4096}
    if kind == "product":
        return {"kind": kind, "m": _log_int(rng, 17, 2047), "q": _log_int(rng, 17, 2047),
                "p": _log_int(rng, 17, 2047), "dtype": rng.choice(["int32", "int32", "int64"])}
    if kind == "squaring":
        return {"kind": kind, "n": _log_int(rng, 1000, 900_000), "dtype": rng.choice(["int32", "int64"])}
    if kind == "sparse_product":
        return {"kind": kind, "n": _log_int(rng, 1000, 1_000_000)}
    if kind == "dag":
        return {"kind": kind, "n": _log_int(rng, 1000, 1_900_000)}
    return {"kind": kind, "queries": _log_int(rng, 32, 512), "graphs": rng.randint(1, 8), "n": _log_int(rng, 64, 4096)}


# ------------------------------------------------------------------------------- inputs
def _pedigree(n, generations, seed, dtype, renumbered=False):
    """The dense matrix of synth.pedigree, filled in on the GPU; ``renumbered`` shuffles the
    vertices (entries on both sides of the diagonal)."""
    colors, c, p, v = synth.pedigree_edges(n, generations, seed)
    new = np.random.default_rng(seed + 1).permutation(n) if renumbered else np.arange(n)
    A = torch.zeros((n, n), dtype=getattr(torch, dtype), device="cuda")
    rows = torch.from_numpy(np.concatenate([new, new[c]])).cuda()
    cols = torch.from_numpy(np.concatenate([new, new[p]])).cuda()
    A[rows, cols] = torch.from_numpy(np.concatenate([colors, v])).cuda().to(A.dtype)
    return A


def _layered_dag(n, layers, seed, dtype):
    """Vertices in layers, numbered in layer order, each linked to every vertex of an earlier layer
    with probability one half (values 2 / 3); the diagonal holds the colours."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    layer = torch.randint(0, layers, (n,), generator=g, device="cuda").sort().values
    link = (layer[:, None] > layer[None, :]) & (torch.rand((n, n), generator=g, device="cuda") < 0.5)
    val = torch.randint(2, 4, (n, n), generator=g, device="cuda")
    A = torch.where(link, val, torch.zeros_like(val)).to(getattr(torch, dtype))
    colors = torch.randint(0, 2, (n,), generator=g, device="cuda") * 2 - 1
    A.diagonal().copy_(colors.to(A.dtype))
    return A


FAMILY = 64   # vertices of a family of a forest


def _forest(n, seed, dtype):
    """The forest of n vertices with its families (blocks of FAMILY vertices) laid out in an order
    drawn from the seed: other inputs for another seed, with the same number of entries."""
    F = synth.forest(n, 25, n, family=FAMILY, reach=3, p_parent=0.97, dtype=np.dtype(dtype))
    blocks = n // FAMILY
    order = np.random.default_rng(seed).permutation(blocks)
    old = (order[:, None] * FAMILY + np.arange(FAMILY)).reshape(-1)    # old row of each new row
    old = np.concatenate([old, np.arange(blocks * FAMILY, n)])
    length = np.diff(F.indptr).astype(np.int64)[old]
    indptr = np.concatenate([[0], np.cumsum(length)])
    at = np.repeat(F.indptr[:-1][old] - indptr[:-1], length) + np.arange(indptr[-1])
    shift = np.repeat(np.arange(n) - old, length)                      # a family moves as one
    return type(F)((F.data[at], (F.indices[at] + shift).astype(np.int32), indptr.astype(F.indptr.dtype)),
                   shape=F.shape)


def _pedigrees(case):
    """Sizes and seeds of the case's pedigrees."""
    return synth.batch_components(case["count"], case["lo"], case["hi"], seed=case["count"])


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "array":
        A = synth.pedigree(case["n"], max(2, round(1.5 * math.log2(case["n"]))), seed, dtype=np.dtype(case["dtype"]))
        state["A"] = rb_array(A)
    elif kind in ("closure", "dense_dag"):
        if kind == "closure":
            state["A"] = _pedigree(case["n"], case["generations"], seed, case["dtype"], case["renumbered"])
        else:
            state["A"] = _layered_dag(case["n"], case["layers"], seed, case["dtype"])
        state["out"] = torch.empty_like(state["A"])
    elif kind == "batch":
        sizes, seeds = _pedigrees(case)
        seeds = (seeds + 7 * seed) % (2 ** 31 - 1)
        idx, val, offsets = synth.batch_edges(sizes, seeds)
        buf = torch.zeros(int((sizes * sizes).sum()), dtype=torch.int32, device="cuda")
        buf[torch.from_numpy(idx).cuda()] = torch.from_numpy(val).cuda().to(torch.int32)
        state.update(buf=buf, out=torch.empty_like(buf), sizes=sizes, offsets=offsets)
    elif kind == "components":
        # the same pedigrees in another order for another seed
        sizes, seeds = _pedigrees(case)
        order = np.random.default_rng(seed).permutation(sizes.size)
        state["forest"], _ = synth.batch_forest(sizes[order], seeds[order])
    elif kind == "product":
        # the closure of a pedigree times its matrix, cut to m x q and q x p
        n = max(case["m"], case["q"], case["p"])
        A = _pedigree(n, synth.generations_for(n), seed, case["dtype"])
        W, _ = fw_dense(A)
        state["a"] = W[n - case["m"]:, :case["q"]].contiguous()
        state["b"] = A[:case["q"], :case["p"]].contiguous()
    elif kind == "squaring":
        state["A"] = DeviceCSR.from_scipy(_forest(case["n"], seed, case["dtype"]))
    elif kind == "sparse_product":
        state["A"] = CSRMatrixGPU.from_cpu(_forest(case["n"], seed, "int32"))
        state["B"] = state["A"].copy()
    elif kind == "dag":
        state["A"] = DeviceCSR.from_scipy(_forest(case["n"], seed, "int32"))
    else:
        n = case["n"]
        graphs = [fw_dense(_pedigree(n, synth.generations_for(n), seed + 101 * g, "int32"))[0]
                  for g in range(case["graphs"])]
        pick = np.random.default_rng(seed)
        state["queries"] = [(graphs[int(pick.integers(len(graphs)))], int(pick.integers(n)), int(pick.integers(n)))
                            for _ in range(case["queries"])]
    return state


# ------------------------------------------------------------------------------- one call
def run(state):
    kind = state["kind"]
    if kind == "array":
        r = state["A"].transitive_closure()
        return [r.W, int(r.diameter)]
    if kind in ("closure", "dense_dag"):
        W, res = fw_dense(state["A"], out=state["out"])
        return [W, int(res.diameter), int(res.status)]
    if kind == "batch":
        W, res = fw_batch(state["buf"], state["sizes"], state["offsets"], out=state["out"],
                          mode=_lib.MODE_GRAPH | _lib.MODE_AUTOTUNE, as_array=True)
        return [W, res["diameter"], res["status"]]
    if kind == "components":
        r = component_wise_closure(state["forest"])
        return [r.W.data, r.W.indices, r.W.indptr, int(r.diameter)]
    if kind == "product":
        C, status, flags = matmul_device(state["a"], state["b"])
        return [C, int(status), int(flags)]
    if kind == "squaring":
        R, steps = squaring_closure(state["A"])
        return [R.indptr, R.indices, R.data, int(steps)]
    if kind == "sparse_product":
        C = matmul_gpu(state["A"], state["B"])
        return [C.indptr, C.indices, C.data]
    if kind == "dag":
        C, largest, levels = dag_closure_device(state["A"])
        return [C.indptr, C.indices, C.data, int(largest), int(levels)]
    found = lookup_many(state["queries"])
    names = np.array([r.relationship for r in found], dtype="S48")
    return [np.array([r.common_ancestor for r in found], dtype=np.int64), names.view(np.uint8)]


# ------------------------------------------------------------------------------- what a call must do
def _forest_counts(n):
    """Typical counts of the forests per vertex: stored entries 2.85, closure entries 14.6,
    candidates of the closure by levels 21."""
    return 2.85 * n, 14.6 * n, 21.0 * n


def work(case):
    """Bytes: every input read once, every output written once.  Operations: two (a product and a
    sum of the algebra) per pair of operands that meets."""
    kind = case["kind"]
    if kind == "array":
        return {"bytes": 2 * case["n"] ** 2 * np.dtype(case["dtype"]).itemsize, "flops": 0}
    if kind == "closure":
        return {"bytes": 2 * case["n"] ** 2 * np.dtype(case["dtype"]).itemsize, "flops": 0}
    if kind == "dense_dag":
        n = case["n"]
        return {"bytes": 8 * n * n, "flops": 2 * n ** 3 / 6}
    if kind == "batch":
        # mean of n^2 for n log-uniform in [lo, hi]
        lo, hi = case["lo"], case["hi"]
        return {"bytes": 8 * case["count"] * (hi ** 2 - lo ** 2) / (2 * math.log(hi / lo)), "flops": 0}
    if kind == "components":
        # in: int32 row pointers, columns, values of ~2.6 entries a row; out: ~12 entries a row
        lo, hi = case["lo"], case["hi"]
        rows = case["count"] * (hi - lo) / math.log(hi / lo)
        return {"bytes": rows * (4 + 8 * 2.6 + 4 + 8 * 12), "flops": 0}
    if kind == "product":
        size = np.dtype(case["dtype"]).itemsize
        m, q, p = case["m"], case["q"], case["p"]
        return {"bytes": size * (m * q + q * p + m * p), "flops": 2 * m * q * p}
    n = case.get("n", 0)
    if kind == "squaring":
        a, c, _ = _forest_counts(n)
        return {"bytes": (4 + np.dtype(case["dtype"]).itemsize) * a + 8 * c + 16 * n, "flops": 0}
    if kind == "sparse_product":
        return {"bytes": 2 * (8 * 2.85 * n + 8 * n) + 8 * 6.3 * n + 8 * n, "flops": 0}
    if kind == "dag":
        a, c, cand = _forest_counts(n)
        return {"bytes": 8 * a + 8 * c + 16 * n, "flops": 2 * cand}
    return {"bytes": case["queries"] * (2 * 4 * n + 24), "flops": 0}


# ------------------------------------------------------------------------------- plain 64-bit answers
def _msb(x):
    return torch.frexp(x.to(torch.float64))[1].to(torch.int64) - 1


def _encode(v):
    """Values so that the sum is a minimum: the red one first, no path last."""
    return torch.where(v == 0, torch.full_like(v, 2 ** 62), v)


def _step(acc, x, y):
    """acc (+) x (x) y for a column x (m, 1) and a row y (1, p); acc as _encode gives it."""
    bits = torch.where(y >= 2, _msb(y.clamp(min=1)), torch.zeros_like(y))
    spliced = (x << bits) | (y - (torch.ones_like(y) << bits))
    r = torch.where((x >= 2) & (y >= 2), spliced, torch.zeros_like(spliced))
    r = torch.where((x.abs() == 1) & (y >= 2), y.expand_as(r), r)
    keep = (x >= 2) & (y.abs() == 1) & ((x & 1) == (y == 1).to(x.dtype))
    r = torch.where(keep | ((x.abs() == 1) & (x == y)), x.expand_as(r), r)
    return torch.minimum(acc, _encode(r))


def _decode(acc):
    return torch.where(acc == 2 ** 62, torch.zeros_like(acc), acc)


def exact(case, seed):
    """The sequential loop, or the product, in 64-bit integers; None where that takes too long
    (n = 8192, batches and forests)."""
    kind = case["kind"]
    if kind in ("array", "closure", "dense_dag") and case["n"] <= 3001:
        A = prepare(case, seed)["A"]
        A = torch.from_numpy(np.asarray(A)).cuda() if kind == "array" else A
        A = A.to(torch.int64)
        acc = _encode(A)
        top = torch.zeros((), dtype=torch.int64, device=A.device)
        for k in range(case["n"]):
            W = _decode(acc)
            acc = _step(acc, W[:, k:k + 1], W[k:k + 1, :])
            top = torch.maximum(top, _decode(acc).max())
        largest = int(top)
        W = _decode(acc)
        diameter = largest.bit_length() - 1 if largest > 1 else 0
        return [W.cpu().numpy() if kind == "array" else W, diameter] + ([] if kind == "array" else [0])
    if kind == "product":
        state = prepare(case, seed)
        a, b = state["a"].to(torch.int64), state["b"].to(torch.int64)
        acc = torch.full((a.shape[0], b.shape[1]), 2 ** 62, dtype=torch.int64, device=a.device)
        for j in range(a.shape[1]):
            acc = _step(acc, a[:, j:j + 1], b[j:j + 1, :])
        return [_decode(acc), 0, 0]
    return None
