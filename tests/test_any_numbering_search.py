"""Matrices in any numbering by one search per vertex: the rule in plain Python against the oracle's
sequential loop (CPU), and the kernels past the sizes of the search's shared-memory table (GPU)."""
import numpy as np
import pytest

from oracle import oracle as O


def _msb(x):
    return int(x).bit_length() - 1


def _search(adj, k):
    """Lengths (sums of edge MSBs) of the shortest paths from k whose intermediates are below k."""
    dist, todo = {}, [(k, 0)]
    while todo:
        x, d = todo.pop(0)
        for y, w in adj[x]:
            if y not in dist or d + w < dist[y]:
                dist[y] = d + w
                if y < k:
                    todo.append((y, d + w))
    return dist


def _rule(A):
    """(diameter, largest product MSB, products) of the sequential loop on an acyclic clean matrix."""
    n = A.shape[0]
    edge = {(i, j): _msb(A[i, j]) for i, j in zip(*np.nonzero(A)) if i != j}
    out = [[] for _ in range(n)]
    into = [[] for _ in range(n)]
    for (i, j), w in edge.items():
        out[i].append((j, w))
        into[j].append((i, w))
    first = dict.fromkeys(edge, -1)       # per cell: the step of its first value (-1: an entry of A)
    top, products, diameter = -1, 0, max(list(edge.values()) + [0])
    for k in range(n):
        o, i = _search(out, k), _search(into, k)
        products += len(o) * len(i)
        if o and i:
            top = max(top, max(o.values()) + max(i.values()))
        for a, da in i.items():
            for b, db in o.items():
                if (a, b) not in first:
                    first[a, b] = k
                    diameter = max(diameter, da + db)
    return diameter, top, products


def test_search_rule_matches_the_loop():
    rng = np.random.default_rng(11)
    checked = 0
    for t in range(150):
        n = int(rng.integers(1, 26))
        A = np.zeros((n, n), np.int64)
        low = np.tril(rng.random((n, n)) < rng.uniform(0.02, 0.4), -1)
        A[low] = rng.integers(2, 40, size=int(low.sum()))
        np.fill_diagonal(A, rng.choice([-1, 0, 1], size=n))
        p = rng.permutation(n)
        A = A[p][:, p]
        d, top, products = _rule(A)
        # the loop itself, on MSBs
        W = A.copy()
        np.fill_diagonal(W, 0)
        cur = [[_msb(v) if v else 0 for v in row] for row in W]
        loop_top, loop_products = -1, 0
        for k in range(n):
            for i in range(n):
                for j in range(n):
                    if cur[i][k] and cur[k][j]:
                        s = cur[i][k] + cur[k][j]
                        loop_top, loop_products = max(loop_top, s), loop_products + 1
                        cur[i][j] = min(cur[i][j], s) if cur[i][j] else s
        assert (top, products) == (loop_top, loop_products), t
        if top >= 31:
            continue
        _, do, so, _ = O.warshall(A.astype(np.int32))
        assert so == 0 and d == do, t
        checked += 1
    assert checked > 60


def _hubs(n, hubs, seed, dtype):
    """A few hubs below and above hundreds of vertices each, edge MSBs 1 to 5, in a random numbering:
    searches of up to n vertices, and vertices shortened after they were taken from the queue."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n), dtype)
    layer = np.sort(rng.integers(0, 5, n))
    for v in range(n):
        earlier = np.flatnonzero(layer < layer[v])
        if earlier.size:
            take = rng.choice(earlier, size=min(3, earlier.size), replace=False)
            A[v, take] = rng.integers(2, 64, take.size)
            old = np.flatnonzero(layer[:hubs] < layer[v])
            if old.size:
                A[v, rng.choice(old)] = rng.integers(2, 64)
    np.fill_diagonal(A, rng.choice([-1, 1], n))
    p = rng.permutation(n)
    return A[p][:, p].copy()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 300, 321, 900, 2500])
def test_search_sizes_vs_oracle(native, n):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_dense
    from redblackgraph_gb300.device import to_device, to_host
    for dtype in (np.int32, np.int64):
        A = _hubs(n, max(1, n // 300), n, dtype)
        Wo, do, so, _ = O.warshall(A)
        out, res = fw_dense(to_device(A))
        assert so == 0 and res.status == 0 and res.path == _lib.PATH_DAG
        assert (to_host(out) == Wo).all() and res.diameter == do
        if n <= 400:
            assert res.executed == _rule(A)[2]
