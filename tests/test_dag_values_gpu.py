"""The DAG closure's tiles at the ends of their value range, against the oracle, and with diagonal entries
stored twice, against the levels."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOP = 2 ** 31 - 1


def _families(family, count, side, seed):
    """Families whose entries include 2^31 - 1, and pairs whose product is 2^31 - 1."""
    rng = np.random.default_rng([family, seed])
    M = np.zeros((family * count, family * count), np.int64)
    for f in range(0, family * count, family):
        for i in range(1, family):
            to = f + rng.choice(i, min(i, 2), replace=False)
            M[f + i, to] = rng.integers(2, 4, to.size)
        leaf = f + family - 1
        M[leaf] = 0
        M[leaf, f] = TOP                                         # an edge to a vertex without parents
        if family > 5:
            a, b = 1 + rng.integers(0, 14), f + family - 3       # 2^a - 1 and 2^(32 - a) - 1, splices to the top
            M[b - 2] = M[b - 1] = M[b] = 0
            M[b, b - 1], M[b - 1, b - 2] = 2 ** (a + 1) - 1, 2 ** (31 - a) - 1
    np.fill_diagonal(M, rng.choice([-1, 0, 1], M.shape[0]))
    return sp.csr_matrix((M if side < 0 else M[::-1, ::-1].copy()).astype(np.int32))


@pytest.mark.parametrize("side", [-1, 1])
def test_largest_value(native, side):
    from redblackgraph_gb300.dag import dag_closure_device
    from redblackgraph_gb300.spgemm import DeviceCSR
    for family, count in ((2, 3), (5, 20), (20, 9), (63, 2), (64, 5), (65, 2)):
        A = _families(family, count, side, count)
        W = sp.csr_matrix(O.dag_closure(A)[0])
        W.sort_indices()
        assert (W.data == TOP).sum() >= count
        for tiles in (True, False):
            C, mx, _ = dag_closure_device(DeviceCSR.from_scipy(A), tiles=tiles)
            got = C.to_scipy()
            assert mx == TOP and (got.indptr == W.indptr).all()
            assert (got.indices == W.indices).all() and (got.data == W.data).all(), (family, tiles)


def test_diagonal_stored_twice(native):
    import torch
    from redblackgraph_gb300.dag import dag_closure_device
    from redblackgraph_gb300.device import to_host
    from redblackgraph_gb300.spgemm import DeviceCSR
    twice = [(1, -1), (-1, 1), (1, 1), (-1, -1), (1,), (-1,), ()]
    rows = [[(i - 1, 2)] * (i % 7 > 0) + [(i, v) for v in twice[i % 7]] for i in range(64)]
    ptr = torch.tensor(np.cumsum([0] + [len(r) for r in rows]), device="cuda")
    col = torch.tensor([c for r in rows for c, _ in r], dtype=torch.int32, device="cuda")
    val = torch.tensor([v for r in rows for _, v in r], dtype=torch.int32, device="cuda")
    got, want = (dag_closure_device(DeviceCSR(ptr, col, val, (64, 64)), tiles=t) for t in (True, False))
    assert got[1:] == want[1:]
    for a, b in ((got[0].indptr, want[0].indptr), (got[0].indices, want[0].indices), (got[0].data, want[0].data)):
        assert (to_host(a) == to_host(b)).all()
    assert want[0].to_scipy().diagonal().tolist() == [min(twice[i % 7], default=0) for i in range(64)]


@pytest.mark.parametrize("sizes", [[1], [40], [65] * 4, [64] * 3 + [100] * 2, [100] * 5 + [20],
                                   [64] * 400 + [70] * 300, [64] * 300 + [70] * 400, [3, 90] * 500])
def test_pieces_in_any_share(native, sizes):
    """Pieces a tile holds and larger ones, about half of the rows each, past the positions looked at: with
    the tiles or without, the same closure."""
    from redblackgraph_gb300.dag import dag_closure_device
    from redblackgraph_gb300.device import to_host
    from redblackgraph_gb300.spgemm import DeviceCSR
    rng = np.random.default_rng(len(sizes))
    first = np.repeat(np.concatenate([[0], np.cumsum(sizes)[:-1]]), sizes)
    n = first.size
    i = np.arange(n)
    parent = np.where(i > first, np.maximum(i - rng.integers(1, 12, n), first), -1)
    other = np.where(i > first + 1, first + 1, -1)
    r, c = np.concatenate([i, i, i]), np.concatenate([i, parent, other])
    key = np.unique((r * n + c)[(c >= 0)])
    r, c = key // n, key % n
    v = np.where(r == c, rng.choice([-1, 1], key.size), rng.integers(2, 4, key.size)).astype(np.int32)
    A = DeviceCSR.from_scipy(sp.csr_matrix((v, (r, c)), shape=(n, n)))
    got, want = dag_closure_device(A), dag_closure_device(A, tiles=False)
    assert got[1:] == want[1:]
    for a, b in ((got[0].indptr, want[0].indptr), (got[0].indices, want[0].indices), (got[0].data, want[0].data)):
        assert (to_host(a) == to_host(b)).all()
