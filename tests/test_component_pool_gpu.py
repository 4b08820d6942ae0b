"""Component-wise closure of graphs whose closure rows outgrow the first pool, and of ones with a row or a
span that rows waiting for their parents are not for, against the closure by levels."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _deep(n, generations, per_row, seed, above=False):
    """Vertices in generations, each linked to `per_row` of the generation before."""
    rng = np.random.default_rng(seed)
    gen = np.sort(rng.integers(0, generations, n))
    r = np.repeat(np.arange(n), per_row)
    lo, hi = np.searchsorted(gen, gen[r] - 1), np.searchsorted(gen, gen[r])
    c = lo + (rng.random(r.size) * np.maximum(hi - lo, 1)).astype(int)
    key = np.unique((r * n + c)[c < hi])
    M = sp.coo_matrix((rng.integers(2, 4, key.size), (key // n, key % n)), shape=(n, n)).tolil()
    M.setdiag(rng.choice([-1, 1], n))
    M = M.tocsr()
    return M[::-1, ::-1].tocsr() if above else M


def _both(F, monkeypatch):
    """The closure with a look at what _close_rows gave, and without it."""
    from redblackgraph_gb300 import components
    from redblackgraph_gb300.sparse import component_wise_closure
    rows, seen = components._close_rows, []

    def watched(*a):
        seen.append(rows(*a))
        return seen[-1]
    F.sort_indices()
    monkeypatch.setattr(components, "_close_rows", watched)
    got = component_wise_closure(F)
    monkeypatch.setattr(components, "_close_rows", lambda *a: None)
    want = component_wise_closure(F)
    assert got.diameter == want.diameter
    for x, y in ((got.W.indptr, want.W.indptr), (got.W.indices, want.W.indices), (got.W.data, want.W.data)):
        assert np.array_equal(x, y)
    return seen


# `near`: the first pool nearly suffices, and the rows are closed with the second one
@pytest.mark.parametrize("sizes, generations, per_row, near",
                         [([150], 8, 2, True), ([2000], 7, 2, True), ([200], 12, 3, False), ([1500], 16, 2, False),
                          ([900, 70, 2000, 300], 20, 3, False), ([2000] * 8, 7, 2, True), ([3000] * 4, 14, 2, False)])
def test_pool_grows(native, monkeypatch, sizes, generations, per_row, near):
    F = sp.block_diag([_deep(n, generations, per_row, k, k % 2 == 1) for k, n in enumerate(sizes)], "csr")
    (rows,) = _both(F, monkeypatch)
    edges = F.nnz - int((F.diagonal() != 0).sum())
    assert (rows is not None) == near
    assert not near or rows.cols.numel() > 16 * edges + F.shape[0]


def test_rows_and_spans_past_the_limits(native, monkeypatch):
    small = [_deep(300, 6, 2, k) for k in range(3)]
    assert _both(sp.block_diag(small, "csr"), monkeypatch)[0] is not None
    wide = np.zeros((40, 40), np.int64)
    wide[30, :17] = 2
    assert _both(sp.block_diag(small + [sp.csr_matrix(wide)], "csr"), monkeypatch) == [None]
    apart = sp.block_diag([sp.csr_matrix((1, 1))] + [_deep(2050, 6, 2, k) for k in range(4)] + [sp.csr_matrix((1, 1))], "lil")
    n = apart.shape[0]
    apart[n - 1, 0] = 2                                  # vertices 0 and n - 1, 8201 apart
    assert _both(apart.tocsr(), monkeypatch) == [None]
