"""The closure of a DAG by levels and by tiles (pieces of consecutive vertices no edge leaves): piece
sizes around the tile's, both sides of the diagonal, and pieces the tiles leave to the levels."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _pieces(sizes, side, per_row, seed, hi=8, diag=True):
    """Pieces of the given sizes; side -1: entries below the diagonal, 1: above, 0: in random order."""
    rng = np.random.default_rng(seed)
    rows, cols, vals = [], [], []
    base = 0
    for k, n in enumerate(sizes):
        order = rng.permutation(n) if side == 0 else np.arange(n) if side < 0 else np.arange(n)[::-1]
        for i in range(n):
            if diag and rng.random() < 0.9:
                rows.append(base + order[i]); cols.append(base + order[i]); vals.append(int(rng.choice([-1, 1])))
            lo = max(0, i - 20)
            take = rng.choice(np.arange(lo, i), size=min(per_row, i - lo), replace=False) if i else []
            for j in take:
                rows.append(base + order[i]); cols.append(base + order[int(j)]); vals.append(int(rng.integers(2, hi)))
        base += n
    M = sp.csr_matrix((np.array(vals, np.int32), (np.array(rows), np.array(cols))), shape=(base, base))
    M.sort_indices()
    return M


def _levels(A):
    n = A.shape[0]
    lev = np.zeros(n, int)
    for _ in range(n):                                      # longest chains, by relaxation
        C = A.tocoo()
        off = C.row != C.col
        new = lev.copy()
        np.maximum.at(new, C.row[off], lev[C.col[off]] + 1)
        if (new == lev).all():
            break
        lev = new
    return int(lev.max()) + 1


@pytest.mark.parametrize("side", [-1, 1, 0])
def test_tiles_and_levels(native, side):
    from redblackgraph_gb300.dag import dag_closure_device
    from redblackgraph_gb300.spgemm import DeviceCSR
    for sizes, per_row, hi in (([1], 1, 8), ([64], 2, 4), ([65], 2, 4), ([63, 1, 64, 2, 62], 2, 4), ([20] * 30, 2, 4),
                               ([64] * 9 + [7], 2, 3), ([200, 3, 64, 64, 100, 1, 1, 1, 5], 2, 4),
                               ([64, 64], 12, 3),           # more entries than a tile holds
                               ([40, 64, 30], 2, 1 << 20)): # products past bit 31: Cython wraps
        A = _pieces(sizes, side, per_row, len(sizes) + per_row, hi)
        W, d = O.dag_closure(A)
        C, mx, levels = dag_closure_device(DeviceCSR.from_scipy(A))
        got = C.to_scipy()
        W = sp.csr_matrix(W)
        W.sort_indices()
        assert (got.indptr == W.indptr).all() and (got.indices == W.indices).all() and (got.data == W.data).all(), sizes
        assert (mx.bit_length() - 1 if mx > 1 else 0) == d, sizes
        assert levels == _levels(A), sizes


def test_tiles_pool_growth_and_odd_values(native):
    from redblackgraph_gb300.dag import dag_closure_device
    from redblackgraph_gb300.spgemm import DeviceCSR
    A = _pieces([64] * 20, -1, 3, 5, 3)
    W, _ = O.dag_closure(A)
    for factor in (0, 1, 16):                               # pools too small: the call repeats
        C, _, _ = dag_closure_device(DeviceCSR.from_scipy(A), pool_factor=factor)
        assert (C.to_scipy() != sp.csr_matrix(W)).nnz == 0
    B = A.copy()
    off = np.flatnonzero(B.data > 1)
    B.data[off[::7]] = 1                                    # identities and negatives off the diagonal
    B.data[off[3::11]] = -1
    B.data[off[5::13]] = -7
    W, d = O.dag_closure(B)
    C, mx, _ = dag_closure_device(DeviceCSR.from_scipy(B))
    assert (C.to_scipy() != sp.csr_matrix(W)).nnz == 0 and (mx.bit_length() - 1 if mx > 1 else 0) == d
