"""Diameters of acyclic matrices in which step 0 of the loop lowers an entry: its largest value is looked
at after the step only, so the entry itself never counts.  Against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _matrix(n, seed, dtype):
    """Short rows in any numbering, vertex 0 between others; the largest entries run beside it."""
    rng = np.random.default_rng([n, seed])
    A = np.zeros((n, n), np.int64)
    rank = rng.permutation(n)                        # an edge goes to a lower rank
    mid = int(np.flatnonzero(rank == n // 2)[0])
    rank[[0, mid]] = rank[[mid, 0]]
    up, down = np.flatnonzero(rank > rank[0]), np.flatnonzero(rank < rank[0])
    for i in range(n):
        to = np.flatnonzero(rank < rank[i])
        to = rng.choice(to, min(to.size, 2), replace=False)
        A[i, to] = rng.integers(2, 4, to.size)
    a, b = rng.choice(up, min(up.size, 4), replace=False), rng.choice(down, min(down.size, 6), replace=False)
    A[a, 0] = rng.integers(2, 6, a.size)
    A[0, b] = rng.integers(2, 6, b.size)
    A[a[0], b[0]] = 40000                            # lowered by step 0
    if seed % 3 == 0 and b.size > 1:
        A[a[0], b[1]] = 5000
    if seed % 3 == 1:
        A[a[0], 0] = 1 << 14                         # step 0's product is larger here
    np.fill_diagonal(A, rng.integers(0, 2, n))
    return A.astype(dtype)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_step_zero(native, dtype):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_batch, fw_dense
    from redblackgraph_gb300.device import to_device, to_host
    mats = [_matrix(n, s, dtype) for n in (4, 10, 33, 200, 700) for s in range(6)]
    want = [O.warshall(M) for M in mats]
    lowered = 0
    for M, (Wo, do, so, _) in zip(mats, want):
        W, r = fw_dense(to_device(M))
        assert r.status == so == 0 and r.diameter == do and (to_host(W) == Wo).all(), M.shape
        lowered += do < int(M.max()).bit_length() - 1 and r.path == _lib.PATH_DAG
    assert lowered >= 10
    sizes = np.array([M.shape[0] for M in mats])
    offsets = np.concatenate([[0], np.cumsum(sizes ** 2)[:-1]])
    _, res = fw_batch(to_device(np.concatenate([M.reshape(-1) for M in mats])), sizes, offsets)
    assert [r.diameter for r in res] == [w[1] for w in want] and all(r.path == _lib.PATH_DAG for r in res)
