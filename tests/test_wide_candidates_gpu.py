"""Acyclic matrices in any numbering with entries that a shorter path makes needless: the recurrence over
the closure's rows meets products past 31 bits there that the loop never forms.  Against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _short(dtype):
    A = np.zeros((6, 6), dtype)
    A[0, 2], A[0, 1], A[1, 2], A[2, 3] = 1 << 20, 2, 2, (1 << 15) + 1   # 2^20 (x) (2^15 + 1) wraps to 1
    A[5, 4] = 2                                                          # an entry below the diagonal
    return A


def _chain(n, seed, dtype):
    """Every vertex linked to the next one and with a needless large entry to the one after it; rows of
    up to 12 entries among the last ones."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n), np.int64)
    for i in range(n - 1):
        A[i, i + 1] = 2 if i % 2 else 3
        if i + 2 < n:
            A[i, i + 2] = (1 << int(rng.integers(12, 24))) + int(rng.integers(0, 9))
    for i in range(n - 14, n - 2):
        A[i, i + 2:] = 2
    A[n // 2, [0, 1]] = 0
    p = np.arange(n)
    p[[n - 1, n - 2]] = p[[n - 2, n - 1]]            # two vertices swapped: entries on both sides
    return A[np.ix_(p, p)].astype(dtype)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_products_the_loop_does_not_form(native, dtype):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_batch, fw_dense
    from redblackgraph_gb300.device import to_device, to_host
    mats = [_short(dtype)] + [_chain(n, n + s, dtype) for n in (16, 24, 28, 36) for s in range(3)]
    want = [O.warshall(M) for M in mats]
    assert any(w[2] == 0 for w in want[1:])
    for M, (Wo, do, so, _) in zip(mats, want):
        W, r = fw_dense(to_device(M))
        assert r.status == so
        assert so != 0 or (r.diameter == do and (to_host(W) == Wo).all()), M.shape
    assert fw_dense(to_device(mats[0]))[1].path == _lib.PATH_DAG
    sizes = np.array([M.shape[0] for M in mats])
    offsets = np.concatenate([[0], np.cumsum(sizes ** 2)[:-1]])
    W, res = fw_batch(to_device(np.concatenate([M.reshape(-1) for M in mats])), sizes, offsets)
    W = to_host(W)
    for n, at, r, (Wo, do, so, _) in zip(sizes, offsets, res, want):
        assert r.status == so
        assert so != 0 or (r.diameter == do and (W[at:at + n * n].reshape(n, n) == Wo).all())
