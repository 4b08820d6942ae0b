"""Closures of few rows in all (one warp per row, waiting for its parents): the row sizes, bitmap
sizes and generations where the kernel changes its way, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _layers(n, layers, entries, seed, dtype, hi=8):
    """Rows of up to `entries` entries (values 2 .. hi - 1) in earlier layers, numbered by layer."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n), dtype)
    layer = np.sort(rng.integers(0, layers, n))
    for v in range(n):
        earlier = int(np.searchsorted(layer, layer[v]))
        if earlier:
            take = rng.choice(earlier, size=min(entries, earlier), replace=False)
            A[v, take] = rng.integers(2, hi, take.size)
    np.fill_diagonal(A, rng.choice([-1, 0, 1], n))
    return A


CASES = [(1, 1, 1), (2, 2, 1), (31, 4, 2), (33, 4, 16), (64, 8, 3), (300, 300, 1), (500, 3, 16),
         (1025, 4, 16), (1300, 6, 12)]                        # the last: rows past 512 columns


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_short_closures(native, dtype):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_batch, fw_dense, pack
    from redblackgraph_gb300.device import to_device, to_host
    mats = []
    for k, (n, layers, entries) in enumerate(CASES):
        A = _layers(n, layers, entries, k, dtype, hi=3 if layers > 100 else 8)
        mats += [A, A[::-1, ::-1].copy()]                # below and above the diagonal
    expect = [O.warshall(A) for A in mats]
    for A, (Wo, do, so, _) in zip(mats, expect):
        d = to_device(A)
        for out in (None, d):                            # out of place, then in place
            W, r = fw_dense(d, out=out)
            assert r.status == so
            if so == 0:
                assert (to_host(W) == Wo).all() and r.diameter == do, A.shape
    # one batch of all of them, with matrices in any numbering and a cyclic one among them
    rng = np.random.default_rng(3)
    for k in (8, 10, 12):
        q = rng.permutation(mats[k].shape[0])
        mats.append(mats[k][q][:, q].copy())
    cyclic = mats[8].copy()
    cyclic[:2, :2], cyclic[0, 1], cyclic[1, 0] = 0, 2, 3
    mats.append(cyclic)
    expect += [O.warshall(A) for A in mats[-4:]]
    flat, sizes, offsets = pack(mats)
    d = to_device(flat)
    for out in (None, d):
        W, res = fw_batch(d, sizes, offsets, out=out)
        h = to_host(W)
        for A, o, r, (Wo, do, so, _) in zip(mats, offsets, res, expect):
            n = A.shape[0]
            assert r.status == so
            if so == 0:
                assert (h[o:o + n * n].reshape(n, n) == Wo).all() and r.diameter == do, n
                assert r.path == _lib.PATH_DAG, n
