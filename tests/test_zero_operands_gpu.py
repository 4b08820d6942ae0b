"""Long chains of edges inside one 64-vertex block, beside vertices that reach none or few of them: a
cell without a path stays one however many steps multiply it, in the blocked kernels and in the block
steps of one-sided matrices, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DTYPES = [np.int32, np.int64, np.uint32]


def small_matrices():
    """Entries above the diagonal, n = 64; the closure's values are small, the sums of all shifts along
    the longest chains are past bit 31."""
    chain = np.zeros((64, 64), np.int64)                 # 54 vertices, each linked to all later ones
    for i in range(10, 64):
        chain[i, i + 1:] = 2
    chain[1, 10], chain[0, 63] = 2, 3
    short = np.zeros((64, 64), np.int64)                 # three steps and a short cut past them
    short[0, 2:26] = 2
    short[2, 3] = short[3, 4] = 1024
    short[2, 4], short[4, 8] = 2, 4097
    beside = short.copy()
    beside[[1, 5, 6, 7], 8] = 64
    large = np.zeros((64, 64), np.int64)
    large[1, 10] = large[10, 11] = large[11, 12] = 2
    large[10, 12], large[12, 13], large[0, 13] = 1 << 20, (1 << 12) + 5, 100
    large[20, 21:40] = 2
    return chain, short, beside, large


def dense_dag(n, seed):
    """Nearly every vertex linked to every later one, a few (two in the first block at least) with one
    edge or none."""
    rng = np.random.default_rng(seed)
    A = np.triu((rng.random((n, n)) < 0.9) * rng.integers(2, 4, (n, n)), 1)
    sparse = np.concatenate([rng.choice(min(n, 64) - 8, 2, replace=False), rng.choice(n, 4, replace=False)])
    for v in sparse:
        A[v] = 0
        if v + 1 < n and rng.random() < 0.7:
            A[v, rng.integers(v + 1, n)] = rng.integers(2, 64)
    np.fill_diagonal(A, rng.integers(0, 2, n))
    return A


def numberings(A, seed):
    """As it is, mirrored, and with some neighbours swapped (entries on both sides of the diagonal)."""
    rng = np.random.default_rng(seed)
    p = np.arange(A.shape[0])
    for v in rng.choice(A.shape[0] - 1, max(4, A.shape[0] // 16), replace=False):
        p[[v, v + 1]] = p[[v + 1, v]]
    return A, A[::-1, ::-1].copy(), A[np.ix_(p, p)].copy()


def batch_of(mats):
    """The matrices packed for fw_batch: flat values, sizes, offsets."""
    sizes = np.array([M.shape[0] for M in mats])
    return np.concatenate([M.reshape(-1) for M in mats]), sizes, np.concatenate([[0], np.cumsum(sizes ** 2)[:-1]])


def check_batch(mats, dtype, mode):
    from redblackgraph_gb300.dense import fw_batch
    from redblackgraph_gb300.device import to_device, to_host
    flat, sizes, offsets = batch_of([M.astype(dtype) for M in mats])
    W, res = fw_batch(to_device(flat), sizes, offsets, mode=mode)
    W = to_host(W)
    for M, n, at, r in zip(mats, sizes, offsets, res):
        Wo, do, so, _ = O.warshall(M.astype(dtype))
        assert r.status == so, (n, r.status, so)
        if so == 0:                                      # (an order of steps may overflow where another does not)
            assert r.diameter == do and (W[at:at + n * n].reshape(n, n) == Wo).all(), (n, r.diameter, do)


def check_dense(mats, dtype, mode):
    from redblackgraph_gb300.dense import fw_dense
    from redblackgraph_gb300.device import to_device, to_host
    for M in mats:
        Wo, do, so, _ = O.warshall(M.astype(dtype))
        W, r = fw_dense(to_device(M.astype(dtype)), mode=mode)
        assert r.status == so, (M.shape, r.status, so)
        if so == 0:
            assert r.diameter == do and (to_host(W) == Wo).all(), (M.shape, r.diameter, do)


@pytest.mark.parametrize("dtype", DTYPES)
def test_diagonal_block(native, dtype):
    """One block: the diagonal kernel alone, in a batch and (without the DAG paths) by itself."""
    from redblackgraph_gb300 import _lib
    mats = [N for k, A in enumerate(small_matrices() + tuple(dense_dag(64, s) for s in range(20)))
            for N in numberings(A, k)]
    mats += [N for n in (35, 50, 63) for N in numberings(dense_dag(n, n), n)]
    check_batch(mats, dtype, 0)
    check_dense(mats[:30], dtype, _lib.MODE_NO_DAG)


@pytest.mark.parametrize("dtype", DTYPES)
def test_panels(native, dtype):
    """Several blocks: rows outside a block whose few entries meet the chains inside it."""
    from redblackgraph_gb300 import _lib
    mats = [N for n in (65, 128, 129, 200, 300) for s in range(4) for N in numberings(dense_dag(n, 100 * s + n), n)]
    check_batch(mats, dtype, 0)                          # panels of 64 lines
    check_dense(mats, dtype, _lib.MODE_NO_DAG)           # of 32 lines


@pytest.mark.parametrize("dtype", DTYPES)
def test_block_steps(native, dtype):
    """Through the entry points' own choice of a path: block steps where the entries lie on one side."""
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_dense
    from redblackgraph_gb300.device import to_device
    mats = [N for k, A in enumerate(small_matrices() + tuple(dense_dag(64, s) for s in range(20)))
            for N in numberings(A, k)]
    mats += [N for n in (65, 128, 129, 200, 300) for s in range(4) for N in numberings(dense_dag(n, 100 * s + n), n)]
    check_dense(mats, dtype, 0)
    for A in small_matrices():                           # (none is left to another path for its zeros)
        assert fw_dense(to_device(A.astype(dtype)))[1].path == _lib.PATH_BLOCKED32
