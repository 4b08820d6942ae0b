"""Squaring steps where the tiles' and groups' shortcuts must not show: columns stored twice,
identities that meet other products, and columns that do not ascend."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(rows, n, dtype):
    """DeviceCSR of lists of (column, value) per row, as given."""
    import torch
    from redblackgraph_gb300.device import to_device
    from redblackgraph_gb300.spgemm import DeviceCSR
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    flat = [e for r in rows for e in r]
    return DeviceCSR(torch.from_numpy(ptr).cuda(), torch.tensor([c for c, _ in flat], dtype=torch.int32).cuda(),
                     to_device(np.array([v for _, v in flat], dtype)), (n, n))


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.uint32, np.uint64])
@pytest.mark.parametrize("family", [64, 100])
def test_parent_row_with_a_column_twice(native, dtype, family):
    """Row v of a family: its parent v - 1 holds column 0 of the family twice, the lesser value first or
    last, next to each other or with others between.  The product takes the lesser one."""
    from redblackgraph_gb300.device import to_host
    from redblackgraph_gb300.spgemm import spgemm
    n = 4 * family
    twice, once = [], []
    for i in range(n):
        f = i // family * family
        v, lo, hi = i - f, 4 + i % 3, 9 + i % 4
        pair = [(f, lo), (f, hi)] if v % 4 < 2 else [(f, hi), (f, lo)]
        between = [(f + 1, 60), (f + 2, 61)] if v % 2 and v > 6 else []
        up = [(i - 1, 2)] if v > 3 else []
        odd = v > 3 and v % 3 == 0                  # rows with a column twice, each the parent of one without
        twice.append((pair[:1] + between + pair[1:] if odd else []) + up + [(i, 1)])
        once.append(([(f, lo)] + between if odd else []) + up + [(i, 1)])
    A, B = _csr(twice, n, dtype), _csr(once, n, dtype)
    got, want = spgemm(A, A, R=A)[0].to_scipy().toarray(), spgemm(B, B, R=B)[0].to_scipy().toarray()
    keep = [i for i in range(n) if len({c for c, _ in twice[i]}) == len(twice[i])]
    assert len(keep) > n // 2 and (want[keep] != 0).sum() > 3 * len(keep)
    assert (got[keep] == want[keep]).all()


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_rows_of_many_candidates_in_one_block(native, dtype):
    """64 columns, but more than 8192 candidates a row, as every row holds its columns many times."""
    from redblackgraph_gb300.spgemm import spgemm
    n = 64
    rows = [[(c, 2 + c % 2) for c in range(max(i - 12, 0), i) for _ in range(30)] + [(i, 1)] for i in range(n)]
    once = [[(c, 2 + c % 2) for c in range(max(i - 12, 0), i)] + [(i, 1)] for i in range(n)]
    A, B = _csr(rows, n, dtype), _csr(once, n, dtype)
    got, want = spgemm(A, A, R=A), spgemm(B, B, R=B)
    assert got[1:] == want[1:] and (got[0].to_scipy().toarray() == want[0].to_scipy().toarray()).all()


def _cells(m):
    m = m.tocoo()
    return {(r, c): v for r, c, v in zip(m.row.tolist(), m.col.tolist(), m.data.tolist()) if v != 0}


def _merged(R, S):
    """R (+) R^2 by magnitude (R's value on a tie), as int32."""
    mag = (lambda v: v) if R.dtype.kind == "u" else abs
    r, s = _cells(R), _cells(S)
    out = {k: s[k] if k not in r or (k in s and mag(s[k]) < mag(r[k])) else r[k] for k in {**r, **s}}
    return {k: w for k, w in ((k, int(np.array(v, R.dtype).astype(np.int32))) for k, v in out.items()) if w != 0}


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.uint32, np.uint64])
@pytest.mark.parametrize("n, family", [(1, 1), (64, 64), (300, 64), (320, 100), (400, 200), (90, 3)])
def test_identities_that_meet_products(native, dtype, n, family):
    """Families with entries on both sides of the diagonal (cycles, so that plain products reach the
    diagonal's identities) and a few identities off it, at columns whose diagonal is the same identity."""
    from redblackgraph_gb300.spgemm import DeviceCSR, spgemm
    red = np.array(-1, np.int64).astype(dtype)
    for seed in range(6):
        rng = np.random.default_rng([n, family, seed])
        A = np.zeros((n, n), dtype)
        r = np.repeat(np.arange(n), 3)
        f = r // family * family
        c = f + (rng.random(r.size) * (np.minimum(f + family, n) - f)).astype(int)
        A[r, c] = rng.integers(2, 9, r.size)
        k = rng.choice(r.size, max(1, r.size // 10))
        A[r[k], c[k]] = red if seed % 2 else 1
        A[np.arange(n), np.arange(n)] = np.where(rng.random(n) < 0.7, red, np.array(seed % 3 != 0, dtype))
        M = sp.csr_matrix(A)
        S, fl = O.rb_matmul_csr(M, M)
        assert not fl & 7
        D = DeviceCSR.from_scipy(M)
        C, rc, _ = spgemm(D, D, R=D)
        assert rc == 0 and _cells(C.to_scipy()) == _merged(M, S), (n, family, seed)


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.uint32, np.uint64])
@pytest.mark.parametrize("n, family", [(2, 2), (64, 64), (65, 64), (300, 50), (256, 100)])
def test_columns_in_any_order(native, dtype, n, family):
    """Every row's columns descending, shuffled, or ascending in most rows: the same matrix."""
    from redblackgraph_gb300.spgemm import spgemm
    rng = np.random.default_rng([n, family])
    rows = []
    for i in range(n):
        f = i // family * family
        to = rng.choice(np.arange(f, min(f + family, n)), min(3, min(f + family, n) - f), replace=False)
        rows.append(sorted({int(c): int(rng.integers(2, 9)) for c in to if c != i}.items() | {(i, 1)}))
    B = _csr(rows, n, dtype)
    want = spgemm(B, B, R=B)
    shuffled = [[r[k] for k in rng.permutation(len(r))] for r in rows]
    few = [r[::-1] if i % 17 == 1 else r for i, r in enumerate(rows)]
    for other in ([r[::-1] for r in rows], shuffled, few):
        A = _csr(other, n, dtype)
        got = spgemm(A, A, R=A)
        assert got[1:] == want[1:] and _cells(got[0].to_scipy()) == _cells(want[0].to_scipy())


@pytest.mark.parametrize("n", [1, 8, 5000, 130_003])
def test_rows_left_to_the_warps(native, n):
    """Values past 32 bits in every row: all rows go to the warp kernel, several at a time when many."""
    from redblackgraph_gb300.spgemm import DeviceCSR, spgemm
    rng = np.random.default_rng(n)
    i = np.arange(n)
    r = np.repeat(i, 2)
    c = np.maximum(r - rng.integers(0, 40, r.size), 0)
    k = np.unique(r * n + c)
    A = sp.csr_matrix((rng.integers(2, 5, k.size), (k // n, k % n)), shape=(n, n))
    big = A.copy()
    big.data = big.data + (1 << 33)
    S, fl = O.rb_matmul_csr(big, A)
    S.sort_indices()
    C, rc, _ = spgemm(DeviceCSR.from_scipy(big), DeviceCSR.from_scipy(A))
    got = C.to_scipy()
    assert not fl & 7 and rc == 0 and (got.indptr == S.indptr).all()
    assert (got.indices == S.indices).all() and (got.data == S.data).all()
