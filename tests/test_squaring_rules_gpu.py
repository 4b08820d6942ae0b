"""Squaring steps where the tiles' and groups' shortcuts must not show: columns stored twice."""
import numpy as np
import pytest

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
