"""Sparse products and squaring steps over the row classes of the kernels (tiles of families, short
rows, wide windows, values outside the 32-bit rules), against the oracle's product."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _random(n, family, per_row, seed, dtype, kind):
    """Blocks of `family` vertices with about `per_row` entries below the diagonal in the block;
    diagonal +-1.  kind: "plain" (values 2 .. 99), "ones" (identities off the diagonal as well, and a
    stored zero), "large" (a few products past bit 31)."""
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), per_row)
    first = rows // family * family
    cols = first + (rng.random(rows.size) * np.maximum(rows - first, 1)).astype(np.int64)
    keep = cols < rows
    vals = rng.integers(2, 100, rows.size)
    if kind == "ones":
        one = rng.random(rows.size) < 0.1
        vals[one] = np.where(rng.random(int(one.sum())) < 0.5, 1, -1)
        vals[rng.integers(rows.size)] = 0
    if kind == "large":
        vals[rng.random(rows.size) < 0.02] = 1 << 24
    M = sp.coo_matrix((vals[keep], (rows[keep], cols[keep])), shape=(n, n))
    D = {}
    for r, c, v in zip(M.row.tolist(), M.col.tolist(), M.data.tolist()):
        D[r, c] = v
    for v in range(n):
        D[v, v] = int(rng.choice([-1, 1]))
    keys = sorted(D)
    A = sp.csr_matrix((np.array([D[k] for k in keys], np.int64),
                       (np.array([k[0] for k in keys]), np.array([k[1] for k in keys]))), shape=(n, n))
    A.has_sorted_indices = True
    return sp.csr_matrix((A.data.astype(dtype), A.indices, A.indptr), shape=(n, n))


def _cells(m):
    m = m.tocoo()
    return {(r, c): v for r, c, v in zip(m.row.tolist(), m.col.tolist(), m.data.tolist())}


def _merged(R, S, dtype):
    """R (+) R^2 by magnitude (R's value on a tie), as int32."""
    uns = np.dtype(dtype).kind == "u"
    mag = (lambda v: v) if uns else abs
    out, s = {}, _cells(S)
    for k, r in _cells(R).items():
        v = s.get(k, 0)
        out[k] = v if v != 0 and (r == 0 or mag(v) < mag(r)) else r
    for k, v in s.items():
        out.setdefault(k, v)
    out = {k: int(np.array(v, dtype).astype(np.int32)) for k, v in out.items()}
    return {k: v for k, v in out.items() if v != 0}


@pytest.mark.parametrize("kind", ["plain", "ones", "large"])
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.uint32, np.uint64])
def test_squaring_steps_and_products(native, dtype, kind):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.spgemm import DeviceCSR, spgemm
    for n, family, per_row in ((1, 1, 1), (64, 64, 3), (300, 64, 3), (333, 50, 4), (400, 100, 3), (500, 500, 2),
                               (200, 64, 20)):
        A = _random(n, family, per_row, n + per_row, dtype, kind)
        S, fl = O.rb_matmul_csr(A, A)
        D = DeviceCSR.from_scipy(A)
        C, rc, flags = spgemm(D, D)
        assert (rc == _lib.RBG_ERR_OVERFLOW) == bool(fl & 7), (n, rc, fl)
        # (a sum that the storage type wraps to zero is not stored)
        assert _cells(C.to_scipy()) == {k: v for k, v in _cells(S).items() if v != 0}, n
        C, rc, _ = spgemm(D, D, R=D)
        assert (rc == _lib.RBG_ERR_OVERFLOW) == bool(fl & 7), (n, rc, fl)
        got = C.to_scipy()
        assert _cells(got) == _merged(A, S, dtype), (n, family)
        for r in range(n):
            assert (np.diff(got.indices[got.indptr[r]:got.indptr[r + 1]]) > 0).all()


def test_squaring_step_reports_a_cycle(native):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.spgemm import DeviceCSR, SEM_CY32, spgemm
    for n, family in ((64, 64), (640, 640)):
        A = _random(n, family, 3, 5, np.int32, "plain").tolil()
        for sem in (0, SEM_CY32):
            D = DeviceCSR.from_scipy(A.tocsr())
            assert not spgemm(D, D, R=D, sem=sem)[2] & _lib.EV_CYCLE
        A[3, n - 1], A[n - 1, 3] = 2, 3
        for sem in (0, SEM_CY32):
            D = DeviceCSR.from_scipy(A.tocsr())
            assert spgemm(D, D, R=D, sem=sem)[2] & _lib.EV_CYCLE
            assert spgemm(D, D, sem=sem)[2] & _lib.EV_CYCLE


@pytest.mark.parametrize("n, per_row", [(65, 3), (71, 64), (64, 400), (129, 400), (8, 30)])
def test_tiles_of_full_and_few_rows(native, n, per_row):
    """Rows that fill their tile below the diagonal (up to 63 entries, eight rows at a time), and last
    blocks of fewer than eight rows."""
    from redblackgraph_gb300.spgemm import DeviceCSR, spgemm
    A = _random(n, 64, per_row, n, np.int64, "plain")
    A.data[A.data > 3] = 3                                   # products of two small values: no overflow
    S, fl = O.rb_matmul_csr(A, A)
    D = DeviceCSR.from_scipy(A)
    C, rc, _ = spgemm(D, D, R=D)
    assert not fl & 7 and rc == 0
    assert _cells(C.to_scipy()) == _merged(A, S, np.int64)
