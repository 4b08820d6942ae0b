"""Closures of matrices in a topological order whose rows are too wide for the DAG path (block row by
block row), below and above the diagonal, at the edges of the blocks, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _layered(n, layers, p, seed, dtype, hi=4):
    rng = np.random.default_rng(seed)
    layer = np.sort(rng.integers(0, layers, n))
    link = (layer[:, None] > layer[None, :]) & (rng.random((n, n)) < p)
    A = np.where(link, rng.integers(2, hi, (n, n)), 0).astype(dtype)
    np.fill_diagonal(A, rng.choice([-1, 0, 1], n))
    return A


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_wide_rows(native, dtype):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_dense
    from redblackgraph_gb300.device import to_device, to_host
    for n, layers, p, hi in ((40, 6, 0.9, 4), (127, 8, 0.5, 4), (128, 8, 0.5, 9), (129, 20, 0.5, 4), (256, 4, 0.3, 64),
                             (300, 12, 0.3, 4), (385, 25, 0.2, 4), (700, 10, 0.05, 4), (1025, 9, 0.5, 4)):
        A = _layered(n, layers, p, n, dtype, hi)
        assert ((A != 0).sum(1) > 17).any()
        for M in (A, A[::-1, ::-1].copy()):                 # below, then above the diagonal
            semantics = ((0, O.warshall), (_lib.MODE_CYTHON, O.fw_cython)) if dtype == np.int32 else ((0, O.warshall),)
            for mode, oracle in semantics:
                Wo, do, so, _ = oracle(M)
                d = to_device(M)
                for out in (None, d):                       # out of place, then in place
                    W, r = fw_dense(d, out=out, mode=mode)
                    assert r.status == so == 0 and r.diameter == do, (n, mode)
                    assert (to_host(W) == Wo).all(), (n, mode)
                    assert r.path == _lib.PATH_BLOCKED32


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_wide_rows_leave_the_path(native, dtype):
    """Products reaching the top bit, a cycle, an unclean value and padded strides."""
    import ctypes
    import torch
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_dense
    from redblackgraph_gb300.device import to_device, to_host, stream_handle
    n = 200
    deep = _layered(n, n, 0.5, 3, dtype)                    # paths of tens of edges
    big = _layered(n, 4, 0.5, 4, dtype, hi=1 << 14)
    odd = _layered(n, 6, 0.5, 5, dtype)
    odd[150, 3] = 1
    for M in (deep, deep[::-1, ::-1].copy(), big, big[::-1, ::-1].copy(), odd):
        Wo, do, so, _ = O.warshall(M)
        W, r = fw_dense(to_device(M))
        assert r.status == so
        if so == 0:
            assert (to_host(W) == Wo).all() and r.diameter == do
    A = _layered(301, 9, 0.4, 6, dtype)
    Wo, do, _, _ = O.warshall(A)
    buf = torch.zeros((301, 309), dtype=to_device(A).dtype, device="cuda")
    out = torch.full((301, 305), 7, dtype=buf.dtype, device="cuda")
    buf[:, :301] = to_device(A)
    L, nb = _lib.load(), ctypes.c_int64(0)
    code = _lib.dtype_code(np.dtype(dtype))
    L.rbg_fw_dense_workspace_bytes(code, 301, 0, ctypes.byref(nb))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    res = _lib.RbgResult()
    assert L.rbg_fw_dense(code, 301, buf.data_ptr(), 309, out.data_ptr(), 305, 0, ws.data_ptr(), ws.numel(),
                          ctypes.byref(res), stream_handle()) == 0
    got = to_host(out)
    assert res.status == 0 and res.diameter == do and (got[:, :301] == Wo).all() and (got[:, 301:] == 7).all()
