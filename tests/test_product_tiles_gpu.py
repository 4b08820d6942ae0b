"""The tiled AVOS product at the edges of its tiles, chunks and reduction splits, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (3, 65, 2), (127, 31, 129), (128, 32, 128), (129, 33, 127), (64, 300, 200), (260, 515, 140)]


def _operands(m, q, p, dtype, kind, seed):
    rng = np.random.default_rng(seed)
    info = np.iinfo(dtype)
    red = np.array(-1, np.int64).astype(dtype)
    # the largest clean value: two such MSBs stay below the top bit
    small = 1 << max(1, min(info.bits, 32) // 2 - 2)
    a = rng.integers(2, small + 1, (m, q)).astype(dtype)
    b = rng.integers(2, small + 1, (q, p)).astype(dtype)
    a[rng.random((m, q)) < 0.7] = 0
    b[rng.random((q, p)) < 0.7] = 0
    if kind in ("identities", "wide"):
        for x in (a, b):
            x[rng.random(x.shape) < 0.1] = 1
            x[rng.random(x.shape) < 0.1] = red
    if kind == "wide":     # a few values that need the full scalar semantics in their tiles
        a[rng.random((m, q)) < 0.001] = info.max
        b[-1, -1] = info.max // 2 + (0 if info.min < 0 else 1)
        a[0, 0] = small
    return a, b


@pytest.mark.parametrize("kind", ["plain", "identities", "wide"])
@pytest.mark.parametrize("dtype", [np.int8, np.uint8, np.int16, np.uint16, np.int32, np.uint32, np.int64, np.uint64])
def test_product_tiles(native, dtype, kind):
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.core.avos import matmul_device
    from redblackgraph_gb300.device import to_device, to_host
    for k, (m, q, p) in enumerate(SHAPES):
        a, b = _operands(m, q, p, dtype, kind, 100 + k)
        C, st, fl = O.matmul(a, b)
        out, rc, flags = matmul_device(to_device(a), to_device(b))
        G = to_host(out)
        assert (rc == _lib.RBG_ERR_OVERFLOW) == (st != 0), (m, q, p, rc, st)
        assert (G == C).all(), (m, q, p)
        assert flags & 7 == fl & 7, (m, q, p, flags, fl)


def test_product_strided(native):
    """Row strides and bases without 16-byte alignment, output included."""
    import ctypes
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.device import to_device, to_host, stream_handle
    m, q, p = 131, 70, 133
    a, b = _operands(m, q, p, np.int32, "identities", 7)
    C, _, _ = O.matmul(a, b)
    da = torch.zeros(m * (q + 3) + 1, dtype=torch.int32, device="cuda")[1:]
    db = torch.zeros(q * (p + 1) + 2, dtype=torch.int32, device="cuda")[2:]
    dc = torch.full((m * (p + 5) + 3,), 77, dtype=torch.int32, device="cuda")[3:]
    da.view(m, q + 3)[:, :q] = to_device(a)
    db.view(q, p + 1)[:, :p] = to_device(b)
    ws = torch.empty(256, dtype=torch.uint8, device="cuda")
    flags = ctypes.c_uint32(0)
    rc = native.rbg_avos_matmul(_lib.dtype_code(np.int32), m, q, p, da.data_ptr(), q + 3, db.data_ptr(), p + 1,
                                dc.data_ptr(), p + 5, ws.data_ptr(), 256, ctypes.byref(flags), stream_handle())
    assert rc == 0
    got = to_host(dc).reshape(m, p + 5)
    assert (got[:, :p] == C).all() and (got[:, p:] == 77).all()
