"""Products that leave the lanes, at the edges of the quarters their tiles are redone in and of the
reduction's parts, against the oracle: values, status and events."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _operand(rng, shape, dtype, kind):
    info = np.iinfo(dtype)
    A = np.where(rng.random(shape) < 0.5, rng.integers(2, 7, shape), 0)
    A = A.astype(dtype)
    at = tuple(rng.integers(0, n, 3) for n in shape)
    if kind == "top":                                    # products at and past the top bit
        A[at] = info.max // 2 + 1 if info.min == 0 else 1 << (info.bits - 3)
    if kind == "identities":
        A[at] = 1
        A[tuple(rng.integers(0, n, 3) for n in shape)] = np.array(-1, np.int64).astype(dtype)
        A[0, 0] = info.max - 1                           # off the lanes, whatever the type
    if kind == "negative" and info.min < 0:
        A[at] = -2
    if kind == "wide":
        A[at] = info.max >> 2
    return A


@pytest.mark.parametrize("kind", ["top", "identities", "negative", "wide"])
@pytest.mark.parametrize("dtype", [np.int8, np.uint8, np.int16, np.uint16, np.int32, np.uint32, np.int64, np.uint64])
def test_redone_tiles(native, dtype, kind):
    import torch
    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.core.avos import matmul_device
    from redblackgraph_gb300.device import to_device, to_host
    for m, q, p in ((1, 1, 1), (2, 31, 3), (63, 33, 64), (64, 32, 65), (65, 64, 63), (128, 130, 129), (129, 7, 128),
                    (70, 600, 200), (3, 1100, 70)):
        rng = np.random.default_rng([m, q, p, ord(kind[0])])
        a, b = _operand(rng, (m, q), dtype, kind), _operand(rng, (q, p), dtype, kind)
        C, st, fl = O.matmul(a, b)
        got, rc, flags = matmul_device(to_device(a), to_device(b))
        bits = _lib.EV_OVF_SIZE | _lib.EV_OVF_ONES | _lib.EV_HANG
        assert (rc != 0) == (st != 0) and (flags & bits) == (fl & bits), (m, q, p, rc, st, flags, fl)
        if not fl & _lib.EV_HANG:
            assert (to_host(got) == C).all(), (m, q, p)
