"""Relationship lookups over row lengths, alignments and storage types, against numpy's first minimum."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.int8, np.uint8, np.int16, np.uint16, np.int32, np.uint32, np.int64, np.uint64])
def test_lookup_rows(native, dtype):
    from redblackgraph_gb300.device import to_device
    from redblackgraph_gb300.relationship import Relationship, lookup_many, msb, relationship_name
    rng = np.random.default_rng(3)
    info = np.iinfo(dtype)
    queries, expect = [], []
    for n in (1, 3, 4, 31, 127, 128, 130, 515, 2049):
        W = rng.integers(0, 100, (6, n + 3)).astype(dtype)
        W[rng.random(W.shape) < 0.5] = 0
        W[0, ::3] = info.max                           # sums that wrap
        W[1, ::2] = np.array(-1, np.int64).astype(dtype)
        d = to_device(W)
        for shift in (0, 1):                           # rows on and off 16-byte boundaries
            M, D = W[:, shift:shift + n], d[:, shift:shift + n]
            for u in range(6):
                for v in range(6):
                    queries.append((D, u, v))
                    a, b = M[u], M[v]
                    both = np.flatnonzero((a != 0) & (b != 0))
                    if both.size == 0:
                        expect.append(Relationship(-1, "No Relationship"))
                        continue
                    with np.errstate(over="ignore"):
                        j = both[np.argmin(a[both] + b[both])]
                    expect.append(Relationship(int(j), relationship_name(msb(a[j]), msb(b[j]))))
    assert lookup_many(queries) == expect
    W = torch.zeros((2, 4), dtype=torch.int32, device="cuda")
    for bad in ((W, 0, 2), (W, -1, 0)):
        with pytest.raises(IndexError):
            lookup_many([(W, 0, 1), bad])
    with pytest.raises(ValueError):
        lookup_many([(W[0], 0, 0)])
