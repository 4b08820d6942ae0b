"""Batches of many rows: several rows per warp in the scan and the write, several per ticket in the
closure, both in one call with matrices of every kind; against the blocked kernels on the same
blocks, and matrix by matrix against calls of one matrix."""
import numpy as np
import pytest

from redblackgraph_gb300 import synth

pytestmark = pytest.mark.gpu

EDGES = (1, 2, 3, 7, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1031, 2050)


def _batch(repeat, dtype):
    mats = []
    for k, n in enumerate(EDGES):
        A = synth.pedigree(n, synth.generations_for(n) if n > 1 else 1, k, dtype=dtype)
        mats += [A, A[::-1, ::-1].copy()]                # below and above the diagonal
        if 2 < n < 600:
            q = np.random.default_rng(k).permutation(n)
            mats.append(A[q][:, q].copy())               # any numbering
    chain = np.diag(np.full(400, -1)).astype(dtype)
    chain[np.arange(1, 16), np.arange(15)] = 2           # as deep as values of 32 bits allow
    mats.append(chain)
    for n, rows in ((270, 270), (300, 40)):
        A = np.zeros((n, n), dtype)
        A[rows - 1, :min(rows - 1, 20)] = 2              # a row of more than 16 entries
        A[0, 0] = 1
        mats.append(A)
    cycle = np.zeros((40, 40), dtype)
    cycle[3, 4], cycle[4, 3] = 2, 3
    mats.append(cycle)
    unclean = synth.pedigree(100, 5, 3, dtype=dtype)
    unclean[50, 2] = 1
    mats.append(unclean)
    more = synth.pedigree(270, 12, 9, dtype=dtype)
    return mats + [more] * repeat


# 40: some 27000 rows, one per ticket; 900: some 260000, two per ticket
@pytest.mark.parametrize("repeat, dtype", [(40, np.int32), (40, np.int64), (900, np.int32)])
def test_large_batches(native, repeat, dtype):
    import torch

    from redblackgraph_gb300 import _lib
    from redblackgraph_gb300.dense import fw_batch, fw_dense
    from redblackgraph_gb300.device import to_device
    mats = _batch(repeat, dtype)
    order = np.random.default_rng(repeat).permutation(len(mats))
    mats = [mats[k] for k in order]
    sizes = np.array([A.shape[0] for A in mats], dtype=np.int64)
    gaps = np.random.default_rng(1).integers(0, 5, sizes.size)       # rows at every alignment
    offsets = np.concatenate([[0], np.cumsum(sizes * sizes + gaps)[:-1]])
    flat = np.zeros(int((sizes * sizes + gaps).sum()), dtype)
    for A, o in zip(mats, offsets):
        flat[o:o + A.size] = A.ravel()
    d = to_device(flat)
    slow, expect = fw_batch(d, sizes, offsets, out=torch.zeros_like(d), mode=_lib.MODE_NO_DAG)
    W, res = fw_batch(d, sizes, offsets, out=torch.zeros_like(d))
    for A, o, r, e in zip(mats, offsets, res, expect):
        assert (r.status, r.flags) == (e.status, e.flags)
        if e.status == 0:
            assert r.diameter == e.diameter
            assert torch.equal(W[o:o + A.size], slow[o:o + A.size]), A.shape
    W = d.clone()
    fw_batch(W, sizes, offsets, out=W)                               # in place
    seen = set()
    for A, o, r, e in zip(mats, offsets, res, expect):
        if e.status == 0:
            assert torch.equal(W[o:o + A.size], slow[o:o + A.size]), A.shape
        if id(A) not in seen:                                        # the same route's counts, one by one
            seen.add(id(A))
            _, one = fw_dense(to_device(A))
            assert (r.path == _lib.PATH_DAG) == (one.path == _lib.PATH_DAG), A.shape
            if r.path == _lib.PATH_DAG:
                assert (r.executed, r.diameter) == (one.executed, one.diameter), A.shape
    assert sum(r.path == _lib.PATH_DAG for r in res) >= repeat + 3 * len(EDGES) - 10
