"""Component-wise closure of a graph with rows that wait for their parents, against the closure by
levels with the statistics kernel on the same graph."""
import numpy as np
import pytest
import scipy.sparse as sp

from redblackgraph_gb300 import synth

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 31, 33, 65, 129, 300, 1025, 2050, 64, 700)


def _graph(repeat, above=False, wide=0, spread=False):
    """Pedigrees side by side, every second one upside down when `above`; `wide`: entries of one row;
    `spread`: the last component's vertices around all others."""
    blocks = []
    for r in range(repeat):
        for k, n in enumerate(SIZES):
            A = synth.pedigree(n, synth.generations_for(n) if n > 1 else 1, 7 * r + k, dtype=np.int32)
            blocks.append(sp.csr_matrix(A[::-1, ::-1] if above and k % 2 else A))
    if wide:
        A = np.diag(np.full(60, -1)).astype(np.int32)
        A[50, :wide] = 2
        blocks.append(sp.csr_matrix(A))
    F = sp.block_diag(blocks, format="csr", dtype=np.int32)
    if spread:                                           # the last component's first vertex goes first
        q = np.r_[F.shape[0] - SIZES[-1], np.arange(F.shape[0] - SIZES[-1]), np.arange(F.shape[0] - SIZES[-1] + 1, F.shape[0])]
        F = F[q][:, q]
    F.sort_indices()
    return F


# 3: a row per ticket; 50: 220000 rows, two per ticket.  `taken`: whether the rows are closed this way
@pytest.mark.parametrize("kw, taken", [(dict(repeat=3), True), (dict(repeat=3, above=True), True),
                                       (dict(repeat=50), True), (dict(repeat=2, wide=16), True),
                                       (dict(repeat=2, wide=17), False), (dict(repeat=3, spread=True), False)])
def test_component_rows(native, monkeypatch, kw, taken):
    from redblackgraph_gb300 import components
    from redblackgraph_gb300.sparse import component_wise_closure
    F = _graph(**kw)
    rows, seen = components._close_rows, []

    def watched(*a):
        seen.append(rows(*a) is not None)
        return rows(*a)
    monkeypatch.setattr(components, "_close_rows", watched)
    got = [component_wise_closure(F, method=m) for m in ("FW", "D")]
    assert seen == [taken] * 2
    monkeypatch.setattr(components, "_close_rows", lambda *a: None)
    for g, m in zip(got, ("FW", "D")):
        e = component_wise_closure(F, method=m)
        assert g.diameter == e.diameter
        for x, y in ((g.W.indptr, e.W.indptr), (g.W.indices, e.W.indices), (g.W.data, e.W.data)):
            assert np.array_equal(x, y)
