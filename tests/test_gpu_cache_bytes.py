"""The bytes that momed_hit_cache_info reports are those of what the cache has built: the pair tables with
their workspace, the hit records, or both."""
import pytest

import momed
from momed.core import pair_operator
from momed.synthetic import mesh_para

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["tables", "records", "both"])
def test_reported_bytes(form, monkeypatch):
    monkeypatch.setenv("MOMED_PAIRMAP", "0" if form == "records" else "1")
    para, _ = mesh_para(3, 9, 2)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    h = momed.Handle(0)
    (_, basis), = h.enumerate_basis(para.k_list, para.Gk, 1, 1, (9,), momentum_list=[(1, 4)])
    h.set_basis(basis)
    h.set_scatter_pair(*pair_operator(A, B))
    n, entries = len(basis), len(basis) * 36
    info = h.build_hit_cache()
    if form == "both":
        h.batch_solve([1.0, 1.1], 1, krylovdim=4, maxiter=1)
        info = h.hit_cache_info()
    records, tables = info["hits"] * 8 + (n + 1) * 8 + n * 56, entries * (4 + 16)
    h.close()
    if form == "records":
        assert info["bytes"] == records
    else:                                          # row_ent and the workspace, and at most 2.5 slots per entry
        rest = info["bytes"] - (records if form == "both" else 0) - tables
        assert entries * 4 <= rest <= entries * 10
