"""A served solve takes the map cache that its budget holds: a sector whose states have too few free pairs
for the pair tables gets the hit records when those fit, not the slower forms after them because the tables'
(larger) estimate does not."""
import re
import time

import numpy as np
import pytest

import momed
from momed import _lib
from momed.core import pair_operator
from momed.synthetic import mesh_para

pytestmark = pytest.mark.gpu


def serve(budget, pair, basis, nev):
    srv = _lib.Server(0, slots=1, hbm_budget=budget)
    try:
        op = srv.register_operator(*pair)
        n0 = _lib.kernel_launches()
        rid = srv.submit(op, basis, 1.1, nev, tol=1e-10, precision=_lib.PREC_FP64)
        t0 = time.time()
        while time.time() - t0 < 120:
            st, vals, resid, info, _, _ = srv.poll(rid, nev, wait_ms=100)
            if st == _lib.DONE:
                return vals, (_lib.kernel_launches() - n0) / info["matvecs"], srv.stats()
        raise AssertionError("not served in time")
    finally:
        srv.stop()


def test_records_where_only_they_fit(monkeypatch):
    monkeypatch.setenv("MOMED_SERVE_SPARSE", "0")
    para, _ = mesh_para(4, 6, 3)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    pair = pair_operator(A, B)
    h = momed.Handle(0)
    (_, basis), = h.enumerate_basis(para.k_list, para.Gk, 1, 1, (11,), momentum_list=[(1, 2)])
    h.set_basis(basis)
    h.set_scatter_pair(*pair)
    nnz, n = h.build_sparse(), len(basis)
    h.close()
    records, tables = (n + 1) * 8 + n * 56 + nnz * 8, n * 55 * 92 // 3  # 30 2/3 bytes an entry and more
    assert records + (2 << 20) < tables
    with pytest.raises(Exception) as e:                                 # what the request itself needs
        serve(1 << 20, pair, basis, 4)
    need = int(re.search(r"needs (\d+) bytes", str(e.value)).group(1))
    vals, per_map, stats = serve(need + records + (1 << 20), pair, basis, 4)
    roomy, per_map_roomy, _ = serve(need + 2 * tables, pair, basis, 4)
    assert np.max(np.abs(vals - roomy) / np.abs(roomy)) < 1e-10
    assert per_map < 3 and per_map_roomy < 3       # a cycle per launch over the records; slots: ten launches a map
    assert stats["hbm_used"] == 0
