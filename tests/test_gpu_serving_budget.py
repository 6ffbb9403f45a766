"""A served solve is charged for the map cache that it builds: the pair tables, or the hit records where the
tables are declined (too few free pairs per state), not for the estimate that admitted it."""
import re

import pytest

import momed
from momed import _lib
from momed.core import pair_operator
from momed.synthetic import mesh_para

pytestmark = pytest.mark.gpu


def serve(budget, pair, basis):
    """The budget in use, as seen while the request runs."""
    srv = _lib.Server(0, slots=1, hbm_budget=budget)
    try:
        rid = srv.submit(srv.register_operator(*pair), basis, 1.1, 4, tol=1e-12, precision=_lib.PREC_FP64)
        seen, st = set(), None
        while st != _lib.DONE:
            for _ in range(50):
                seen.add(srv.stats()["hbm_used"])
            st = srv.poll(rid, 4)[0]
        assert srv.stats()["hbm_used"] == 0
        return seen
    finally:
        srv.stop()


# 6 hits per entry: pair tables; 3.4 (half filled): the records
@pytest.mark.parametrize("a,b,ne", [(3, 9, 9), (4, 6, 11)])
def test_charged_for_what_is_built(a, b, ne):
    para, _ = mesh_para(a, b, 3)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    pair = pair_operator(A, B)
    h = momed.Handle(0)
    (_, basis), = h.enumerate_basis(para.k_list, para.Gk, 1, 1, (ne,), momentum_list=[(1, 2)])
    h.set_basis(basis)
    h.set_scatter_pair(*pair)
    cache = h.build_hit_cache()["bytes"]
    h.close()
    with pytest.raises(Exception) as e:            # what the request itself needs
        serve(1 << 20, pair, basis)
    need = int(re.search(r"needs (\d+) bytes", str(e.value)).group(1))
    assert need + cache in serve(1 << 34, pair, basis)
