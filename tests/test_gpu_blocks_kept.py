"""Blocks a handle keeps for its next solve: the same results with blocks kept, given back (a budget)
and taken by solves of other sizes in turn, on several handles and threads."""
import threading

import numpy as np
import pytest

import momed
from momed.core import pair_operator
from momed.synthetic import mesh_para

pytestmark = pytest.mark.gpu


def test_solves_of_changing_size_on_several_handles():
    para, _ = mesh_para(3, 8, 0)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    pair = pair_operator(A, B)
    h = momed.Handle(0)
    secs = {ne: h.enumerate_basis(para.k_list, para.Gk, 1, 1, (ne,))[3][1] for ne in (4, 6, 8)}
    h.close()
    ref = {}

    def solve(hd, ne, nev):
        hd.set_basis(secs[ne])
        return hd.eigsolve(nev, krylovdim=30, tol=1e-12, seed=1, want_vectors=False)[0]

    def work(out, order):
        hd = momed.Handle(0)
        hd.set_scatter_pair(*pair)
        for k, (ne, nev) in enumerate(order):
            if k == 3:
                hd.set_hbm_budget(1 << 36)       # gives the kept blocks back
                hd.set_hbm_budget(0)
            out.append((ne, nev, solve(hd, ne, nev)))
            if nev == 3:
                hd.set_basis(secs[ne])
                out.append((ne, 2, hd.batch_solve([1.0, 1.0, 1.0], 2, krylovdim=30, tol=1e-12)[0][1]))
        hd.close()

    order = [(8, 2), (4, 3), (6, 2), (8, 3), (6, 3), (4, 2), (8, 2), (6, 2)]
    outs = [[] for _ in range(3)]
    threads = [threading.Thread(target=work, args=(o, order[i:] + order[:i])) for i, o in enumerate(outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(len(o) == 11 for o in outs)
    for o in outs:
        for ne, nev, vals in o:
            got = np.asarray(vals)[:2]
            first = ref.setdefault(ne, got)
            assert np.max(np.abs(got - first)) < 1e-10 * np.max(np.abs(first))
