"""The way back from the cooperative Lanczos steps (csrc/cycle.cuh): a grid barrier that gives up
(MOMED_COOP=2: every launch finds the flag that a barrier sets) and a launch that the driver refuses
(MOMED_COOP=3) end in the separate kernels, with the values of a solve that ran them from the start.

Bars: 1e-10 relative to the separate kernels (MOMED_COOP=0), the solvers' target.  The launches say which
kernels ran: a step takes one or two in cooperative form, nine or ten in separate ones.
"""
import os
from contextlib import contextmanager

import numpy as np
import pytest

import momed
from momed import _lib
from momed.core import pair_operator
from momed.synthetic import mesh_para

pytestmark = pytest.mark.gpu


@contextmanager
def env(**kv):
    old = {k: os.environ.get(k) for k in kv}
    os.environ.update({k: str(v) for k, v in kv.items()})
    try:
        yield
    finally:
        for k, v in old.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v


@pytest.fixture(scope="module")
def h():
    para, _ = mesh_para(3, 7, 2)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    hd = momed.Handle(0)
    secs = hd.enumerate_basis(para.k_list, para.Gk, 1, 1, (7,))
    hd.set_basis(secs[4][1])
    hd.set_scatter_pair(*pair_operator(A, B))
    yield hd
    hd.close()


def solve(h, kind, prec):
    n0 = _lib.kernel_launches()
    if kind == "sweep":
        v, _, _, info = h.batch_solve(np.linspace(0.7, 1.4, 5), 3, krylovdim=24, tol=1e-12, precision=prec)
    else:
        v, _, _, info = h.eigsolve(3, krylovdim=24, tol=1e-12, precision=prec, want_vectors=False)
    return np.asarray(v), (_lib.kernel_launches() - n0) / info["matvecs"], info


@pytest.mark.parametrize("kind,prec", [("hits", _lib.PREC_FP64), ("pairs", _lib.PREC_FP64), ("csr", _lib.PREC_FP64),
                                       ("hits", _lib.PREC_MIXED), ("pairs", _lib.PREC_MIXED),
                                       ("sweep", _lib.PREC_FP64), ("sweep", _lib.PREC_MIXED)])
def test_separate_kernels_take_over(h, kind, prec):
    h.release_hit_cache()
    if kind == "csr":
        h.build_sparse()
    with env(MOMED_PAIRMAP=1 if kind == "pairs" else 0):
        solve(h, kind, prec)                                # builds the tables
        coop, few, _ = solve(h, kind, prec)
        with env(MOMED_COOP=0, MOMED_GRAPHS=0):
            ref, many, i0 = solve(h, kind, prec)
        assert np.max(np.abs(coop - ref) / np.abs(ref)) < 1e-10
        for sw in (2, 3):
            with env(MOMED_COOP=sw):
                v, n, info = solve(h, kind, prec)
            assert np.max(np.abs(v - ref) / np.abs(ref)) < 1e-10
            assert info["converged"] == i0["converged"]
            assert few < 0.6 * many and n > 0.7 * many      # the cycle that gave up counts its maps twice
    if kind == "csr":
        h.release_sparse()
