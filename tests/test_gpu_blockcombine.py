"""The recombinations of the lockstep block solver (csrc/blockcombine.cu) and its Gram blocks
(csrc/blockgram.cu: 5 to 24 FP64 columns, 11 to 46 FP32 ones, so one pass of 32 columns and two) against
LAPACK at the edges of their tiles: 1 to 20 wanted pairs (kept combinations and Ritz vectors of one tile, a full one,
two and three), bases that are no multiple of a run of sources, an odd and an even number of rows, and
block widths with one and two values per packet, in both precisions.

Bars: eigenvalues within 1e-10 relative; vectors of the wanted pairs satisfy |H x - E x| <= 1e-6
max(1, |E|) in both forms (the mixed form stops on the eigenvalue's error).
"""
import numpy as np
import pytest

import momed
from momed import _lib
from test_gpu_blockstep import eigs, setup, _eigs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    hd = momed.Handle(0)
    yield hd
    hd.close()


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("nu", [1, 2, 7, 32])
@pytest.mark.parametrize("nev,m", [(1, 18), (2, 23), (4, 25), (5, 31), (8, 40), (11, 45), (14, 60), (20, 70)])
@pytest.mark.parametrize("sec", [(3, 6, 5, 0), (4, 4, 5, 3)])
def test_wanted_pairs(h, sec, nev, m, nu, prec):
    basis, *ops = setup(h, *sec)
    u = np.linspace(0.5, 1.5, nu)
    v, x, _, _ = h.batch_solve(u, nev, krylovdim=m, tol=1e-11, maxiter=300, precision=prec, want_vectors=True)
    ref = eigs(sec, basis, *ops, u)[:, :nev]
    assert np.max(np.abs(v - ref) / np.maximum(1, np.abs(ref))) < 1e-10
    a, b = _eigs[sec]
    for q in {0, nu - 1}:
        r = (a + u[q] * b) @ x[q].T - x[q].T * v[q]
        assert np.max(np.linalg.norm(r, axis=0) / np.maximum(1, np.abs(v[q]))) < 1e-6
