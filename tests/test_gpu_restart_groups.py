"""Restart recombination (csrc/vecops.cu) where its groups of outputs change: a warp per group of 4 up to 32
kept vectors (3 krylovdim / 5), groups of 8 from 33, on tiles of 64 rows with a remainder.

Bars: eigenvalues within 1e-10 relative of LAPACK, vectors orthonormal to 1e-9 (those of the other sizes,
test_gpu_restart_and_scan.py).
"""
import numpy as np
import pytest

import momed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylovdim,nev", [(52, 5), (54, 5), (54, 32), (55, 5), (55, 33), (57, 34)])   # 31, 32, 33, 34 kept
def test_restart_recombination_at_the_change(krylovdim, nev):
    import scipy.sparse as sps
    n = 1201
    rng = np.random.default_rng(n)
    a = sps.random(n, n, 12.0 / n, random_state=n, data_rvs=rng.standard_normal).tocsr()
    m = sps.csr_matrix((a + a.conj().T) / 2 + 1j * (a - a.T) / 4 + sps.diags(rng.uniform(-1, 1, n)))
    m.sort_indices()
    w = np.linalg.eigvalsh(m.toarray())
    h = momed.Handle(0)
    h.set_sparse_csr(m.indptr, m.indices, m.data)
    vals, vecs, resid, info = h.eigsolve(nev, krylovdim=krylovdim, tol=1e-12, seed=5, maxiter=500)
    h.close()
    assert info["converged"] == nev and info["restarts"] >= 1
    assert np.max(np.abs(vals - w[:nev]) / np.maximum(np.abs(w[:nev]), 1.0)) < 1e-10
    assert np.max(np.abs(vecs.conj() @ vecs.T - np.eye(nev))) < 1e-9
