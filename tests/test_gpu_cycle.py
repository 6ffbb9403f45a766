"""The cooperative Lanczos steps (csrc/cycle.cu) against LAPACK, or, where the matrix is too large for
it, against the separate kernels (MOMED_COOP=0), at the edges of its row blocks: sectors of one row
to one block, the first row of a further block, the sizes where a block's projections are split in
chunks and its updates over 4, 2 and 1 lanes, and both maps inside the kernel (hit records, CSR) and
the one beside it (pair tables).

Bars: eigenvalues within 1e-10 relative of LAPACK; against the separate kernels 1e-11 (both converge
to residual 1e-12); residuals <= 1e-10 max(1, |E|).
"""
import os
from contextlib import contextmanager

import numpy as np
import pytest
import scipy.sparse as sps

import oracle as O
import momed
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
    hd = momed.Handle(0)
    yield hd
    hd.close()


def matrix(n, seed):
    """A sparse Hermitian matrix with separated low eigenvalues: a few diagonal wells below a band."""
    rng = np.random.default_rng(seed)
    d = rng.uniform(0.0, 4.0, n)
    d[rng.permutation(n)[:min(n, 8)]] -= 3.0 + np.arange(min(n, 8))
    k = min(3 * n, 3 * n)
    i, j = rng.integers(0, n, k), rng.integers(0, n, k)
    v = 0.2 * (rng.standard_normal(k) + 1j * rng.standard_normal(k))
    off = sps.coo_matrix((v, (i, j)), (n, n)).tocsr()
    m = (off + off.conj().T) / 2 + sps.diags(d)
    m = sps.csr_matrix(m)
    m.sort_indices()
    return m


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 64, 97, 1000, 148 * 32, 148 * 32 + 1])
def test_csr_steps_vs_lapack(h, n):
    m = matrix(n, n)
    h.set_sparse_csr(m.indptr, m.indices, m.data)
    nev = min(n, 4)
    vals, vecs, resid, info = h.eigsolve(nev, krylovdim=24, tol=1e-12, seed=3)
    if n <= 1000:
        w = np.linalg.eigvalsh(m.toarray())[:nev]
    else:
        with env(MOMED_COOP=0):
            w, _, _, _ = h.eigsolve(nev, krylovdim=24, tol=1e-12, seed=3)
    assert np.max(np.abs(vals - w) / np.maximum(np.abs(w), 1.0)) < 1e-10
    for i in range(nev):
        r = np.linalg.norm(m @ vecs[i] - vals[i] * vecs[i])
        assert r <= 1e-10 * max(1.0, abs(vals[i])) and abs(np.linalg.norm(vecs[i]) - 1.0) < 1e-12
    h.release_sparse()


# chunked projections from 256 rows a block, 4 / 2 / 1 lanes per row up to 512 / 2048 / more
@pytest.mark.parametrize("rows", [255, 256, 512, 513, 2048, 2049])
def test_csr_steps_vs_separate_kernels(h, rows):
    n = 148 * rows - 5
    m = matrix(n, rows)
    h.set_sparse_csr(m.indptr, m.indices, m.data)
    vals, _, resid, info = h.eigsolve(3, krylovdim=20, tol=1e-12, seed=4, want_vectors=False)
    with env(MOMED_COOP=0):
        ref, _, _, i0 = h.eigsolve(3, krylovdim=20, tol=1e-12, seed=4, want_vectors=False)
    assert np.max(np.abs(vals - ref) / np.abs(ref)) < 1e-11
    assert np.max(resid) <= 1e-10 * np.max(np.abs(vals))
    assert info["converged"] == 3 and abs(info["restarts"] - i0["restarts"]) <= 1
    h.release_sparse()


@pytest.mark.parametrize("pairs", [0, 1])
def test_hit_and_pair_maps_vs_lapack(h, pairs):
    """The map over the hit records inside the kernel, and the pair map beside it, H(u) included."""
    para, _ = mesh_para(3, 6, 0)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    amp_a, amp_b, in_, out, pm = momed.core.pair_operator(A, B)
    subs, _ = O.momentum_subspaces(O.mesh_klist(3, 6), (3, 6), (6,))
    f = np.zeros(len(in_), O.SCAT_DTYPE)
    with env(MOMED_PAIRMAP=pairs):
        for s, u in ((2, 1.0), (7, 0.6)):
            h.set_basis(subs[s])
            h.set_scatter_pair(amp_a, amp_b, in_, out, pm)
            h.set_param(u)
            amp = amp_a + u * amp_b
            f["re"], f["im"], f["out"], f["in"], f["pm"] = amp.real, amp.imag, out, in_, pm
            w = np.linalg.eigvalsh(O.dense_hamiltonian(subs[s], f))[:5]
            n0 = momed._lib.kernel_launches()
            vals, vecs, resid, info = h.eigsolve(5, krylovdim=30, tol=1e-12, seed=2)
            launches = momed._lib.kernel_launches() - n0
            assert np.max(np.abs(vals - w) / np.abs(w)) < 1e-10 and np.max(resid) < 1e-10
            # a cycle in one launch, or three per step
            assert launches < (60 + 4 * info["restarts"] if pairs == 0 else 60 + 5 * info["matvecs"])
    h.set_param(1.0)


def test_invariant_subspace_inside_a_cycle(h):
    """A start vector in a small invariant subspace: the recurrence ends inside the first cycle and goes
    on from fresh directions."""
    n = 400
    d = np.linspace(-2.0, 3.0, n)
    m = sps.csr_matrix(sps.diags(d + 0j))
    h.set_sparse_csr(m.indptr, m.indices, m.data)
    v0 = np.zeros(n, np.complex128)
    v0[[3, 50, 200]] = 1.0
    vals, _, resid, _ = h.eigsolve(4, krylovdim=30, tol=1e-12, vec0=v0, maxiter=200)
    with env(MOMED_COOP=0):
        ref, _, _, _ = h.eigsolve(4, krylovdim=30, tol=1e-12, vec0=v0, maxiter=200)
    assert np.max(np.abs(vals - ref)) < 1e-10 and np.max(resid) < 1e-9
    h.release_sparse()
