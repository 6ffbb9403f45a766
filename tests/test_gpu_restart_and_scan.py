"""Edges of the restart recombination (csrc/vecops.cu) and of the basis scan (csrc/index.cu).

The recombination works on groups of 4 outputs below 24 kept vectors and of 8 from there, with a
remainder, on tiles of 64 rows; the scan on batches of 32 states, two per warp, split points up to 64.

Bars: eigenvalues within 1e-10 relative of LAPACK, products within 1e-13 of the oracle.
"""
import numpy as np
import pytest

import oracle as O
import momed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    hd = momed.Handle(0)
    yield hd
    hd.close()


@pytest.fixture(scope="module")
def problem():
    import scipy.sparse as sps
    out = {}
    for n in (63, 64, 65, 1201):
        rng = np.random.default_rng(n)
        a = sps.random(n, n, 12.0 / n, random_state=int(n), data_rvs=rng.standard_normal).tocsr()
        m = sps.csr_matrix((a + a.conj().T) / 2 + 1j * (a - a.T) / 4 + sps.diags(rng.uniform(-1, 1, n)))
        m.sort_indices()
        out[n] = (m, np.linalg.eigvalsh(m.toarray()))
    return out


# kept vectors (3 krylovdim / 5): 4-groups without and with remainder, 23 / 24 at the change, 8-groups,
# the widest basis
@pytest.mark.parametrize("n,krylovdim,nev", [(63, 14, 1), (64, 14, 2), (65, 14, 5), (1201, 14, 3), (1201, 38, 4),
                                             (1201, 40, 4), (1201, 41, 24), (1201, 64, 6), (1201, 135, 30)])
def test_restart_recombination(h, problem, n, krylovdim, nev):
    m, w = problem[n]
    h.set_sparse_csr(m.indptr, m.indices, m.data)
    vals, vecs, resid, info = h.eigsolve(nev, krylovdim=krylovdim, tol=1e-12, seed=5, maxiter=500)
    assert info["converged"] == nev and info["restarts"] >= 1
    assert np.max(np.abs(vals - w[:nev]) / np.maximum(np.abs(w[:nev]), 1.0)) < 1e-10
    g = vecs.conj() @ vecs.T
    assert np.max(np.abs(g - np.eye(nev))) < 1e-9
    h.release_sparse()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 511, 512, 513, 4097])
def test_basis_scan_finds_order_and_ranges(h, n):
    """A one-body diagonal operator on n states of mixed particle numbers with orbital 63 among them:
    the product needs the right lookup tables; a fault in the order at any place is refused."""
    rng = np.random.default_rng(n)
    basis = np.unique(rng.integers(1, 1 << 63, 2 * n, dtype=np.uint64) & rng.integers(1, 1 << 63, 2 * n, dtype=np.uint64))[:n]
    basis = np.unique(np.concatenate([basis[:max(n - 1, 0)], np.array([(1 << 63) | 5], np.uint64)]))
    h.set_basis(basis)
    one = np.uint64(1) << np.arange(64, dtype=np.uint64)
    eps = rng.standard_normal(64) + 0j
    h.set_scatter(eps, one, one)
    x = rng.standard_normal(len(basis)) + 1j * rng.standard_normal(len(basis))
    occ = (basis[:, None] >> np.arange(64, dtype=np.uint64)) & np.uint64(1)
    ref = (occ @ eps.real) * x
    assert np.max(np.abs(h.matvec(x) - ref)) < 1e-13 * np.max(np.abs(ref))
    for at in {0, len(basis) // 2, len(basis) - 2}:
        if 0 <= at < len(basis) - 1:
            bad = basis.copy()
            bad[at] = bad[at + 1]
            h.set_basis(bad)
            with pytest.raises(momed.MomedError):
                h.matvec(x)


@pytest.mark.parametrize("n", [1, 31, 33, 513])
def test_rdm_of_mixed_spaces(h, n):
    """Occupations and transfers on spaces where c+_i c_j stays inside, up to orbital 63."""
    rng = np.random.default_rng(n)
    orbs = np.array([0, 1, 2, 3, 30, 31, 32, 33, 62, 63], np.uint64)
    picks = rng.permutation(1 << len(orbs))[:n]
    basis = np.unique(np.array([sum(1 << int(o) for k, o in enumerate(orbs) if p >> k & 1) for p in picks], np.uint64))
    psi = rng.standard_normal(len(basis)) + 1j * rng.standard_normal(len(basis))
    h.set_basis(basis)
    got = h.rdm1(psi, 64)
    index = {int(s): k for k, s in enumerate(basis)}
    ref = np.zeros((64, 64), complex)
    for x, s in enumerate(map(int, basis)):
        for j in map(int, orbs):
            if not s >> j & 1:
                continue
            mid = s & ~(1 << j)
            for i in map(int, orbs):
                if mid >> i & 1:
                    continue
                y = index.get(mid | 1 << i)
                if y is not None:
                    sign = (-1) ** (bin(mid >> (i + 1)).count("1") + bin(mid >> (j + 1)).count("1"))
                    ref[i, j] += sign * np.conj(psi[y]) * psi[x]
    assert np.max(np.abs(got - ref)) < 1e-12 * max(1.0, np.max(np.abs(ref)))
