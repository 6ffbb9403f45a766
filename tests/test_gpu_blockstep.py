"""The cooperative step of the lockstep block solver (csrc/blockstep.cu) against LAPACK at the edges of
its work split: block widths 1 to 32 (ragged counts of right-hand sides included) in both precisions,
sectors of a few rows to several row blocks, bases of 8 / 9 / 16 / 17 / 64 / 65 columns (one read of
w, two, a further round); and, where LAPACK would take too long, against the separate kernels
(MOMED_COOP=0).

Bars: eigenvalues within 1e-10 relative (the solver's target), residuals of the FP64 form <= 1e-9
max(1, |E|); two FP64 runs agree to the bit (the step's sums have a fixed order).
"""
import os
from contextlib import contextmanager

import numpy as np
import pytest

import oracle as O
import momed
from momed import _lib
from test_gpu_pairmap import full_list, pair_terms

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


def setup(h, a, b, ne, i, seed=5):
    """H0 (one-body) + u V (two-body) on a sector: union term list with amplitudes A and B."""
    subs, _ = O.momentum_subspaces(O.mesh_klist(a, b), (a, b), (ne,), Nc_conserve=1)
    basis = subs[i]
    amp, in_, out = pair_terms(a, b, 1, seed)
    two = np.array([bin(int(o)).count("1") == 2 for o in out])
    A, B = np.where(two, 0, amp), np.where(two, amp, 0)
    h.set_basis(basis)
    h.set_scatter_pair(A, B, in_, out)
    return basis, A, B, in_, out


def dense(basis, amp, in_, out):
    f = full_list(amp, in_, out)
    n = len(basis)
    return np.column_stack([O.matvec(basis, f, np.eye(n, dtype=complex)[:, k]) for k in range(n)])


_eigs = {}


def eigs(key, basis, A, B, in_, out, u):
    if key not in _eigs:
        _eigs[key] = dense(basis, A, in_, out), dense(basis, B, in_, out)
    a, b = _eigs[key]
    return np.array([np.linalg.eigvalsh(a + x * b) for x in u])


def run(h, nu, nev, m, prec):
    u = np.linspace(0.5, 1.5, nu)
    v, _, r, info = h.batch_solve(u, nev, krylovdim=m, tol=1e-11, maxiter=300, precision=prec)
    return u, v, r


# sectors of 9, 116 and 476 states: one row block to 60, at 8 (32 right-hand sides) to 32 rows a block
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("sec", [(3, 3, 3, 1, 1), (4, 4, 4, 0, 2), (3, 6, 5, 0, 4)])
@pytest.mark.parametrize("nu", [1, 2, 3, 5, 8, 13, 16, 21, 32])
def test_block_widths(h, sec, nu, prec):
    a, b, ne, i, nev = sec
    basis, *ops = setup(h, a, b, ne, i)
    u, v, r = run(h, nu, nev, 24, prec)
    ref = eigs(sec, basis, *ops, u)[:, :nev]
    assert np.max(np.abs(v - ref) / np.maximum(1, np.abs(ref))) < 1e-10
    if prec == _lib.PREC_FP64:
        assert np.max(r / np.maximum(1, np.abs(v))) < 1e-9


@pytest.mark.parametrize("m", [7, 8, 9, 16, 17, 33, 64, 65, 66, 100])
@pytest.mark.parametrize("nu,prec", [(4, _lib.PREC_FP64), (32, _lib.PREC_MIXED)])
def test_basis_sizes(h, m, nu, prec):
    sec = (3, 6, 5, 0, 4)
    basis, *ops = setup(h, *sec[:4])
    u, v, r = run(h, nu, 2, m, prec)
    ref = eigs(sec, basis, *ops, u)[:, :2]
    assert np.max(np.abs(v - ref) / np.maximum(1, np.abs(ref))) < 1e-10


# 5538 states: 148 blocks of 38 rows; 31k states: 207 rows a block, several passes of every loop
@pytest.mark.parametrize("a,b,ne,nu,prec", [(3, 7, 7, 11, _lib.PREC_MIXED), (3, 7, 7, 6, _lib.PREC_FP64),
                                            (4, 6, 8, 32, _lib.PREC_MIXED), (4, 6, 8, 2, _lib.PREC_MIXED)])
def test_against_separate_kernels(h, a, b, ne, nu, prec):
    setup(h, a, b, ne, 2)
    u, v, _ = run(h, nu, 3, 30, prec)
    _, v1, _ = run(h, nu, 3, 30, prec)
    with env(MOMED_COOP=0):
        _, v2, _ = run(h, nu, 3, 30, prec)
    if prec == _lib.PREC_FP64:
        assert np.array_equal(v, v1)
    assert np.max(np.abs(v - v1) / np.maximum(1, np.abs(v1))) < 1e-10
    assert np.max(np.abs(v - v2) / np.maximum(1, np.abs(v2))) < 1e-10
