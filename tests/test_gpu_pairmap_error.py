"""Rounding of products over the pair tables (csrc/pairmap.cu): complex64 no further from the complex128
product of the same vector, complex128 no further from sums in 80 bits, than the map over the hit records is.
Bar: 1.05 times its relative error in the 2-norm, as both are sums of thousands of independent roundings."""
import numpy as np
import pytest

import momed
from test_gpu_pairmap import env, full_list, pair_terms, sector, vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b,ne,i,shift", [(3, 7, (7,), 2, 0.0), (3, 7, (7,), 2, 4.0), (5, 5, (6,), 3, 4.0),
                                            (3, 8, (8,), 1, 1.0), (3, 5, (3, 4), 2, 4.0), (4, 5, (3, 3), 4, 1.0)])
def test_error_of_complex64_products(a, b, ne, i, shift):
    """shift: the diagonal's weight, which dominates the rows of an ordinary interaction."""
    basis = sector(a, b, ne, i)
    amp, in_, out = pair_terms(a, b, len(ne), 31)
    amp = np.where(in_ == out, amp + shift, 0.1 * amp)
    h = momed.Handle(0)
    h.set_basis(basis)
    h.set_scatter(amp, in_, out)
    err = {}
    for form in (1, 0):
        with env(MOMED_PAIRMAP=form):
            h.build_hit_cache()
            e = []
            for seed in range(4):
                x = vec(len(basis), seed).astype(np.complex64)
                y64, y32 = h.matvec(x.astype(np.complex128)), h.matvec(x)
                e.append(np.linalg.norm(y32 - y64) / np.linalg.norm(y64))
            err[form] = np.mean(e)
    h.close()
    assert err[1] < 1.05 * err[0], err


def product80(basis, full, x):
    y, x = np.zeros(len(basis), np.clongdouble), x.astype(np.clongdouble)
    for t in full:
        out, in_, pm = np.uint64(t["out"]), np.uint64(t["in"]), np.uint64(t["pm"])
        r = np.flatnonzero((basis & out) == out)
        rest = basis[r] & ~out
        r, rest = r[(rest & in_) == 0], rest[(rest & in_) == 0]
        j = np.minimum(np.searchsorted(basis, rest | in_), len(basis) - 1)
        ok = basis[j] == (rest | in_)
        r, j, par = r[ok], j[ok], rest[ok] & pm
        for shift in (32, 16, 8, 4, 2, 1):
            par = par ^ (par >> np.uint64(shift))
        z = (np.longdouble(t["re"]) + 1j * np.longdouble(t["im"])) * x[j]
        y[r] += np.where(par & np.uint64(1), -z, z)
    return y


@pytest.mark.parametrize("a,b,ne,i", [(3, 7, (7,), 2), (4, 5, (2, 3), 2)])
def test_error_of_complex128_products(a, b, ne, i):
    basis = sector(a, b, ne, i)
    amp, in_, out = pair_terms(a, b, len(ne), 1)
    amp = np.where(in_ == out, amp + 4.0, 0.1 * amp)
    x = vec(len(basis))
    ref = product80(basis, full_list(amp, in_, out), x)
    h = momed.Handle(0)
    h.set_basis(basis)
    h.set_scatter(amp, in_, out)
    err = {}
    for form in (1, 0):
        with env(MOMED_PAIRMAP=form):
            h.build_hit_cache()
            err[form] = float(np.sqrt(np.sum(np.abs(h.matvec(x) - ref).astype(float) ** 2)) / np.linalg.norm(x))
    h.close()
    assert err[1] < 1.05 * err[0], err
