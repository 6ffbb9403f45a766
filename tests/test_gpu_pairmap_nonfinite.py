"""Infinities and NaN in the pair-factorised map (csrc/pairmap.cu): they reach the rows that the list
connects to them and no others, as in the map that evaluates term by term, though the product over a class
also takes couplings that the list lacks and pairs that a state lacks.  Where the result is finite it keeps
the bars of test_gpu_pairmap.py (1e-13 and 2e-6 relative)."""
import numpy as np
import pytest

import momed
from test_gpu_pairmap import env, pair_terms, sector, vec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    with env(MOMED_PAIRMAP=1):
        hd = momed.Handle(0)
        yield hd
        hd.close()


def both(h, basis, terms, x):
    """The product term by term, and over the pair tables (three launches: values, classes, rows)."""
    h.set_basis(basis)
    h.set_scatter(*terms)
    with env(MOMED_HITCACHE=0):
        ref = h.matvec(x)
    h.build_hit_cache()
    n0 = momed._lib.kernel_launches()
    y = h.matvec(x)
    assert momed._lib.kernel_launches() - n0 == 3
    return ref, y


def compare(ref, y, bar):
    rf, yf = np.isfinite(ref), np.isfinite(y)
    assert 0 < np.count_nonzero(~rf) < len(ref)
    assert np.array_equal(rf, yf)
    assert np.max(np.abs(y[rf] - ref[rf])) < bar * np.max(np.abs(ref[rf]))


# classes of 6 (padded), 13 and 15 pairs; two components with classes below and above half the largest
@pytest.mark.parametrize("a,b,ne,i", [(3, 4, (5,), 0), (3, 9, (4,), 5), (3, 5, (3, 2), 2)])
@pytest.mark.parametrize("dtype,bar", [(np.complex128, 1e-13), (np.complex64, 2e-6)])
@pytest.mark.parametrize("value", [np.inf, -np.inf + 0j, complex(0.5, np.nan)])
def test_value_of_x(h, a, b, ne, i, dtype, bar, value):
    basis = sector(a, b, ne, i)
    amp, in_, out = pair_terms(a, b, len(ne), 21, keep=0.4)
    some = np.random.default_rng(1).random(len(amp)) < 0.5          # diagonal terms missing, too
    keep = (in_ != out) | some
    terms = amp[keep], in_[keep], out[keep]
    x = vec(len(basis)).astype(dtype)
    x[[1, len(basis) // 2]] = value
    compare(*both(h, basis, terms, x), bar)


@pytest.mark.parametrize("dtype,bar", [(np.complex128, 1e-13), (np.complex64, 2e-6)])
def test_amplitude(h, dtype, bar):
    """One listed coupling not finite: rows that lack one of its pairs stay finite."""
    basis = sector(3, 7, (5,), 2)
    amp, in_, out = pair_terms(3, 7, 1, 22)
    amp = amp.copy()
    off = np.flatnonzero(in_ != out)
    amp[off[len(off) // 3]] = np.inf
    compare(*both(h, basis, (amp, in_, out), vec(len(basis)).astype(dtype)), bar)
    if dtype == np.complex64:                                       # finite in FP64, not in FP32
        amp[off[len(off) // 3]] = 1e39
        compare(*both(h, basis, (amp, in_, out), vec(len(basis)).astype(dtype)), bar)
