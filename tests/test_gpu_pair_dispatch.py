"""Which map runs, seen from the launches of a product: two over the pair tables (classes, rows), one over
the hit records or the candidates."""
import numpy as np
import pytest

import momed
from momed import _lib
from test_gpu_pairmap import env, pair_terms, sector, vec

pytestmark = pytest.mark.gpu

RECORDS, PAIRS = 1, 2


@pytest.fixture(scope="module")
def h():
    hd = momed.Handle(0)
    yield hd
    hd.close()


def launches(h, x):
    n0 = _lib.kernel_launches()
    h.matvec(x)
    return _lib.kernel_launches() - n0


def form(h, basis, amp, in_, out):
    """Launches of a product over the full cache, values formed before."""
    h.set_basis(basis)
    h.set_scatter(amp, in_, out)
    h.build_hit_cache()
    x = vec(len(basis))
    h.matvec(x)
    return launches(h, x)


# entries (rows x pairs) and hits per entry: 6.2M, 6.0 | 5.7M, 3.4 (half filled) | 858k below 2^20 | 1.2M
@pytest.mark.parametrize("a,b,ne,i,want", [(3, 9, 9, 5, PAIRS), (4, 6, 11, 2, RECORDS), (3, 8, 8, 1, RECORDS),
                                           (5, 5, 8, 3, PAIRS)])
def test_size_and_density(h, a, b, ne, i, want):
    assert form(h, sector(a, b, (ne,), i), *pair_terms(a, b, 1, 12)) == want


def test_operators(h):
    basis = sector(3, 5, (5,), 1)
    amp, in_, out = pair_terms(3, 5, 1, 9)
    with env(MOMED_PAIRMAP=1):                             # whatever the size
        assert form(h, basis, amp, in_, out) == PAIRS
        twice = np.concatenate([np.arange(len(amp)), [40, 41]])
        assert form(h, basis, amp[twice], in_[twice], out[twice]) == RECORDS
        hop = np.array([1.0 + 0.5j, 1.0 - 0.5j])           # a one-body term off the diagonal
        assert form(h, np.arange(1, 256, dtype=np.uint64), np.concatenate([amp, hop]),
                    np.concatenate([in_, np.array([1, 2], np.uint64)]),
                    np.concatenate([out, np.array([2, 1], np.uint64)])) == RECORDS
        for orb, want in ((8, PAIRS), (9, RECORDS)):       # no conservation: one class of 28, of 36 pairs
            p, q = np.triu_indices(orb, 1)
            m = (np.uint64(1) << p.astype(np.uint64)) | (np.uint64(1) << q.astype(np.uint64))
            v = np.random.default_rng(10).standard_normal((len(m), len(m)))
            states = np.array([s for s in range(1 << orb) if bin(s).count("1") == 4], np.uint64)
            assert form(h, states, (v + v.T).reshape(-1) + 0j, np.tile(m, len(m)), np.repeat(m, len(m))) == want
    with env(MOMED_PAIRMAP=0):
        assert form(h, basis, amp, in_, out) == RECORDS


def test_repeated_products(h):
    """Without a cache: the candidate map, and from the second call on the pair tables where they are due."""
    for (a, b, ne, i), late in (((5, 5, 8, 3), PAIRS), ((3, 8, 8, 1), 1)):
        basis = sector(a, b, (ne,), i)
        h.set_basis(basis)
        h.set_scatter(*pair_terms(a, b, 1, 12))
        x = vec(len(basis))
        h.matvec(x)
        h.matvec(x)
        assert launches(h, x) == late
        assert h.hit_cache_info() is None
        with env(MOMED_HITCACHE=0):
            h.set_basis(basis)
            assert [launches(h, x) for _ in range(4)][1:] == [1, 1, 1]
