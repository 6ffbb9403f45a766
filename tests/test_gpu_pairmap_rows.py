"""Second half of the product over the pair tables (csrc/pairmap.cu): 8, 4, 2 and 1 warps share 32 rows by the
sector's size, each summing its pairs six (c128) or twelve (c64) at a time with a remainder.

Bars against the map over the hit records: complex128 1e-13, complex64 2e-6 relative (those of
test_gpu_pairmap.py).
"""
import numpy as np
import pytest

import momed
from test_gpu_pairmap import env, pair_terms, rel, sector, vec

pytestmark = pytest.mark.gpu


# 3, 15, 28, 36 and 45 pairs a row; 8 (to 18.9k states), 4, 2 and 1 (from 75.8k) warps
@pytest.mark.parametrize("a,b,ne,warps", [(3, 5, (3,), 8), (3, 7, (6,), 8), (3, 8, (8,), 4), (5, 5, (8,), 2),
                                          (3, 9, (9,), 1), (5, 5, (10,), 1)])
def test_rows_shared_by_warps(a, b, ne, warps):
    basis = sector(a, b, ne, 1)
    n = len(basis)
    assert warps == min([g for g in (1, 2, 4, 8) if (n + 31) // 32 * g >= 148 * 16] + [8])
    amp, in_, out = pair_terms(a, b, len(ne), 5)
    h = momed.Handle(0)
    h.set_basis(basis)
    h.set_scatter(amp, in_, out)
    y = {}
    x = vec(n)
    for form in (1, 0):
        with env(MOMED_PAIRMAP=form):
            h.build_hit_cache()
            y[form] = h.matvec(x), h.matvec(x.astype(np.complex64))
    h.close()
    assert rel(y[1][0], y[0][0]) < 1e-13
    assert rel(y[1][1], y[0][1]) < 2e-6
