"""The solver of a single solve does not depend on what the handle did before: over the pair tables it is
the single-vector one, also after a sweep has built the hit records that block maps read."""
import pytest

import momed
from momed import _lib
from momed.core import pair_operator
from momed.synthetic import mesh_para

pytestmark = pytest.mark.gpu


def test_single_solve_after_a_sweep_keeps_the_pair_map():
    para, _ = mesh_para(4, 6, 1, Nc_conserve=2)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    h = momed.Handle(0)
    (_, basis), = h.enumerate_basis(para.k_list, para.Gk, 1, 2, (4, 4), momentum_list=[(3, 1)])
    assert len(basis) >= 2_000_000                 # from here the records alone mean the block solver for 6 pairs
    h.set_basis(basis)
    h.set_scatter_pair(*pair_operator(A, B))
    h.batch_solve([0.9, 1.1], 1, krylovdim=4, maxiter=1)     # builds the records
    h.profile(True)
    h.eigsolve(6, krylovdim=10, maxiter=1, want_vectors=False)
    block, single = (h.profile_read(k)[0] for k in (_lib.KERNEL_HC_BLOCK_C128, _lib.KERNEL_HC_MATVEC_C128))
    h.profile(False)
    h.close()
    assert block == 0 and single >= 10
