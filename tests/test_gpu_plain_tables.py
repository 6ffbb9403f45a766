"""momed_matvec asks for the pair tables at calls 2, 3, 5, 9, ... on a basis and operator, not at every
call: where they are not admitted the question itself costs time."""
import numpy as np
import pytest

import momed
from momed import _lib
from momed.core import pair_operator
from momed.synthetic import mesh_para

pytestmark = pytest.mark.gpu


def test_refused_tables_are_asked_for_less_and_less():
    import torch

    para, _ = mesh_para(3, 10, 1)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    h = momed.Handle(0)
    (_, basis), = h.enumerate_basis(para.k_list, para.Gk, 1, 1, (10,), momentum_list=[(2, 9)])
    h.set_basis(basis)
    h.set_scatter_pair(*pair_operator(A, B))
    rng = np.random.default_rng(0)
    x = torch.as_tensor(rng.standard_normal(len(basis)) + 1j * rng.standard_normal(len(basis)), device="cuda")
    y = torch.empty_like(x)

    def launches():
        n0 = _lib.kernel_launches()
        h.matvec_device(x.data_ptr(), y.data_ptr(), _lib.C128)
        return _lib.kernel_launches() - n0

    launches()                                     # call 1: index, validation, candidate map
    ref = y.clone()
    # 1.0M states x 45 pairs at 30 bytes: 1.4 GB, more than a quarter of what is left
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (4 << 30), dtype=torch.uint8, device="cuda")
    assert [launches(), launches()] == [1, 1]      # calls 2 and 3: asked, not admitted
    del filler
    torch.cuda.empty_cache()
    assert launches() == 1                         # call 4: not asked
    assert launches() > 3                          # call 5: asked and built
    assert float((y - ref).abs().max() / ref.abs().max()) < 1e-13
    assert launches() == 2
    h.close()
