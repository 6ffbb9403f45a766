"""Graph replay of the lockstep solver's restart cycles, which runs where its cooperative steps do not
(MOMED_COOP=0): the cycles after the first really are graph launches, and give what eager launches give
(to 1e-12: the norms of the separate kernels are summed with atomics)."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import momed
from momed import _lib
from momed.core import pair_operator
from momed.synthetic import mesh_para, u_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
def test_replayed_cycles(prec, monkeypatch):
    para, _ = mesh_para(3, 8, 5)
    A = momed.MBOperator(momed.ED_scatterlist_onebody(para), upper_hermitian=True)
    B = momed.MBOperator(momed.ED_scatterlist_twobody(para), upper_hermitian=True)
    h = momed.Handle(0)
    (_, basis), = h.enumerate_basis(para.k_list, para.Gk, 1, 1, (8,), momentum_list=[(1, 3)])
    h.set_basis(basis)
    h.set_scatter_pair(*pair_operator(A, B))
    u = u_grid(8, 0.5, 2.0)
    got = {}
    for form, env in (("replays", {"MOMED_COOP": "0"}), ("eager", {"MOMED_COOP": "0", "MOMED_GRAPHS": "0"}), ("coop", {})):
        for k in ("MOMED_COOP", "MOMED_GRAPHS"):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            v, _, _, info = h.batch_solve(u, 4, krylovdim=30, tol=1e-12, precision=prec)
        calls = p.key_averages()
        if not any("LaunchKernel" in e.key or "LaunchCooperative" in e.key for e in calls):
            pytest.skip("no records of launches in this environment")
        graphs = sum(e.count for e in calls if "GraphLaunch" in e.key)
        got[form] = v, info, graphs
    h.close()
    v, info, graphs = got["replays"]
    assert info["restarts"] >= 2 and graphs >= info["restarts"] - 1
    for form in ("eager", "coop"):
        assert got[form][2] == 0
        assert np.max(np.abs(got[form][0] - v) / np.abs(v)) < 1e-11
    assert np.max(np.abs(got["eager"][0] - v) / np.abs(v)) < 1e-12
