"""A multigrid plan launches kernels for the levels that it has, not for those that a
finer active set or a smaller dense level would need: at most eleven a coarse level,
one for the finest level's rows and one for the totals."""
import ctypes as C

import pytest
import torch

from test_gpu_mg_rows import _Gpu, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nf,levels", [(6, 4, 2, 1), (8, 8, 3, 2), (20, 15, 3, 3), (20, 15, 2, 3)])
def test_launches_of_a_plan(cuda, nx, ny, nf, levels):
    G = _Gpu(_system(nx, ny, nf, 3, 0.0, 0.0), False, cuda)
    lib, L = G.lib, G.L
    nb = lib.gw_gmres_mg_workspace_bytes(C.byref(G.g), G.A.n_rows, nf, 20)
    ws = torch.empty(nb, dtype=torch.uint8, device=cuda)
    plan = L.MgPlan()
    before = lib.gw_launch_count()
    L.call("gw_mg_plan_build", C.byref(G.g), C.byref(G.A), G.p(ws), nb, C.byref(plan), None)
    n = lib.gw_launch_count() - before
    assert plan.levels == levels
    assert n <= (1 if levels == 1 else 11 * (levels - 1) + 2)
