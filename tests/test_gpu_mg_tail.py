"""The fused coarse tail on assembled systems: GW_TUNE_MG_TAIL = 1 runs one launch per
phase, 0 (the default) and 4096 fuse the levels up to 2,048 and 4,096 rows.  Same bytes,
in fewer launches."""
import numpy as np
import pytest
import torch

import cases
from test_gpu_mg import _assembled, _solve, _system_footing

pytestmark = pytest.mark.gpu


def _column(precision):
    from geowarp_b200.solvers import quasi_static_coupled_solver_2d
    grid, parts, it, mat, porous, load = cases.terzaghi_dicts(n_cells_y=60)
    s = quasi_static_coupled_solver_2d(grid, parts, it, mat, porous, load, cases.terzaghi_boundary_kernel,
                                       precision=precision, precond="mg")
    top = cases.top_flags(s.x_particles, grid["end_y"], grid["dx"], parts["PPD"])
    s.particle_pressure_boundary_flag_array[:] = top
    s.particle_traction_flag_array[:] = top
    s.advance_one_step(0, 600)
    return s.engine  # its last system, still assembled


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("system", ["footing", "column"])
def test_tail_is_bitwise_the_separate_levels_on_assembled_systems(cuda, system, precision):
    from geowarp_b200 import _lib as L
    lib = L.load()
    e = _column(precision) if system == "column" else _assembled(*_system_footing(precision))
    default = lib.gw_tune_get(L.TUNE_MG_TAIL)
    out = {}
    b = torch.Generator().manual_seed(1)
    e._R[: e.n_rows * e.nf] = torch.randn(e.n_rows * e.nf, dtype=torch.float64, generator=b).to(cuda)
    try:
        for knob in (1, 0, 4096):
            assert lib.gw_tune_set(L.TUNE_MG_TAIL, knob) == L.GW_OK
            e._mg_plan = None
            e._gm_hint = (0, 0)
            n0 = lib.gw_launch_count()
            x, it, rr, rc = _solve(e, "mg", 1e-8)
            out[knob] = (x.cpu().numpy(), it, rc, lib.gw_launch_count() - n0)
    finally:
        lib.gw_tune_set(L.TUNE_MG_TAIL, default)
    assert default == 0
    x1, it1, rc1, n1 = out[1]
    assert it1 > 3
    for knob in (0, 4096):
        x, it, rc, n = out[knob]
        assert it == it1 and rc == rc1 and np.array_equal(x, x1)
        assert n < n1 - 10 * it1  # at least ten phases a V-cycle in one launch
