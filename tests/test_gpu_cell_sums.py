"""The 2D assembly's cell and row passes at the places where they can go wrong: cells
with one particle, with more than a batch of eight, particles clamped at the grid's
edges, cells without particles, and both ways of indexing the cells' sums (fewer cells
than particles, and more), against the atomic assembly of the same particles.

Same terms in another order: R to 1e-12 of its largest entry; K to 1e-12 where the
values are FP64 and 1e-6 (a few roundings of 2^-24) where they are FP32."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(n_cells, x, lp, precision, material, dev):
    from geowarp_b200.solvers.quasi_static_solver_2d import quasi_static_solver_2d
    h = 0.1
    nx, ny = n_cells
    grid = dict(n_grid_x=nx, n_grid_y=ny, max_x=nx * h, dx=h, start_x=0.0, end_x=nx * h, start_y=0.0, end_y=ny * h,
                domain_min_x=0.0, domain_max_x=nx * h, domain_min_y=0.0, domain_max_y=ny * h)
    parts = dict(n_particles=len(x), PPD=2, p_vol=(h / 2) ** 2, p_rho=2000.0)
    mat = dict(youngs_modulus=1e7, poisson_ratio=0.3, material_name=material, kappa=1e4)
    s = quasi_static_solver_2d(grid, parts, dict(n_iter=5, tol=1e-8), mat, dict(gravity_mag=9.81), precision=precision,
                               device=dev, x_particles=x * h)
    s.engine.lp.copy_(torch.as_tensor(lp * h, device=dev))
    return s


def _clouds():
    rng = np.random.default_rng(0)
    one = np.array([[3.5, 2.5]])
    crowd = np.concatenate([rng.uniform([2.05, 2.05], [2.95, 2.95], (37, 2)), rng.uniform([4.0, 3.0], [7.0, 5.0], (60, 2))])
    edge = np.concatenate([rng.uniform([0.3, 0.3], [1.0, 6.7], (30, 2)), rng.uniform([8.0, 0.3], [8.7, 6.7], (30, 2))])
    return {"one particle": ((9, 7), one), "crowded cells": ((9, 7), crowd), "grid edges": ((9, 7), edge),
            "sparse grid": ((60, 50), rng.uniform([20, 20], [30, 30], (200, 2)))}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(_clouds()))
@pytest.mark.parametrize("lp", [0.2499, 0.4])
def test_sorted_assembly_equals_atomic(cuda, name, lp, precision):
    n_cells, x = _clouds()[name]
    s = _engine(n_cells, x, np.full((len(x), 2), lp), precision, "Hencky elasticity", cuda)
    e = s.engine
    s._set_step_params()
    s.dofStruct.boundary_flag_array[::7] = True
    s.reset()
    e.sort_and_activate()
    e.build_system()
    g = torch.Generator().manual_seed(2)
    e.u_new.copy_(1e-4 * torch.randn(e.u_new.shape, dtype=torch.float64, generator=g))
    vt = torch.float64 if precision == "fp64" else torch.float32
    nv, n = e.nnzb * 4, e.n_rows * 2
    out = []
    for det in (True, False):
        e.deterministic_assembly = det
        e._vals.t.fill_(0xFF)  # nothing may be left of what was there before
        e._R.fill_(float("nan"))
        e.assemble(s._mat, 0, 10)
        K = e._vals.t[: nv * (8 if vt == torch.float64 else 4)].view(vt).double().cpu().numpy()
        out.append((K, e._R[:n].cpu().numpy(), e.device_status()))
        if det:
            e.assemble(s._mat, 0, 10, want_K=False)
            assert np.array_equal(e._R[:n].cpu().numpy(), out[0][1])
    (K, R, st), (Ka, Ra, sta) = out
    # a particle that reaches past the grid is reported by both (the right edge with
    # lp = 0.4), and nothing else is
    past = bool((x + lp > np.array(n_cells)).any())
    assert st == sta == (1 if past else 0)
    assert np.abs(R - Ra).max() <= 1e-12 * np.abs(Ra).max()
    assert np.abs(K - Ka).max() <= (1e-12 if precision == "fp64" else 1e-6) * np.abs(Ka).max()
