"""What the 2D assembly reports about a state it cannot place in the matrix, against
the atomic assembly of the same particles: a contribution outside the pattern sets the
device status (bit 0), and a node that no row belongs to is not such a contribution; a free node whose row
number is outside the matrix (a stale row map) fails the index guard.

R and K of both assemblies are the same terms in another order: 1e-12 of the largest
entry in FP64, 1e-6 (a few roundings of 2^-24) where K is FP32."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

H = 0.05


def _engine(kind, past, precision, dev):
    """A 4 x 5-cell block on a fixed base; the particles' domains reach `past` cells
    beyond the cell edges in y, so beyond the free surface too."""
    from geowarp_b200.engine import Engine, material_struct
    nx, ny = 8, 9
    c = (np.arange(8) + 0.5) / 2
    gx, gy = np.meshgrid(2 + c, 2 + np.append(c, [4.25, 4.75]), indexing="ij")
    x = np.stack([gx.ravel(), gy.ravel()], 1) * H
    e = Engine(kind, (nx, ny), (H, H), (H, H), (0.0, 0.0), (nx * H, ny * H), x, device=dev, precision=precision,
               precond="block")
    e.lp[:, 0] = 0.25 * H - 1e-6
    e.lp[:, 1] = (0.25 + past) * H
    e.step_params = dict(gravity_mag=9.81, p_vol=(H / 2) ** 2, p_rho=2000.0, PPD=2, lp0=0.25 * H - 1e-6, dt=10.0,
                         phi_initial=0.4, mobility=1e-9)
    e.reset(True)
    nn = (nx + 1) * (ny + 1)
    base = torch.arange(nx + 1, device=dev) + 2 * (nx + 1)
    e.boundary[base] = True
    e.boundary[nn + base] = True
    e.sort_and_activate()
    e.build_system()
    g = torch.Generator().manual_seed(5)
    e.u_new.copy_(1e-4 * H * torch.randn(e.u_new.shape, dtype=torch.float64, generator=g))
    return e, material_struct(dict(youngs_modulus=1e7, poisson_ratio=0.3, material_name="Neo-Hookean"))


def _assemble(e, mat, det, want_K=True):
    e.deterministic_assembly = det
    e.device_status()
    e.assemble(mat, 0, 10, want_K=want_K)
    bb = e.nf * e.nf * e.nnzb
    f64 = e.precision == "fp64"
    K = e._vals.t[: bb * (8 if f64 else 4)].view(torch.float64 if f64 else torch.float32).double().cpu().numpy()
    return e._R[: e.n_rows * e.nf].cpu().numpy(), K, e.device_status()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["solid2d", "coupled2d"])
@pytest.mark.parametrize("past", [0.0, 5e-4, 9e-4, 0.02])
def test_surface_nodes_without_a_row_are_not_reported(cuda, kind, past, precision):
    """u-p: a node whose weight is below 1e-6 (a domain less than 1e-3 of a cell past
    the surface: weight past^2) is inactive, though its gradient weight is not zero."""
    e, mat = _engine(kind, past, precision, cuda)
    if kind == "coupled2d":
        assert bool(e.node_active.view(10, 9)[8].any()) == (past > 1e-3)
    R, K, st = _assemble(e, mat, True)
    Ra, Ka, sta = _assemble(e, mat, False)
    assert st == sta == 0
    assert np.abs(R - Ra).max() <= 1e-12 * np.abs(Ra).max()
    assert np.abs(K - Ka).max() <= (1e-12 if precision == "fp64" else 1e-6) * np.abs(Ka).max()


@pytest.mark.parametrize("kind", ["solid2d", "coupled2d"])
@pytest.mark.parametrize("past", [0.0, 0.02])
def test_contribution_outside_the_pattern_is_reported(cuda, kind, past):
    """The last stencil bit of a free node taken out: its block has no place, whether
    its entries are zero (the domains end on a node) or not."""
    e, mat = _engine(kind, past, "fp64", cuda)
    node = 4 + 4 * 9
    assert int(e.free_mask[node]) == (1 << e.nf) - 1
    st = int(e.stencil[node])
    e.stencil[node] = st & ~(1 << (st.bit_length() - 1))
    assert _assemble(e, mat, True)[2] == 1
    assert _assemble(e, mat, False)[2] == 1


@pytest.mark.parametrize("want_K", [True, False])
@pytest.mark.parametrize("kind", ["solid2d", "coupled2d"])
@pytest.mark.parametrize("row", [-1, 10000])
def test_stale_row_map_fails_the_index_guard(cuda, kind, row, want_K):
    from geowarp_b200 import _lib as L
    lib = L.load()

    def guard():
        site, val = C.c_int32(0), C.c_int64(0)
        assert lib.gw_guard_read(C.byref(site), C.byref(val), e.stream) == L.GW_OK
        return lib.gw_guard_site_name(site.value).decode(), val.value

    e, mat = _engine(kind, 0.0, "fp64", cuda)
    R, K, st = _assemble(e, mat, True, want_K)
    assert st == 0 and guard() == ("none", 0)
    node = 4 + 4 * 9
    keep = int(e.node2row[node])
    e.node2row[node] = row
    assert _assemble(e, mat, True, want_K)[2] == 1
    assert guard() == ("assembly scatter", row)
    e.node2row[node] = keep
    R1, K1, st = _assemble(e, mat, True, want_K)
    assert st == 0 and guard() == ("none", 0)
    assert np.array_equal(R, R1) and np.array_equal(K, K1)
