"""Kernels of the 3D u-p path: the warp-per-row product of node-block GMRES on rows
of 1 to 125 blocks, and the assembly's two particle groupings.

GMRES tolerances: rows are diagonally dominant by a factor 1.25 with unit-size
entries, so |A^-1| |A| <= 9 in the maximum norm (see the multigrid row tests); no
diagonal stencil bit is set, so the preconditioner is the identity.  The assembly's
groupings add the same terms with atomics in another order: 1e-12 of the largest
entry for sums of at most a few hundred FP64 terms, 2e-5 where the values are FP32."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,lo,hi,nf", [(1, 1, 1, 4), (33, 16, 33, 4), (200, 60, 125, 4), (203, 90, 101, 3), (150, 20, 64, 2),
                                        (501, 16, 40, 1), (400, 4, 9, 4)])
def test_node_block_gmres_on_long_rows(cuda, n, lo, hi, nf, single):
    from geowarp_b200 import _lib as L
    from geowarp_b200.engine import _p
    lib = L.load()
    rng = np.random.default_rng(n + nf)
    rows, cols = [], []
    for r in range(n):
        m = min(n, int(rng.integers(lo, hi + 1)))
        c = np.sort(np.append(rng.choice(np.delete(np.arange(n), r), m - 1, replace=False), r)) if n > 1 else np.array([0])
        rows.append(np.full(c.size, r)); cols.append(c)
    i, j = np.concatenate(rows), np.concatenate(cols).astype(int)
    vals = rng.uniform(-1, 1, (i.size, nf, nf)).astype(np.float32).astype(np.float64)
    k = np.arange(nf)
    d = np.nonzero(i == j)[0]
    vals[d[:, None], k, k] = 0
    off = np.zeros((n, nf))
    np.add.at(off, i, np.abs(vals).sum(2))
    vals[d[:, None], k, k] = (1.25 * off[i[d]] + 0.1).astype(np.float32)
    rr_, cc_ = (i[:, None, None] * nf + k[:, None]) + 0 * k[None, :], (j[:, None, None] * nf + k[None, :]) + 0 * k[:, None]
    M = sp.csr_matrix((vals.ravel(), (rr_.ravel(), cc_.ravel())), shape=(n * nf,) * 2)
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a).astype(dt), device=cuda)  # noqa: E731
    keep = dict(row_ptr=t(np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]), np.int32), cols=t(j, np.int32),
                row2node=t(np.arange(n), np.int32), node2row=t(np.arange(n), np.int32),
                stencil=t(np.zeros(4 * n), np.int32), vals=t(vals, np.float32 if single else np.float64))
    A = L.Bsr()
    A.n_rows, A.nf, A.nnzb, A.mask_words = n, nf, i.size, 4
    for name, v in keep.items():
        setattr(A, name, _p(v))
    xs = rng.uniform(-1, 1, n * nf)
    b = M @ xs
    bt, x = torch.as_tensor(b, device=cuda), torch.zeros(n * nf, dtype=torch.float64, device=cuda)
    restart = 24
    ws = torch.full((lib.gw_gmres_workspace_bytes(n, nf, restart),), 0xFF, dtype=torch.uint8, device=cuda)
    it, rr = C.c_int32(0), C.c_double(0.0)
    rc = lib.gw_bsr_gmres_solve(C.byref(A), L.PREC_F32 if single else L.PREC_F64, 1, _p(bt), _p(x), 1e-12, 2000, restart,
                                _p(ws), C.byref(it), C.byref(rr), None)
    torch.cuda.synchronize()
    x = x.cpu().numpy()
    assert rc == L.GW_OK
    assert np.linalg.norm(M @ x - b) <= 2e-12 * np.linalg.norm(b)
    assert np.abs(x - xs).max() <= 9 * 2e-12 * np.sqrt(x.size) * np.abs(b).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_assembly_groupings_agree(cuda, precision):
    """2,744 particles in groups of 32 against the same particles in two launches
    of fewer than 2,368, in groups of eight."""
    from geowarp_b200 import _lib as L
    from geowarp_b200 import problems
    from geowarp_b200.engine import _p
    from geowarp_b200.launch import launch
    s = problems.indentation_3d(precision=precision, precond="block", block_cells=(7, 7, 7), grid_cells=(9, 9, 9), dx=0.25,
                                E=1e3, material="Neo-Hookean", permeability=1e-11, indenter=0.5, depth=0.5, n_steps=25,
                                penalty=1000.0)
    e = s.engine
    s._sync_grid()
    s._set_step_params()
    s.reset()
    launch(s.set_boundary_dofs, (s.n_grid_x + 1, s.n_grid_y + 1, s.n_grid_z + 1),
           [e.boundary, s.n_grid_x, s.n_grid_y, s.n_nodes, s.dx, s.dy, s.end_x, s.end_y])
    e.sort_and_activate()
    e.project_pressure()
    e.build_system()
    e.u_new += 1e-4 * torch.randn(e.u_new.shape, dtype=torch.float64, generator=torch.Generator().manual_seed(1)).to(cuda)
    g, st, nv, n = e.grid_struct(), e.step_struct(0, 25), e.nnzb * 16, e.n_rows * 4
    vt = torch.float64 if precision == "fp64" else torch.float32

    def run(lo, hi):
        pt = e.particles_struct()
        pt.n = hi - lo
        A = e.bsr_struct()
        R = torch.zeros(n, dtype=torch.float64, device=cuda)
        perm = e.perm[lo:hi].contiguous()
        e.force.zero_()
        L.call("gw_assemble", C.byref(g), C.byref(s._mat), C.byref(st), C.byref(pt), _p(perm), _p(e.free_mask), _p(e.u_new),
               _p(e.u_old), C.byref(A), e.prec, _p(R), _p(e.force), e.stream)
        return R, e._vals.t[: nv * (8 if vt == torch.float64 else 4)].view(vt).double().clone(), float(e.force.item())

    assert e.N == 2744
    R, K, f = run(0, e.N)
    parts = [run(0, 1400), run(1400, e.N)]
    # the identity rows of Dirichlet DOFs are written by both launches
    K2 = parts[0][1] + parts[1][1]
    both = (parts[0][1] == 1.0) & (parts[1][1] == 1.0) & (K == 1.0)
    K2[both] = 1.0
    tol = 1e-12 if precision == "fp64" else 2e-5
    assert float((R - parts[0][0] - parts[1][0]).abs().max()) <= 1e-12 * float(R.abs().max())
    assert float((K - K2).abs().max()) <= tol * float(K.abs().max())
    assert abs(f - parts[0][2] - parts[1][2]) <= 1e-12 * abs(f)


@pytest.mark.parametrize("single", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("mx,my,mz,nf,holes", [(3, 4, 2, 3, 0.0), (9, 8, 7, 1, 0.1), (11, 7, 9, 3, 0.05), (8, 9, 10, 4, 0.0)])
def test_multigrid_on_a_3d_lattice(cuda, mx, my, mz, nf, holes, single):
    """27-point rows on an mx x my x mz lattice with missing nodes: the tolerances
    of the row tests above."""
    from geowarp_b200 import _lib as L
    from geowarp_b200.engine import _p
    lib = L.load()
    rng = np.random.default_rng(mx + nf)
    nn = mx * my * mz
    active = rng.random(nn) >= holes
    id_ = np.arange(nn)
    x, y, z = id_ % mx, id_ // mx % my, id_ // (mx * my)
    row2node = np.nonzero(active)[0]
    node2row = np.full(nn, -1)
    node2row[row2node] = np.arange(row2node.size)
    stencil = np.zeros((nn, 4), np.uint32)
    ii, jj, bit = [], [], []
    for oz in (-1, 0, 1):
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                q = (ox + 2) + 5 * (oy + 2) + 25 * (oz + 2)
                ok = (x + ox >= 0) & (x + ox < mx) & (y + oy >= 0) & (y + oy < my) & (z + oz >= 0) & (z + oz < mz) & active
                j = np.where(ok, id_ + ox + mx * (oy + my * oz), 0)
                ok &= active[j]
                stencil[ok, q // 32] |= np.uint32(1 << (q % 32))
                ii.append(node2row[id_[ok]]); jj.append(node2row[j[ok]]); bit.append(np.full(int(ok.sum()), q))
    i, j = np.concatenate(ii), np.concatenate(jj)
    order = np.lexsort((np.concatenate(bit), i))
    i, j = i[order], j[order]
    n = row2node.size
    vals = rng.uniform(-1.0, 0.2, (i.size, nf, nf)).astype(np.float32).astype(np.float64)
    k = np.arange(nf)
    d = np.nonzero(i == j)[0]
    vals[d[:, None], k, k] = 0
    off = np.zeros((n, nf))
    np.add.at(off, i, np.abs(vals).sum(2))
    vals[d[:, None], k, k] = (1.25 * off[i[d]] + 0.1).astype(np.float32)
    rr_, cc_ = (i[:, None, None] * nf + k[:, None]) + 0 * k[None, :], (j[:, None, None] * nf + k[None, :]) + 0 * k[:, None]
    M = sp.csr_matrix((vals.ravel(), (rr_.ravel(), cc_.ravel())), shape=(n * nf,) * 2)
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a).astype(dt), device=cuda)  # noqa: E731
    keep = dict(row_ptr=t(np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]), np.int32), cols=t(j, np.int32),
                row2node=t(row2node, np.int32), node2row=t(node2row, np.int32),
                stencil=t(stencil.view(np.int32), np.int32), vals=t(vals, np.float32 if single else np.float64))
    A, g = L.Bsr(), L.Grid()
    A.n_rows, A.nf, A.nnzb, A.mask_words = n, nf, i.size, 4
    for name, v in keep.items():
        setattr(A, name, _p(v))
    g.dim, g.nf, g.n_nodes = 3, nf, nn
    for a, m in enumerate((mx, my, mz)):
        g.n_grid[a], g.h[a], g.inv_h[a], g.h_nodes[a] = m - 1, 1.0, 1.0, 1.0
    xs = rng.uniform(-1, 1, n * nf)
    b = M @ xs
    bt, xt = torch.as_tensor(b, device=cuda), torch.zeros(n * nf, dtype=torch.float64, device=cuda)
    nb = lib.gw_gmres_mg_workspace_bytes(C.byref(g), n, nf, 20)
    ws = torch.full((nb,), 0xFF, dtype=torch.uint8, device=cuda)
    it, rr = C.c_int32(0), C.c_double(0.0)
    rc = lib.gw_bsr_gmres_mg_solve(C.byref(g), C.byref(A), L.PREC_F32 if single else L.PREC_F64, None, _p(bt), _p(xt), 1e-12,
                                   1000, 20, _p(ws), nb, C.byref(it), C.byref(rr), None)
    torch.cuda.synchronize()
    got = xt.cpu().numpy()
    assert rc == L.GW_OK
    assert np.linalg.norm(M @ got - b) <= 2e-12 * np.linalg.norm(b)
    assert np.abs(got - xs).max() <= 9 * 2e-12 * np.sqrt(got.size) * np.abs(b).max()
