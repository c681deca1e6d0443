"""A small active set in a lattice whose first coarse level has room for 2^32 + 1,204
blocks (3D, one field, 34.4 million coarse nodes): the sizes that limit a plan are those
of the matrix, not of the lattice.  Takes 93 GB of device memory.

Rows are diagonally dominant by a factor 1.25: |A^-1| |A| <= 9 in the maximum norm, so a
residual of 1e-10 |b|_2 leaves at most 9e-10 sqrt(n) of the largest |b| (diagonals >= 1)."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def test_plan_and_solve_in_a_large_3d_lattice(cuda):
    from geowarp_b200 import _lib as L
    from geowarp_b200.engine import _p
    lib = L.load()
    m, k, at = (602, 650, 696), 12, 300  # nodes per axis, active patch of k^3 nodes from node (at, at, at)
    if torch.cuda.mem_get_info()[0] < 110 * 2 ** 30:
        pytest.skip("needs 110 GiB of device memory")
    q = np.arange(k ** 3)
    x, y, z = q % k, q // k % k, q // k ** 2
    row2node = (at + x) + m[0] * ((at + y) + m[1] * (at + z))
    ii, jj, bit = [], [], []
    words = np.zeros((k ** 3, 4), np.uint32)
    for oz in (-1, 0, 1):
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                b = (ox + 2) + 5 * (oy + 2) + 25 * (oz + 2)
                ok = (x + ox >= 0) & (x + ox < k) & (y + oy >= 0) & (y + oy < k) & (z + oz >= 0) & (z + oz < k)
                words[ok, b // 32] |= np.uint32(1 << (b % 32))
                ii.append(q[ok]); jj.append((q + ox + k * (oy + k * oz))[ok]); bit.append(np.full(int(ok.sum()), b))
    i, j = np.concatenate(ii), np.concatenate(jj)
    order = np.lexsort((np.concatenate(bit), i))
    i, j = i[order], j[order]
    rng = np.random.default_rng(0)
    vals = rng.uniform(-1.0, 0.2, i.size)
    d = i == j
    vals[d] = 0.0
    off = np.zeros(k ** 3)
    np.add.at(off, i, np.abs(vals))
    vals[d] = np.maximum(1.25 * off, 1.0)
    M = sp.csr_matrix((vals, (i, j)))
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a).astype(dt), device=cuda)  # noqa: E731
    nn = m[0] * m[1] * m[2]
    r2n = t(row2node, np.int64)
    node2row = torch.full((nn,), -1, dtype=torch.int32, device=cuda)
    node2row[r2n] = t(q, np.int32)
    stencil = torch.zeros((nn, 4), dtype=torch.int32, device=cuda)
    stencil[r2n] = t(words.view(np.int32), np.int32)
    keep = dict(row_ptr=t(np.concatenate([[0], np.cumsum(np.bincount(i))]), np.int32), cols=t(j, np.int32),
                row2node=t(row2node, np.int32), node2row=node2row, stencil=stencil, vals=t(vals, np.float64))
    A, g = L.Bsr(), L.Grid()
    A.n_rows, A.nf, A.nnzb, A.mask_words = k ** 3, 1, i.size, 4
    for name, v in keep.items():
        setattr(A, name, _p(v))
    g.dim, g.nf, g.n_nodes = 3, 1, nn
    for a in range(3):
        g.n_grid[a], g.h[a], g.inv_h[a], g.h_nodes[a] = m[a] - 1, 1.0, 1.0, 1.0
    assert (m[0] // 2 + 1) * (m[1] // 2 + 1) * (m[2] // 2 + 1) * 125 == 2 ** 32 + 1204
    xs = rng.uniform(-1, 1, k ** 3)
    b = M @ xs
    bt, xt = t(b, np.float64), torch.zeros(k ** 3, dtype=torch.float64, device=cuda)
    nb = lib.gw_gmres_mg_workspace_bytes(C.byref(g), k ** 3, 1, 20)
    ws = torch.empty(nb, dtype=torch.uint8, device=cuda)
    plan = L.MgPlan()
    L.call("gw_mg_plan_build", C.byref(g), C.byref(A), _p(ws), nb, C.byref(plan), None)
    assert plan.levels == 3
    it, rr = C.c_int32(0), C.c_double(0.0)
    rc = lib.gw_bsr_gmres_mg_solve(C.byref(g), C.byref(A), L.PREC_F64, C.byref(plan), _p(bt), _p(xt), 1e-10, 500, 20,
                                   _p(ws), nb, C.byref(it), C.byref(rr), None)
    torch.cuda.synchronize()
    got = xt.cpu().numpy()
    del ws, stencil, node2row, keep
    torch.cuda.empty_cache()
    assert rc == L.GW_OK
    assert np.linalg.norm(M @ got - b) <= 2e-10 * np.linalg.norm(b)
    assert np.abs(got - xs).max() <= 9 * 2e-10 * np.sqrt(got.size) * np.abs(b).max()
