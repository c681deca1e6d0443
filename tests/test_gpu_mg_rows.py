"""The 2D multigrid V-cycle on the sliced row layout, and the Gram-Schmidt step
around it, against a SciPy restatement of the same V-cycle.

One flexible-GMRES iteration from x = 0 returns x = y z with z the V-cycle of
b / |b| and y the minimiser of |b - y A z|, so the solution after max_iter = 1
shows every entry of the V-cycle.  Lattices: dense level only, two levels,
levels around the chunk sizes of 8 and 32 rows, 25-point and 9-point rows side
by side, nodes missing from the active set, fixed DOFs, and a lattice above
24,576 rows, where a row is one lane's.  Matrices hold FP32-representable values,
so both precisions solve the same finest system.

Tolerances.  FP64: the library and SciPy sum the same terms in another order:
1e-11 is four orders above the rounding of a V-cycle on diagonally dominant
rows.  Mixed: the coarse operators are stored in FP32 (2^-24 relative each), so
the V-cycle moves by a few 1e-7 of its size: 1e-5.  Converged solves: rows are
diagonally dominant by a factor 1.25, so |A^-1| |A| <= (1 + 0.8) / (1 - 0.8) = 9 in
the maximum norm and a residual of 1e-12 |b|_2 leaves at most 9e-12 sqrt(n)."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla
import torch

pytestmark = pytest.mark.gpu

OMEGA = 0.7


def _system(nx, ny, nf, seed, holes, wide):
    """Block rows on the active nodes of an (nx+1) x (ny+1) lattice: 3 x 3
    neighbourhoods, 5 x 5 on the share `wide` of the nodes (symmetric pattern)."""
    rng = np.random.default_rng(seed)
    mx, my = nx + 1, ny + 1
    nn = mx * my
    active = np.ones(nn, bool)
    active[rng.random(nn) < holes] = False
    big = rng.random(nn) < wide
    ix, iy = np.arange(nn) % mx, np.arange(nn) // mx
    stencil = np.zeros(nn, np.int64)
    pairs = []
    for oy in range(-2, 3):
        for ox in range(-2, 3):
            jx, jy = ix + ox, iy + oy
            ok = (jx >= 0) & (jx < mx) & (jy >= 0) & (jy < my) & active
            j = np.where(ok, jx + jy * mx, 0)
            ok &= active[j]
            if max(abs(ox), abs(oy)) == 2:
                ok &= big | big[j]
            stencil[ok] |= 1 << ((ox + 2) + 5 * (oy + 2))
            pairs.append((np.nonzero(ok)[0], j[ok], (ox + 2) + 5 * (oy + 2)))
    row2node = np.nonzero(active)[0]
    node2row = np.full(nn, -1)
    node2row[row2node] = np.arange(row2node.size)
    i = node2row[np.concatenate([p[0] for p in pairs])]
    j = node2row[np.concatenate([p[1] for p in pairs])]
    bit = np.concatenate([np.full(p[0].size, p[2]) for p in pairs])
    order = np.lexsort((bit, i))
    i, j = i[order], j[order]
    n_rows = row2node.size
    row_ptr = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n_rows))])
    vals = rng.uniform(-1.0, 0.2, size=(i.size, nf, nf)).astype(np.float32).astype(np.float64)
    diag = np.nonzero(i == j)[0]
    k = np.arange(nf)
    vals[diag[:, None], k, k] = 0.0
    off = np.zeros((n_rows, nf))
    np.add.at(off, i, np.abs(vals).sum(2))
    vals[diag[:, None], k, k] = (1.25 * off[i[diag]] + 0.1).astype(np.float32)
    fixed = rng.random((n_rows, nf)) < 0.05
    if nf > 2:
        fixed[:, 2:] = False
    # Dirichlet DOFs: identity rows, zero columns
    vals = np.where(fixed[i][:, :, None] | fixed[j][:, None, :], 0.0, vals)
    for f in range(nf):
        m = fixed[i[diag], f]
        vals[diag[m], f, f] = 1.0
    r = (i[:, None, None] * nf + k[:, None]) + 0 * k[None, :]
    c = (j[:, None, None] * nf + k[None, :]) + 0 * k[:, None]
    A = sp.csr_matrix((vals.ravel(), (r.ravel(), c.ravel())), shape=(n_rows * nf,) * 2)
    return dict(mx=mx, my=my, nf=nf, active=active, row2node=row2node, node2row=node2row, row_ptr=row_ptr, cols=j,
                vals=vals, stencil=stencil, A=A, n_rows=n_rows)


# ---------------------------------------------------------------- SciPy V-cycle
def _hierarchy(S, single):
    """Levels of (A, inverse node blocks, P to the next level); the last one dense."""
    nf, mx, my = S["nf"], S["mx"], S["my"]
    A, active = S["A"], S["active"]
    levels = []
    while True:
        nodes = np.nonzero(active)[0]
        n = nodes.size
        if n * nf <= 160:
            levels.append((A.toarray(), None, None))
            return levels
        # node blocks; u-p systems (three fields in 2D) take the Schur diagonal
        M = np.zeros((n, nf, nf))
        for f in range(nf):
            for g in range(nf):
                M[:, f, g] = A[np.arange(n) * nf + f, np.arange(n) * nf + g]
        if nf == 3:
            coo = A.tocoo()
            keep = (coo.row // nf != coo.col // nf)
            Ao = sp.csr_matrix((coo.data[keep], (coo.row[keep], coo.col[keep])), shape=A.shape)
            pr = np.arange(n) * nf + 2
            for g in range(2):
                d = A.diagonal()[np.arange(n) * nf + g]
                B, Bt = Ao[pr][:, np.arange(n) * nf + g], Ao[np.arange(n) * nf + g][:, pr]
                w = np.where(d != 0, 1.0 / np.where(d != 0, d, 1.0), 0.0)
                M[:, 2, 2] -= np.asarray(B.multiply(Bt.T).multiply(w[None, :]).sum(1)).ravel()
        Minv = np.linalg.inv(M)
        # identity rows are fixed DOFs
        absrow = np.asarray(abs(A).sum(1)).ravel()
        fixed = (absrow == 1.0) & (A.diagonal() == 1.0)
        cx, cy = mx // 2 + 1, my // 2 + 1  # coarse lattice: cells (n + 1) / 2, nodes one more
        jx, jy = nodes % mx, nodes // mx
        rows, cols, w = [], [], []
        for a in range(2):
            for b in range(2):
                px, py = jx // 2 + a, jy // 2 + b
                ok = ((a == 0) | (jx % 2 == 1)) & ((b == 0) | (jy % 2 == 1))
                wt = np.where(jx % 2 == 1, 0.5, 1.0) * np.where(jy % 2 == 1, 0.5, 1.0)
                rows.append(np.nonzero(ok)[0]); cols.append((px + py * cx)[ok]); w.append(wt[ok])
        rows, cols, w = np.concatenate(rows), np.concatenate(cols), np.concatenate(w)
        cact = np.zeros(cx * cy, bool)
        cact[cols] = True
        cmap = np.cumsum(cact) - 1
        P = sp.csr_matrix((w, (rows, cmap[cols])), shape=(n, int(cact.sum())))
        P = sp.kron(P, sp.identity(nf), format="csr")
        P = sp.diags((~fixed).astype(float)) @ P
        Ac = (P.T @ A @ P).tolil()
        empty = np.asarray(abs(Ac).sum(1)).ravel() == 0
        Ac = Ac.tocsr() + sp.diags(empty.astype(float))
        if single:
            Ac.data = Ac.data.astype(np.float32).astype(np.float64)
        levels.append((A, Minv, P))
        A, active, mx, my = Ac.tocsr(), cact, cx, cy


def _vcycle(levels, b, l=0):
    A, Minv, P = levels[l]
    if P is None:
        return np.linalg.solve(A, b)
    nf = Minv.shape[1]
    sm = lambda r: OMEGA * np.einsum("nij,nj->ni", Minv, r.reshape(-1, nf)).ravel()  # noqa: E731
    sweeps = 1 if l == 0 else 2
    x = sm(b)
    for _ in range(sweeps - 1):
        x = x + sm(b - A @ x)
    x = x + P @ _vcycle(levels, P.T @ (b - A @ x), l + 1)
    for _ in range(sweeps):
        x = x + sm(b - A @ x)
    return x


# ---------------------------------------------------------------- the library
class _Gpu:
    def __init__(self, S, single, dev):
        from geowarp_b200 import _lib as L
        from geowarp_b200.engine import _p
        self.L, self.lib, self.p = L, L.load(), _p
        t = lambda a, d: torch.as_tensor(np.ascontiguousarray(a).astype(d), device=dev)  # noqa: E731
        self.keep = dict(row_ptr=t(S["row_ptr"], np.int32), cols=t(S["cols"], np.int32),
                         row2node=t(S["row2node"], np.int32), node2row=t(S["node2row"], np.int32),
                         stencil=t(S["stencil"], np.int32),
                         vals=t(S["vals"], np.float32 if single else np.float64))
        A = L.Bsr()
        A.n_rows, A.nf, A.nnzb, A.mask_words = S["n_rows"], S["nf"], S["cols"].size, 1
        for k, v in self.keep.items():
            setattr(A, k, _p(v))
        g = L.Grid()
        g.dim, g.nf = 2, S["nf"]
        for k, n in enumerate((S["mx"] - 1, S["my"] - 1)):
            g.n_grid[k], g.h[k], g.inv_h[k], g.h_nodes[k] = n, 1.0, 1.0, 1.0
        g.n_nodes = S["mx"] * S["my"]
        self.A, self.g, self.prec, self.dev = A, g, (L.PREC_F32 if single else L.PREC_F64), dev

    def solve(self, b, max_iter, rtol, restart=30):
        lib, p = self.lib, self.p
        nb = lib.gw_gmres_mg_workspace_bytes(C.byref(self.g), self.A.n_rows, self.A.nf, restart)
        # scratch that was never written must not reach a result
        ws = torch.full((nb,), 0xFF, dtype=torch.uint8, device=self.dev)
        bt = torch.as_tensor(b, device=self.dev)
        x = torch.zeros_like(bt)
        it, rr = C.c_int32(0), C.c_double(0.0)
        rc = lib.gw_bsr_gmres_mg_solve(C.byref(self.g), C.byref(self.A), self.prec, None, p(bt), p(x), rtol, max_iter,
                                       restart, p(ws), nb, C.byref(it), C.byref(rr), None)
        torch.cuda.synchronize()
        return x.cpu().numpy(), it.value, rr.value, rc


CASES = [  # nx, ny, nf, missing nodes, 25-point share
    (6, 4, 2, 0.0, 0.0),      # dense level only
    (9, 9, 2, 0.05, 0.3),     # two levels
    (15, 15, 1, 0.0, 0.0),    # 256 rows: whole chunks
    (30, 16, 2, 0.02, 1.0),   # 25-point rows throughout
    (41, 27, 3, 0.05, 0.2),   # u-p rows
    (63, 50, 4, 0.0, 0.1),
    (182, 180, 2, 0.0, 0.02),  # 33,123 rows: one lane per row on the finest level
    (130, 3, 2, 0.0, 0.5),    # a strip: coarse levels a few nodes wide
]


@pytest.mark.parametrize("single", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nf,holes,wide", CASES)
def test_one_iteration_shows_the_vcycle(cuda, nx, ny, nf, holes, wide, single):
    S = _system(nx, ny, nf, 7, holes, wide)
    rng = np.random.default_rng(1)
    b = rng.standard_normal(S["n_rows"] * nf)
    z = _vcycle(_hierarchy(S, single), b / np.linalg.norm(b))
    Az = S["A"] @ z
    want = z * (Az @ b) / (Az @ Az)
    x, it, rr, rc = _Gpu(S, single, cuda).solve(b, 1, 1e-30)
    assert it == 1
    err = np.abs(x - want).max() / np.abs(want).max()
    print(f"{nx}x{ny} nf {nf} {'mixed' if single else 'fp64'}: {err:.1e}")
    assert err < (1e-5 if single else 1e-11)


@pytest.mark.parametrize("single", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nf,holes,wide", CASES)
def test_converged_solve(cuda, nx, ny, nf, holes, wide, single):
    S = _system(nx, ny, nf, 8, holes, wide)
    rng = np.random.default_rng(2)
    xs = rng.uniform(-1, 1, S["n_rows"] * nf)
    b = S["A"] @ xs
    G = _Gpu(S, single, cuda)
    x, it, rr, rc = G.solve(b, 400, 1e-12, restart=10)  # a short basis: several cycles
    assert rc == G.L.GW_OK
    assert np.linalg.norm(S["A"] @ x - b) <= 2e-12 * np.linalg.norm(b)
    assert np.abs(x - xs).max() <= 9 * 2e-12 * np.sqrt(x.size) * np.abs(b).max()


def test_second_gram_schmidt_passes_do_not_change_the_solution(cuda):
    """GW_TUNE_GS_CANCEL = 0 repeats every projection, 300 none: same solution,
    and the count of second passes says so."""
    S = _system(30, 16, 2, 9, 0.02, 0.3)
    rng = np.random.default_rng(3)
    xs = rng.uniform(-1, 1, S["n_rows"] * 2)
    b = S["A"] @ xs
    G = _Gpu(S, False, cuda)
    default = G.lib.gw_tune_get(G.L.TUNE_GS_CANCEL)
    try:
        for knob in (0, 3, 300):
            assert G.lib.gw_tune_set(G.L.TUNE_GS_CANCEL, knob) == G.L.GW_OK
            x, it, rr, rc = G.solve(b, 400, 1e-12)
            re = G.lib.gw_gmres_last_reorths()
            assert rc == G.L.GW_OK
            assert np.abs(x - xs).max() <= 9 * 2e-12 * np.sqrt(x.size) * np.abs(b).max()
            assert (knob != 0 or re == it) and (knob != 300 or re == 0)
    finally:
        G.lib.gw_tune_set(G.L.TUNE_GS_CANCEL, default)


@pytest.mark.parametrize("single", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nf,holes,wide", [
    (9, 9, 2, 0.05, 0.3),     # one smoothed level: one CTA
    (15, 15, 1, 0.0, 0.0),    # 256 rows: two CTAs, every chunk whole
    (30, 16, 2, 0.02, 1.0),   # 25-point rows
    (41, 27, 3, 0.05, 0.2),
    (63, 50, 4, 0.0, 0.1),    # rows of a level over several passes of a warp
    (100, 80, 2, 0.0, 0.1),   # tail below the finest level by default, with it at 16384
])
def test_fused_tail_is_bitwise_the_separate_levels(cuda, nx, ny, nf, holes, wide, single):
    """GW_TUNE_MG_TAIL = 1 leaves every level its own launches; the default and
    16384 start the cluster at other levels.  Same arithmetic, same bytes."""
    S = _system(nx, ny, nf, 10, holes, wide)
    b = np.random.default_rng(4).standard_normal(S["n_rows"] * nf)
    G = _Gpu(S, single, cuda)
    default = G.lib.gw_tune_get(G.L.TUNE_MG_TAIL)
    out = []
    try:
        for knob in (1, 0, 16384):
            assert G.lib.gw_tune_set(G.L.TUNE_MG_TAIL, knob) == G.L.GW_OK
            out.append(G.solve(b, 12, 1e-30))
    finally:
        G.lib.gw_tune_set(G.L.TUNE_MG_TAIL, default)
    for x, it, rr, rc in out[1:]:
        assert it == out[0][1] and np.array_equal(x, out[0][0])
