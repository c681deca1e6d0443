"""Grids of more cells than the 2D assembly sums at once go in bands of rows of cells.
The particles of a part of the width, few enough to be summed at once, are assembled
in the same grid: away from the cut the rows are bitwise the same, across every band.

Against the atomic assembly (same terms in another order): R to 1e-12 of its largest
entry; K to 1e-12 where the values are FP64 and 1e-6 (a few roundings of 2^-24) where
they are FP32.  Not for the wide grid, where a position is 40,000 cells from the origin
and a weight's rounding in the two kernels is no longer 1e-12."""
import numpy as np
import pytest
import torch

from test_gpu_cell_sums import _engine

pytestmark = pytest.mark.gpu


def _rows(e, K, nodes):
    """Blocks of the rows of these nodes, one after the other, and their lengths."""
    r = e.node2row[nodes].long()
    rp = e._row_ptr.long()
    n = rp[r + 1] - rp[r]
    start = torch.repeat_interleave(rp[r] - (n.cumsum(0) - n), n)
    return K.view(-1, 4)[start + torch.arange(int(n.sum()), device=K.device)], n, r


@pytest.mark.parametrize("n_cells,n,cut,precision,atomic", [
    ((760, 760), 620000, 400, "fp64", True),   # two bands (689 rows of cells and the rest), all cells
    ((800, 760), 560000, 400, "mixed", True),  # fewer particles than cells, more than a band
    ((40000, 30), 1300000, 15000, "mixed", False),  # wide: bands of 16 rows of cells
])
def test_banded_assembly(cuda, n_cells, n, cut, precision, atomic):
    rng = np.random.default_rng(1)
    x = rng.uniform([0.5, 0.5], [n_cells[0] - 0.5, n_cells[1] - 0.5], (n, 2))
    vt = torch.float64 if precision == "fp64" else torch.float32
    g = torch.Generator().manual_seed(2)
    u = 1e-4 * torch.randn(2 * (n_cells[0] + 1) * (n_cells[1] + 1), dtype=torch.float64, generator=g)

    def run(x, det=True):
        s = _engine(n_cells, x, np.full((len(x), 2), 0.2499), precision, "Hencky elasticity", cuda)
        e = s.engine
        s._set_step_params()
        s.reset()
        e.sort_and_activate()
        e.build_system()
        e.u_new.copy_(u)
        e.deterministic_assembly = det
        e._vals.t.fill_(0xFF)  # nothing may be left of what was there before
        e._R.fill_(float("nan"))
        e.assemble(s._mat, 0, 10)
        K = e._vals.t[: e.nnzb * 4 * (8 if precision == "fp64" else 4)].view(vt).clone()
        R = e._R[: e.n_rows * 2].clone()
        assert e.device_status() == 0
        e.assemble(s._mat, 0, 10, want_K=False)
        if det:
            assert torch.equal(e._R[: e.n_rows * 2], R)
        return e, R, K

    e, R, K = run(x)
    p, Rp, Kp = run(x[x[:, 0] < cut])
    nodes = torch.nonzero(e.node_active).flatten()
    nodes = nodes[nodes % (n_cells[0] + 1) < cut - 4]
    B, nb, r = _rows(e, K, nodes)
    Bp, nbp, rp = _rows(p, Kp, nodes)
    assert int(nodes.numel()) > 0.3 * cut * n_cells[1]
    assert torch.equal(nb, nbp) and torch.equal(B, Bp)
    assert torch.equal(R.view(-1, 2)[r], Rp.view(-1, 2)[rp])
    if atomic:
        _, Ra, Ka = run(x, det=False)
        assert float((R - Ra).abs().max()) <= 1e-12 * float(Ra.abs().max())
        tol = 1e-12 if precision == "fp64" else 1e-6
        assert float((K.double() - Ka.double()).abs().max()) <= tol * float(Ka.abs().max())
