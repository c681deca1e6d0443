"""What a row or a particle costs in the workspaces that the library asks for (host
arithmetic: no GPU)."""
import ctypes as C

import pytest

from geowarp_b200 import _lib as L


def _grid(kind, nx, ny):
    g = L.Grid()
    g.dim, g.kind, g.nf, g.n_nodes = 2, kind, 2 if kind == L.KIND_SOLID2D else 3, (nx + 1) * (ny + 1)
    for k, n in enumerate((nx, ny)):
        g.n_grid[k], g.h[k], g.inv_h[k], g.h_nodes[k] = n, 1.0, 1.0, 1.0
    return g


@pytest.mark.parametrize("nf", [2, 3])
@pytest.mark.parametrize("lo,hi,slots", [(40000, 200000, 25), (4000, 20000, 28)])
def test_multigrid_bytes_per_finest_row(lo, hi, slots, nf):
    """The basis, the row vectors and one copy of the matrix in sliced rows (25 slots,
    28 below 24,576 rows), whose FP64 slots also hold the mixed solve's BF16 copy."""
    lib = L.load()
    g = _grid(L.KIND_SOLID2D, 499, 499)
    restart = 30
    a, b = (lib.gw_gmres_mg_workspace_bytes(C.byref(g), n, nf, restart) for n in (lo, hi))
    vectors = 8 * nf * (2 * restart + 2 + 4) + 8 * nf * nf + 4 * 4 + 1
    matrix = slots * (4 + 8 * nf * nf) + 4 / 8
    assert (b - a) / (hi - lo) <= vectors + matrix + 0.5  # every array is rounded to 256 bytes


@pytest.mark.parametrize("kind,nf", [(L.KIND_SOLID2D, 2), (L.KIND_COUPLED2D, 3)])
@pytest.mark.parametrize("nx,ny,n", [(2000, 2000, 16000000), (2000, 2000, 3000000), (100000, 60, 24000000)])
def test_assembly_bytes_are_bounded(kind, nf, nx, ny, n):
    """Beside the particle records and three words a cell: the sums (81 blocks and nine
    nodes' residuals, FP64) of half a million cells, or of 16 rows of cells."""
    lib = L.load()
    g = _grid(kind, nx, ny)
    rec = (lib.gw_assemble_workspace_bytes(C.byref(_grid(kind, 1, 1)), 200000, L.PREC_F64)
           - lib.gw_assemble_workspace_bytes(C.byref(_grid(kind, 1, 1)), 100000, L.PREC_F64)) / 100000
    sums = 8 * (81 * nf * nf + 9 * nf + 1) * max(2 ** 19, 16 * nx)
    assert lib.gw_assemble_workspace_bytes(C.byref(g), n, L.PREC_F64) <= (rec + 0.01) * n + 12 * nx * ny + sums + 4096
