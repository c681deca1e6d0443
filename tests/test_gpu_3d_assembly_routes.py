"""The 3D assembly's two kernels: which one a call takes, and that both give the same
residual, tangent and footing force.

Both add the same terms with atomics in another order: 1e-12 of the largest entry."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(cells, dev):
    from geowarp_b200 import problems
    s = problems.indentation_3d(precision="fp64", precond="block", block_cells=cells,
                                grid_cells=tuple(c + 2 for c in cells), dx=0.25, E=1e3, material="Neo-Hookean",
                                permeability=1e-11, indenter=0.5, depth=0.5, n_steps=25, penalty=1000.0)
    e = s.engine
    s._sync_grid()
    s._set_step_params()
    s.reset()
    e.sort_and_activate()
    e.project_pressure()
    e.build_system()
    g = torch.Generator().manual_seed(1)
    e.u_new += 1e-4 * torch.randn(e.u_new.shape, dtype=torch.float64, generator=g).to(dev)
    return e, s._mat


@pytest.mark.parametrize("cells,want_K,single_thread", [
    ((10, 10, 10), False, False),  # 8,000 particles
    ((11, 11, 11), False, True),   # 10,648
    ((16, 16, 16), True, False),   # 32,768: a wave 86% full
    ((17, 17, 16), True, True),    # 36,992: 98% full
])
def test_route_and_values(cuda, cells, want_K, single_thread):
    from geowarp_b200 import _lib as L
    from geowarp_b200.engine import _p
    e, mat = _engine(cells, cuda)
    g, st, n = e.grid_struct(), e.step_struct(0, 25), e.n_rows * 4
    K = e._vals.t[: e.nnzb * 16 * 8].view(torch.float64)

    def run(parts):
        R, f = torch.zeros(n, dtype=torch.float64, device=cuda), torch.zeros(1, dtype=torch.float64, device=cuda)
        Ks, Rs = torch.zeros_like(K), torch.zeros_like(R)
        for lo, hi in parts:
            pt, A = e.particles_struct(), e.bsr_struct()
            pt.n = hi - lo
            if not want_K:
                A.vals = None
            L.call("gw_assemble", C.byref(g), C.byref(mat), C.byref(st), C.byref(pt), _p(e.perm[lo:hi].contiguous()),
                   _p(e.free_mask), _p(e.u_new), _p(e.u_old), C.byref(A), e.prec, _p(R), _p(f), e.stream)
            Rs += R
            if want_K:
                Ks += K
        return Rs, Ks, float(f.item())

    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        R, Kw, f = run([(0, e.N)])
    names = [ev.name for ev in prof.events()]
    assert any("k_assemble3" in k for k in names) != single_thread
    assert any("k_assemble" in k and "k_assemble3" not in k for k in names) == single_thread
    third = e.N // 3  # 3,552 or fewer particles a call without a tangent, 12,331 with one: the other kernel
    R3, K3, f3 = run([(0, third), (third, 2 * third), (2 * third, e.N)])
    assert float((R - R3).abs().max()) <= 1e-12 * float(R.abs().max())
    assert abs(f - f3) <= 1e-12 * abs(f)
    if want_K:
        # the identity rows of Dirichlet DOFs are written by every launch
        one = (Kw == 1.0) & (K3 == 3.0)
        K3[one] = 1.0
        assert float((Kw - K3).abs().max()) <= 1e-12 * float(Kw.abs().max())
