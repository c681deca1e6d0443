"""Solves on several host threads of one device, each with its own matrix, vectors,
workspace and stream: every result is bitwise the one the same solve gives alone."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(seed, n=150, nf=4):
    """Diagonally dominant block rows of 20 to 60 blocks."""
    rng = np.random.default_rng(seed)
    cols = [np.sort(np.append(rng.choice(np.delete(np.arange(n), r), int(rng.integers(19, 60)), replace=False), r))
            for r in range(n)]
    i, j = np.concatenate([np.full(c.size, r) for r, c in enumerate(cols)]), np.concatenate(cols)
    vals = rng.uniform(-1, 1, (i.size, nf, nf))
    k = np.arange(nf)
    d = np.nonzero(i == j)[0]
    vals[d[:, None], k, k] = 60 * nf
    return np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]), j, vals


class _Block:
    """A node-block GMRES solve that runs to max_iter."""

    def __init__(self, seed, dev):
        from geowarp_b200 import _lib as L
        from geowarp_b200.engine import _p
        self.L, self.lib, self.p = L, L.load(), _p
        rp, cols, vals = _rows(seed)
        n, nf = rp.size - 1, vals.shape[1]
        t = lambda a, d: torch.as_tensor(np.ascontiguousarray(a).astype(d), device=dev)  # noqa: E731
        self.keep = dict(row_ptr=t(rp, np.int32), cols=t(cols, np.int32), row2node=t(np.arange(n), np.int32),
                         node2row=t(np.arange(n), np.int32), stencil=t(np.zeros(4 * n), np.int32), vals=t(vals, np.float64))
        self.A = L.Bsr()
        self.A.n_rows, self.A.nf, self.A.nnzb, self.A.mask_words = n, nf, cols.size, 4
        for name, v in self.keep.items():
            setattr(self.A, name, _p(v))
        self.b = torch.as_tensor(np.random.default_rng(seed).standard_normal(n * nf), device=dev)
        self.x = torch.zeros_like(self.b)
        self.ws = torch.empty(self.lib.gw_gmres_workspace_bytes(n, nf, 40), dtype=torch.uint8, device=dev)

    def solve(self, q):
        s = torch.cuda.current_stream()
        self.x.zero_()
        it, rr = C.c_int32(0), C.c_double(0.0)
        # 9 .. 99 columns: with and without replayed columns, one to three cycles
        rc = self.lib.gw_bsr_gmres_solve(C.byref(self.A), self.L.PREC_F64, 1, self.p(self.b), self.p(self.x), 1e-300,
                                         9 + 30 * (q % 4), 40, self.p(self.ws), C.byref(it), C.byref(rr),
                                         C.c_void_p(s.cuda_stream))
        s.synchronize()
        return rc, it.value, self.x.cpu().numpy()


def _run(make, n_threads, n_solves):
    jobs = [make(t) for t in range(n_threads)]
    torch.cuda.synchronize()
    want = [[j.solve(q) for q in range(n_solves)] for j in jobs]
    got, errors = [[] for _ in jobs], []
    start = threading.Barrier(n_threads)

    def work(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for q in range(n_solves):
                    got[t].append(jobs[t].solve(q))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(n_threads)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, w in zip(got, want):
        for (rc, it, x), (rc0, it0, x0) in zip(g, w):
            assert rc == rc0 and it == it0 and np.array_equal(x, x0)
    return want


def test_node_block_gmres_on_several_host_threads(cuda):
    from geowarp_b200 import _lib as L
    want = _run(lambda t: _Block(t, cuda), 4, 24)
    assert all(rc == L.GW_ENOCONV and it == 9 + 30 * (q % 4) for w in want for q, (rc, it, _) in enumerate(w))


class _Multigrid:
    """A multigrid solve; each restart length is a graph of its own, so the threads
    together need more graphs than the library keeps."""

    def __init__(self, seed, dev):
        from test_gpu_mg_rows import _Gpu, _system
        self.g = _Gpu(_system(20 + seed, 17, 2, seed, 0.02, 0.2), False, dev)
        g, lib = self.g, self.g.lib
        n = g.A.n_rows * 2
        self.nb = lib.gw_gmres_mg_workspace_bytes(C.byref(g.g), g.A.n_rows, 2, 20)
        self.ws = torch.empty(self.nb, dtype=torch.uint8, device=dev)
        self.b = torch.as_tensor(np.random.default_rng(seed).standard_normal(n), device=dev)
        self.x = torch.zeros_like(self.b)

    def solve(self, q):
        g, s = self.g, torch.cuda.current_stream()
        self.x.zero_()
        it, rr = C.c_int32(0), C.c_double(0.0)
        rc = g.lib.gw_bsr_gmres_mg_solve(C.byref(g.g), C.byref(g.A), g.prec, None, g.p(self.b), g.p(self.x), 1e-300, 25,
                                         15 + q % 6, g.p(self.ws), self.nb, C.byref(it), C.byref(rr),
                                         C.c_void_p(s.cuda_stream))
        s.synchronize()
        return rc, it.value, self.x.cpu().numpy()


def test_multigrid_gmres_on_several_host_threads(cuda):
    from geowarp_b200 import _lib as L
    want = _run(lambda t: _Multigrid(t, cuda), 4, 24)
    assert all(rc == L.GW_ENOCONV and it == 25 for w in want for rc, it, _ in w)
