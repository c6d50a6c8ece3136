"""3D p = 2 (blocks of 30, products added as neighbours arrive): the promises of the same bits that the header and
the serving layer make.  The allocation-free GMRES against the allocating one; Newton solves on three threads and
streams at once, plain and through a combiner, against the same solves one after another."""
import ctypes as ct
import threading

import numpy as np
import pytest

from hdg_b200 import configs
from test_sweep_gpu import _system


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 5])
def test_allocation_free_gmres(oracle, n):
    import torch
    from hdg_b200._lib import check, lib
    P, ts, dM, DArray = _system(oracle, "c4", dict(n=n, porder=2))
    gen = torch.Generator("cuda").manual_seed(1)
    b = DArray(torch.randn(ts.bs * ts.nf, dtype=torch.float64, device="cuda", generator=gen), (ts.bs, ts.nf))
    H = ts.empty_blocks()
    H.t.copy_(dM.t)                                      # any matrix of the pattern: its factors precondition themselves
    x, y = ts.empty_vec(), ts.empty_vec()
    for _ in range(3):
        x.t.zero_()
        y.t.zero_()
        ref = ts.gmres(H, dM, b, x, 20, 1e-10, 45)
        it, fl, rr = ct.c_int(0), ct.c_int(0), ct.c_double(0.0)
        check(lib().hdgx_gmres_bilu0_noalloc(ct.byref(ts.bsr), H.ptr, dM.ptr, b.ptr, y.ptr, 20, 1e-10, 45, ct.byref(it),
                                             ct.byref(fl), ct.byref(rr), None, None), "hdgx_gmres_bilu0_noalloc")
        torch.cuda.synchronize()
        assert (it.value, fl.value, rr.value) == ref[:3] and it.value > 1
        assert torch.equal(x.t.view(torch.int64), y.t.view(torch.int64))


@pytest.mark.gpu
@pytest.mark.parametrize("combined", [False, True])
def test_solves_alone_and_together(combined):
    import torch
    from hdg_b200.solve import Combiner, hdgx_solve
    problems = [configs.by_name("c4", n=n, porder=2) for n in (3, 4, 3)]

    def solve(P, stream=None, comb=None):
        U, H, rep = hdgx_solve(P.master, P.mesh, P.app, P.UDG, P.UH, P.SH, tol=1e-10, maxiter=2, stream=stream, combiner=comb)
        return U, H, rep["residuals"], rep["gmres_iters"]
    alone = [solve(P) for P in problems]
    comb = Combiner(1000) if combined else None
    out = [None] * len(problems)

    def run(i):
        torch.cuda.set_device(0)
        st = torch.cuda.Stream()
        out[i] = solve(problems[i], st, comb)
    ts = [threading.Thread(target=run, args=(i,)) for i in range(len(problems))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, b in zip(alone, out):
        assert np.array_equal(a[0].view(np.int64), b[0].view(np.int64)) and np.array_equal(a[1].view(np.int64), b[1].view(np.int64))
        assert a[2:] == b[2:]
