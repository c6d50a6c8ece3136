"""The fused Gram-Schmidt step of GMRES at the edges of its work split: one to more than twelve values of w a
thread (the last kind keeps w in memory), and columns past the 64 whose rotations are done in shared memory.

Reference: a known solution.  The preconditioned residual ends below 1e-12 of its start; block diagonally dominant
systems (condition below 10 with the diagonal's inverses, below 50 without) then give x to 1e-10 in the 2-norm."""
import ctypes as ct
from types import SimpleNamespace

import numpy as np
import pytest


def _chains(copies, n):
    """Block rows in `copies` chains of n, the diagonal first in each row."""
    i = np.arange(copies * n)
    cols = [[k + 1] + [j + 1 for j in (k - 1, k + 1) if 0 <= j < copies * n and j // n == k // n] for k in i]
    return SimpleNamespace(nf=copies * n, cbsr_rowpts=np.cumsum([0] + [len(c) for c in cols]), cbsr_colind=np.concatenate(cols))


def _solve(copies, n, bs, offdiag, diag, restart, precondition, seed=0):
    import torch
    from hdg_b200._lib import HdgxBsr, check, lib
    from hdg_b200.elemental import DArray
    from hdg_b200.ordering import levels_of_order, sweep_plan
    mesh = _chains(copies, n)
    nf, nnzb = mesh.nf, len(mesh.cbsr_colind)
    order = np.arange(nf, dtype=np.int32)
    lv = levels_of_order(mesh.cbsr_rowpts, mesh.cbsr_colind, order, order)
    plan, maxd = sweep_plan(lv, mesh.cbsr_rowpts, mesh.cbsr_colind)
    keep = [DArray.from_numpy(mesh.cbsr_rowpts, dtype=torch.int64)] + [
        DArray.from_numpy(a, dtype=torch.int32) for a in (mesh.cbsr_colind, lv.color_rows, lv.pos, plan)]
    ptr = np.ascontiguousarray(lv.color_ptr, dtype=np.int32)
    A = HdgxBsr(nf, bs, nnzb, keep[0].ptr, keep[1].ptr, lv.ncolors, ptr.ctypes.data, keep[2].ptr, keep[3].ptr, None,
                keep[4].ptr, maxd)
    g = torch.Generator("cuda").manual_seed(seed)
    at = torch.as_tensor(mesh.cbsr_rowpts[:-1], device="cuda")
    eye = torch.eye(bs, dtype=torch.float64, device="cuda")
    H = offdiag(torch.randn(nnzb, bs, bs, generator=g, dtype=torch.float64, device="cuda"), eye)
    H[at] = diag * eye + (H[at] if precondition else 0.0)
    M = torch.zeros_like(H)                              # the diagonal's inverses (BILU(0) of a chain would be exact)
    M[at] = torch.linalg.inv(H[at].transpose(1, 2)).transpose(1, 2).contiguous() if precondition else eye
    x0 = torch.randn(nf * bs, generator=g, dtype=torch.float64, device="cuda")
    b, x = torch.empty_like(x0), torch.zeros_like(x0)
    check(lib().hdgx_matvec(ct.byref(A), H.data_ptr(), x0.data_ptr(), b.data_ptr(), None), "hdgx_matvec")
    it, fl, rr = ct.c_int(0), ct.c_int(0), ct.c_double(0.0)
    check(lib().hdgx_gmres_bilu0(ct.byref(A), H.data_ptr(), M.data_ptr(), b.data_ptr(), x.data_ptr(), restart, 1e-12, 400,
                                 ct.byref(it), ct.byref(fl), ct.byref(rr), None, None, None), "hdgx_gmres_bilu0")
    torch.cuda.synchronize()
    assert fl.value == 0
    assert float((x - x0).norm() / x0.norm()) < 1e-10
    return it.value


@pytest.mark.gpu
@pytest.mark.parametrize("copies,bs", [(1, 8), (1300, 8), (3600, 8), (6000, 8), (4400, 30)])
def test_values_per_thread(copies, bs):
    """56 to 924,000 unknowns: 1, 1, 3, 5 and 13 a thread of 148 blocks of 512."""
    assert _solve(copies, 7, bs, lambda r, eye: r / bs, 4.0, 20, True) > 1


@pytest.mark.gpu
def test_more_columns_than_rotations_in_shared_memory():
    """One long chain like -u'' + 0.1 u without a preconditioner: more than 64 steps of one cycle."""
    assert _solve(1, 200, 8, lambda r, eye: -eye + 0.0 * r, 2.1, 150, False) > 64
