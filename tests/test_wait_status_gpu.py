"""A sweep whose wait for a value runs out is an error of the solve that contains it, not a converged solve.

The plan of tests/test_sweep_gpu.py that is no schedule: a row is said to need itself, its bounded wait ends and
the sweep goes on with NaN.  hdgx_gmres_bilu0 and its mixed and allocation-free forms then return status -16; the
next solve, with the right plan, converges.  A right-hand side that is not a number is no converged solve either
(flag 3, as for a residual that is not finite); one of zeros is (flag 0, x as it was)."""
import ctypes as ct

import numpy as np
import pytest

from test_sweep_gpu import _system


def _solve(ts, form, H, M, b, x):
    import torch
    from hdg_b200._lib import check, lib
    if form == "noalloc":
        it, fl, rr = ct.c_int(0), ct.c_int(0), ct.c_double(0.0)
        check(lib().hdgx_gmres_bilu0_noalloc(ct.byref(ts.bsr), H.ptr, M.ptr, b.ptr, x.ptr, 20, 1e-10, 200, ct.byref(it),
                                             ct.byref(fl), ct.byref(rr), None, None), "hdgx_gmres_bilu0_noalloc")
        return it.value, fl.value, rr.value
    if form == "mixed":
        return ts.gmres_mixed(H, M, torch.empty(M.t.numel(), dtype=torch.float32, device="cuda"), b, x, 20, 1e-10, 200)[:3]
    return ts.gmres(H, M, b, x, 20, 1e-10, 200)[:3]


def _identity(ts):
    import torch
    I = ts.empty_blocks()
    I.t.zero_()
    I.t.view(ts.nnzb, ts.bs, ts.bs)[torch.as_tensor(ts.rowpts_h[:-1], device="cuda")] = torch.eye(
        ts.bs, dtype=torch.float64, device="cuda")
    return I


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "mixed", "noalloc"])
def test_wait_that_runs_out(oracle, form):
    import torch
    from hdg_b200._lib import HdgxError
    P, ts, dM, DArray = _system(oracle, "c1", dict(n=3, porder=2))
    good, plan = ts.bsr.sweep_plan, ts.d["sweep_plan"].numpy().copy().ravel()
    rec = plan[ts.bsr.ncolors + 1:].reshape(ts.nf, 2 + 4 * ts.bsr.sweep_maxd)
    q = int(np.flatnonzero(rec[:, 2] >= 0)[0])
    rec[q, 3] = rec[q, 0]
    bad = DArray.from_numpy(plan, dtype=torch.int32)
    b = DArray.from_numpy(np.random.default_rng(7).standard_normal((ts.bs, ts.nf)))
    x = ts.empty_vec()
    x.t.zero_()
    ts.bsr.sweep_plan = bad.ptr
    try:
        with pytest.raises(HdgxError) as e:
            _solve(ts, form, _identity(ts), dM, b, x)
        assert "status -16" in str(e.value)
    finally:
        ts.bsr.sweep_plan = good
    x.t.zero_()
    it, fl, rr = _solve(ts, form, _identity(ts), _identity(ts), b, x)
    assert fl == 0 and it >= 1 and np.abs(x.numpy() - b.numpy()).max() < 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "mixed", "noalloc"])
def test_right_hand_side_that_is_not_a_number(oracle, form):
    P, ts, dM, DArray = _system(oracle, "c1", dict(n=3, porder=2))
    b, x = np.zeros((ts.bs, ts.nf)), ts.empty_vec()
    x.t.fill_(0.5)
    it, fl, rr = _solve(ts, form, _identity(ts), dM, DArray.from_numpy(b), x)
    assert (it, fl, rr) == (0, 0, 0.0) and (x.numpy() == 0.5).all()
    b[1, 2] = np.nan
    it, fl, rr = _solve(ts, form, _identity(ts), dM, DArray.from_numpy(b), x)
    assert fl == 3
