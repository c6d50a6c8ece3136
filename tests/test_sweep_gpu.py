"""The data-driven BILU(0) sweeps (one launch per apply) at the edges of their work split.

Reference: the oracle's applyBILU0 on the oracle's factors of the same order.  Tolerance 1e-12
of the largest entry, that of the other trace-system tests.  Block sizes 8 to 30 (2D p = 1..4,
3D p = 1, 2), FP64 and FP32 factors (the FP32 reference is the oracle on the rounded factors),
grids from one cluster of one CTA to a cooperative launch, and the solution written over the
right-hand side."""
import ctypes as ct

import numpy as np
import pytest

from hdg_b200 import configs

CASES = [("c1", dict(n=1, porder=1)), ("c1", dict(n=9, porder=1)), ("c1", dict(n=5, porder=2)), ("c2", dict(n=7, porder=3)),
         ("c1", dict(n=3, porder=4)), ("c4", dict(n=1, porder=1)), ("c4", dict(n=3, porder=1)), ("c4", dict(n=1, porder=2)),
         ("c4", dict(n=5, porder=2))]


def _system(oracle, name, kw):
    from hdg_b200.elemental import DArray, hdg_elemental
    from hdg_b200.solve import TraceSystem
    P = configs.by_name(name, **kw)
    r = hdg_elemental(P.master, P.app, P.mesh.dgnodes, P.mesh.bf, P.UDG, P.uh_elem(), P.SH)
    ts = TraceSystem(P.mesh, P.master, P.app)
    dH, dR, dM = ts.empty_blocks(), ts.empty_vec(), ts.empty_blocks()
    ts.assemble(r.AE, r.FE, dH, dR)
    ts.bilu0(dH, dM)
    assert ts.bsr.sweep_plan
    return P, ts, dM, DArray


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", CASES)
def test_apply_matches_oracle(oracle, name, kw):
    P, ts, dM, DArray = _system(oracle, name, kw)
    x = np.random.default_rng(3).standard_normal((ts.bs, ts.nf))
    ref = oracle.bilu0_apply(P.mesh, dM.numpy(), x, ts.o2u, ts.u2o)
    v, w = ts.empty_vec(), ts.empty_vec()
    for _ in range(3):                                   # the vectors hold the last call's values
        ts.bilu0_apply(dM, DArray.from_numpy(x), v, w)
        assert _rel(v.numpy(), ref) < 1e-12
    d = DArray.from_numpy(x)
    ts.bilu0_apply(dM, d, d, w)                          # in place
    assert _rel(d.numpy(), ref) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", CASES)
def test_fp32_factors_match_oracle(oracle, name, kw):
    import torch
    from hdg_b200._lib import lib
    P, ts, dM, DArray = _system(oracle, name, kw)
    # one GMRES step from x0 = 0 with a single basis vector: x is a multiple of P^-1 b
    Mg32 = torch.empty(dM.t.numel(), dtype=torch.float32, device="cuda")
    b = np.random.default_rng(4).standard_normal((ts.bs, ts.nf))
    x, I = ts.empty_vec(), ts.empty_blocks()
    x.t.zero_()
    I.t.zero_()                                          # the identity as the system matrix
    blocks = I.t.view(ts.nnzb, ts.bs, ts.bs)
    blocks[torch.as_tensor(ts.rowpts_h[:-1], device="cuda")] = torch.eye(ts.bs, dtype=torch.float64, device="cuda")
    ts.gmres_mixed(I, dM, Mg32, DArray.from_numpy(b), x, 1, 1e-30, 1)
    M32 = dM.numpy().astype(np.float32).astype(np.float64)
    z = oracle.bilu0_apply(P.mesh, M32, b, ts.o2u, ts.u2o)
    Az = oracle.bilu0_apply(P.mesh, M32, z, ts.o2u, ts.u2o)
    ref = z * ((Az * z).sum() / (Az * Az).sum())
    assert _rel(x.numpy(), ref) < 1e-11                  # two applications and the two products' ratio


@pytest.mark.gpu
def test_not_a_number_in_is_not_a_number_out(oracle):
    """A right-hand side of NaNs with every bit set (the marker of a value not yet written) ends, and ends in NaN."""
    import torch
    P, ts, dM, DArray = _system(oracle, "c1", dict(n=3, porder=2))
    x = ts.empty_vec()
    x.t.view(torch.int64).fill_(-1)
    v, w = ts.empty_vec(), ts.empty_vec()
    ts.bilu0_apply(dM, x, v, w)
    assert bool(torch.isnan(v.t).all())


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [("c1", dict(n=5, porder=2)), ("c4", dict(n=3, porder=2))])
def test_factors_at_8_byte_alignment(oracle, name, kw):
    """Factors that no 16-byte copy can read: each value is staged by itself."""
    import torch
    from hdg_b200._lib import check, lib
    P, ts, dM, DArray = _system(oracle, name, kw)
    x = np.random.default_rng(5).standard_normal((ts.bs, ts.nf))
    ref = oracle.bilu0_apply(P.mesh, dM.numpy(), x, ts.o2u, ts.u2o)
    M = torch.empty(dM.t.numel() + 1, dtype=torch.float64, device="cuda")[1:]
    M.copy_(dM.t.view(-1))
    assert M.data_ptr() % 16 == 8
    d, v, w = DArray.from_numpy(x), ts.empty_vec(), ts.empty_vec()
    check(lib().hdgx_bilu0_apply(ct.byref(ts.bsr), M.data_ptr(), d.ptr, v.ptr, w.ptr, None), "hdgx_bilu0_apply")
    torch.cuda.synchronize()
    assert _rel(v.numpy(), ref) < 1e-12


@pytest.mark.gpu
def test_vectors_that_share_storage_in_part(oracle):
    """The work vector over the right-hand side: one launch per level instead."""
    P, ts, dM, DArray = _system(oracle, "c1", dict(n=5, porder=2))
    x = np.random.default_rng(6).standard_normal((ts.bs, ts.nf))
    ref = oracle.bilu0_apply(P.mesh, dM.numpy(), x, ts.o2u, ts.u2o)
    d, v = DArray.from_numpy(x), ts.empty_vec()
    ts.bilu0_apply(dM, d, v, d)
    assert _rel(v.numpy(), ref) < 1e-12


@pytest.mark.gpu
def test_plan_that_is_no_schedule_ends_in_nan(oracle):
    """A row that is said to need itself: its wait runs out, the result is NaN, and the next call is right."""
    import torch
    P, ts, dM, DArray = _system(oracle, "c1", dict(n=3, porder=2))
    x = np.random.default_rng(7).standard_normal((ts.bs, ts.nf))
    good, plan = ts.bsr.sweep_plan, ts.d["sweep_plan"].numpy().copy().ravel()
    rec = plan[ts.bsr.ncolors + 1:].reshape(ts.nf, 2 + 4 * ts.bsr.sweep_maxd)
    q = int(np.flatnonzero(rec[:, 2] >= 0)[0])
    rec[q, 3] = rec[q, 0]
    bad = DArray.from_numpy(plan, dtype=torch.int32)
    v, w = ts.empty_vec(), ts.empty_vec()
    ts.bsr.sweep_plan = bad.ptr
    ts.bilu0_apply(dM, DArray.from_numpy(x), v, w)
    torch.cuda.synchronize()
    ts.bsr.sweep_plan = good
    assert np.isnan(v.numpy()).any()
    ts.bilu0_apply(dM, DArray.from_numpy(x), v, w)
    assert _rel(v.numpy(), oracle.bilu0_apply(P.mesh, dM.numpy(), x, ts.o2u, ts.u2o)) < 1e-12
