"""The FP64 elemental kernel's tensor-core products over every compiled shape and output form.

Reference: the oracle.  AE, FE and DUDG_DUH within 1e-12 of their largest entry, the bound of the
other elemental tests; DUDG, an ill-conditioned difference, within 10 x the change that one-ulp
perturbations of the inputs make in the oracle's own DUDG, or 1e-12 (tests/test_elemental_gpu.py).
An odd number of elements; jittered, mid-Newton states (gradients and a trace off the element
values); with and without the q rows (getdqdg), time-dependent, and into outputs that are only
8-byte aligned."""
import copy

import numpy as np
import pytest

from hdg_b200.app import freestream, make_app
from hdg_b200.configs import Problem
from hdg_b200.master import mkmaster
from hdg_b200.mesh import mkmesh_cube, mkmesh_square

SHAPES = [(nd, p, v) for nd, ps in ((2, (1, 2, 3, 4)), (3, (1, 2, 3))) for p in ps for v in (False, True)]

# launches of more elements than one wave of the shape for few elements: the narrower CTAs of the small plans
NARROW = [(2, 1, False), (2, 1, True), (2, 2, False), (2, 2, True), (2, 3, False), (3, 1, False), (3, 1, True)]


class _Elements(Problem):
    def uh_elem(self, UH=None):
        return self.UH if UH is None else UH


def _state(nd, p, visc, tdep=False, n=None):
    r = np.random.default_rng(100 * nd + 10 * p + visc)
    mesh = mkmesh_square(n or 4, n or 4, p) if nd == 2 else mkmesh_cube(n or 2, n or 2, n or 2, p)
    master = mkmaster(nd, p, 2 * p)
    app = make_app(nd, re=300.0 if visc else np.inf, minf=0.5)
    if tdep:
        app.tdep, app.fc_u = 1, 20.0
    ne = mesh.ne - 1 if mesh.ne % 2 == 0 else mesh.ne
    mesh = copy.copy(mesh)
    J = np.eye(nd) + 0.15 * r.standard_normal((nd, nd))              # one affine map: straight-sided, not aligned
    mesh.dgnodes = np.asfortranarray(np.einsum("ij,kje->kie", J, mesh.dgnodes[..., :ne]))
    mesh.bf = np.asfortranarray(mesh.bf[:, :ne])
    base = freestream(nd, 1.4, 0.5)
    ncu, ndf = app.ncu, master.npf * master.nfe
    u = base[None, :, None] * (1 + 0.05 * r.standard_normal((master.npv, ncu, ne)))
    q = 0.2 * r.standard_normal((master.npv, ncu * nd, ne))
    uh = base[:, None, None] * (1 + 0.05 * r.standard_normal((ncu, ndf, ne)))
    udg = np.asfortranarray(np.concatenate([u, q], 1))
    sh = np.zeros_like(udg)
    if tdep:
        sh[:, :ncu] = app.fc_u * (u + 0.01)
    return _Elements("state", master, mesh, app, udg, np.asfortranarray(uh), sh)


def _check(oracle, P, out):
    from test_elemental_gpu import ulp_sensitivity
    m = P.mesh
    ref = oracle.hdg_elemental(P.master, P.app, m.dgnodes, m.bf, P.UDG, P.UH, P.SH)
    assert ref["nbad"] == 0 and int(out.status.numpy().max()) == 0
    for k in ("AE", "FE", "DUDG_DUH", "DUDG"):
        tol = max(1e-12, 10 * ulp_sensitivity(oracle, P)) if k == "DUDG" else 1e-12
        err = float(np.abs(getattr(out, k).numpy() - ref[k]).max() / np.abs(ref[k]).max())
        assert err < tol, f"{k} {err:.2e}"


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,visc", SHAPES)
@pytest.mark.parametrize("getdqdg,tdep", [(1, False), (0, False), (1, True)])
def test_every_shape_matches_oracle(oracle, nd, p, visc, getdqdg, tdep):
    from hdg_b200.elemental import hdg_elemental
    P = _state(nd, p, visc, tdep)
    P.app.getdqdg = getdqdg
    _check(oracle, P, hdg_elemental(P.master, P.app, P.mesh.dgnodes, P.mesh.bf, P.UDG, P.UH, P.SH))


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,visc", NARROW)
def test_many_elements_match_oracle(oracle, nd, p, visc):
    from hdg_b200.elemental import hdg_elemental
    P = _state(nd, p, visc, n=25 if nd == 2 else 6)                      # 1,249 and 1,079 elements
    _check(oracle, P, hdg_elemental(P.master, P.app, P.mesh.dgnodes, P.mesh.bf, P.UDG, P.UH, P.SH))


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,visc", SHAPES)
def test_outputs_at_8_byte_alignment(oracle, nd, p, visc):
    import torch
    from hdg_b200.elemental import DArray, ElementalOutputs, alloc_elemental_outputs, hdg_elemental
    P = _state(nd, p, visc)

    def shifted(a):
        t = torch.empty(a.t.numel() + 1, dtype=a.t.dtype, device="cuda")
        return DArray(t[1:], a.shape)
    o = alloc_elemental_outputs(P.master, P.app, P.mesh.dgnodes.shape[-1])
    o = ElementalOutputs(shifted(o.AE), shifted(o.FE), shifted(o.DUDG), shifted(o.DUDG_DUH), o.status)
    assert o.AE.ptr % 16 == 8
    _check(oracle, P, hdg_elemental(P.master, P.app, P.mesh.dgnodes, P.mesh.bf, P.UDG, P.UH, P.SH, out=o))
