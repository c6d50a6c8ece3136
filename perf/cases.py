"""The work this framework is used for, as cases that can be timed and compared.

Sizes are those of the configurations (``hdg_b200.configs``), of the serving mix
(``hdg_b200.serve.request_mix``: degree 1 to 4, inviscid or Navier--Stokes with Re 200 to 2000,
Mach 0.3 to 0.8) and of the benchmark's tetrahedral samples.  ``n`` is the number of squares
(two triangles each) or cubes (six tetrahedra each) per side.  Kinds:

* ``elemental``  ``hdg_elemental`` on resident arrays: the assembly of one Newton step;
* ``residual``   ``residual``: the element residual alone, q recovered from the trace;
* ``schur_uq``   ``schur_uq``: the local Schur complement of blocks that a caller assembled;
* ``linear``     ``HDGSolver.linear_solve``: BILU(0) factors and GMRES on the condensed system;
* ``newton``     ``hdgx_solve``: a whole Newton solve from host arrays, as a serving request.

The first three take a state in mid-Newton (a smooth field, its gradient, a trace 1 % off it);
the last two start where a solve starts (freestream with a 1 % smooth perturbation, q = 0).
"""
import itertools
import math

import numpy as np
import torch

from hdg_b200.app import freestream, init_udg, inituhat, make_app, state_fourier
from hdg_b200.configs import Problem
from hdg_b200.elemental import DArray, DeviceMaster, alloc_elemental_outputs, hdg_elemental, residual, schur_uq
from hdg_b200.master import mkmaster
from hdg_b200.mesh import mkmesh_cube, mkmesh_square
from hdg_b200.perfmodel import element_counts
from hdg_b200.solve import HDGSolver, hdgx_solve

GAM = 1.4


def _case(kind, nd, p, visc, n, name=None, **more):
    c = dict(kind=kind, nd=nd, p=p, visc=visc, n=n, **more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest workload: 512 triangles, one launch, less than one wave of the GPU
        _case("elemental", 2, 2, False, 16, "tri_p2_euler"),
        # low degree, as the lowest-degree bucket of the mixed-degree workload (13,122 elements)
        _case("elemental", 2, 1, False, 81, "tri_p1_euler"),
        # the headline workload: 32,768 triangles, Navier-Stokes, p = 3
        _case("elemental", 2, 3, True, 128, "tri_p3_ns"),
        # the highest 2D degree at a middle size of the serving range (6,498 elements)
        _case("elemental", 2, 4, True, 57, "tri_p4_ns"),
        # tetrahedra, 24,576 elements: the benchmark's 3D sample
        _case("elemental", 3, 2, False, 16, "tet_p2_euler"),
        # the largest element: p = 3 tetrahedra, Navier-Stokes, 3,072 elements
        _case("elemental", 3, 3, True, 8, "tet_p3_ns"),
        # residual-only evaluation (explicit stepping, line search of a matrix-free caller)
        _case("residual", 2, 3, True, 65, "residual_tri_p3"),
        # drop-in for the MEX Schur complement on a caller's blocks (4,050 elements)
        _case("schur_uq", 2, 3, True, 45, "schur_tri_p3"),
        # the linear system of a Newton step: 12,416 faces of 16 unknowns
        _case("linear", 2, 3, True, 64, "linear_tri_p3_ns"),
        # the same in 3D: 6,528 faces of 30 unknowns
        _case("linear", 3, 2, False, 8, "linear_tet_p2_euler"),
        # one serving request, start to end, from and to host memory
        _case("newton", 2, 2, False, 16, "newton_tri_p2", mixed=False),
        # the same with FP32 factors and elimination behind the FP64 residual
        _case("newton", 2, 3, True, 24, "newton_tri_p3_mixed", mixed=True),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["elemental"] * 6 + ["residual", "schur_uq", "linear", "newton"])
    visc = rng.random() < 0.5
    if kind == "newton":
        return _case(kind, 2, rng.randint(1, 4), visc, _spread(rng, 8, 24), mixed=rng.random() < 0.25)
    if kind == "linear":
        if rng.random() < 0.3:
            return _case(kind, 3, rng.choice([1, 2]), False, _spread(rng, 3, 8))
        return _case(kind, 2, rng.randint(1, 3), visc, _spread(rng, 8, 60))
    if kind == "schur_uq":
        return _case(kind, 2, rng.randint(1, 4), visc, _spread(rng, 4, 45))
    if rng.random() < 0.65:
        p = rng.randint(1, 4)
        c = _case(kind, 2, p, visc, _spread(rng, 4, {1: 181, 2: 150, 3: 128, 4: 81}[p]))
    else:
        p = rng.choice([1, 2, 2, 3])
        c = _case(kind, 3, p, visc, _spread(rng, 2, {1: 20, 2: 16, 3: 8}[p]))
    if kind == "elemental" and rng.random() < 0.2:
        c["tdep"] = True                     # the stage systems of the implicit time integrators
    return c


# ------------------------------------------------------------------------------- inputs
def _grid(nd, p, n, gen):
    """dg [ne, nd, npv] (straight-sided elements of a jittered unit grid) and bf [ne, nfe]."""
    m = mkmaster(nd, p, 2 * p)
    dev = "cuda"
    ax = torch.arange(n + 1, dtype=torch.float64, device=dev) / n
    X = torch.stack(torch.meshgrid(*[ax] * nd, indexing="ij"), -1)                 # vertices
    inner = ((X > 1e-9) & (X < 1 - 1e-9)).to(X.dtype)
    Y = X + inner * (0.15 / n) * (2 * torch.rand(X.shape, generator=gen, dtype=X.dtype, device=dev) - 1)
    if nd == 2:
        simplices = [[(0, 0), (1, 0), (0, 1)], [(1, 1), (0, 1), (1, 0)]]
    else:
        simplices = []
        for axes in itertools.permutations(range(3)):
            v = [(0, 0, 0)]
            for a in axes:
                v.append(tuple(x + (i == a) for i, x in enumerate(v[-1])))
            if np.linalg.det(np.array(v[1:], float) - np.array(v[0], float)) < 0:
                v[1], v[2] = v[2], v[1]
            simplices.append(v)

    def corners(V):                                      # [cells, simplices, nd + 1, nd]
        cut = [torch.stack([V[tuple(slice(o, n + o) for o in v)].reshape(-1, nd) for v in s], 1) for s in simplices]
        return torch.stack(cut, 1).reshape(-1, nd + 1, nd)

    loc = torch.tensor(m.plocvl, dtype=torch.float64, device=dev)
    lam = torch.cat([1 - loc.sum(1, keepdim=True), loc], 1)                        # barycentric coordinates
    dg = torch.einsum("kv,evd->edk", lam, corners(Y)).contiguous()
    flat = torch.einsum("kv,evd->ekd", lam, corners(X))
    ne, nfe = dg.shape[0], nd + 1
    bf = torch.ones(ne, nfe, dtype=torch.int32, device=dev)
    for j in range(nfe):
        x = flat[:, torch.tensor(m.perm[:, j] - 1, device=dev)]                    # [ne, npf, nd]
        for side, (d, at) in enumerate(itertools.product(range(nd), (0.0, 1.0))):
            bf[(x[:, :, d] - at).abs().amax(1) < 1e-9, j] = -(side + 1)
    return m, dg, bf


def _field(x, base, amp, gen, modes=6):
    """base (1 + amp sum of modes) at x [..., nd]: values [..., ncu] and gradients [..., ncu, nd]."""
    nd, ncu = x.shape[-1], base.numel()
    dev = x.device
    k = 2 * math.pi * torch.randint(1, 4, (modes, nd), generator=gen, device=dev).to(x.dtype)
    ph = 2 * math.pi * torch.rand(modes, ncu, generator=gen, dtype=x.dtype, device=dev)
    a = torch.randn(modes, ncu, generator=gen, dtype=x.dtype, device=dev) * amp / math.sqrt(modes / 2)
    scale = base.abs().clamp_min(0.5)
    u, g = base.expand(x.shape[:-1] + (ncu,)).clone(), torch.zeros(x.shape[:-1] + (ncu, nd), dtype=x.dtype, device=dev)
    for i in range(modes):
        arg = (x @ k[i])[..., None] + ph[i]
        u += scale * a[i] * torch.sin(arg)
        g += (scale * a[i] * torch.cos(arg))[..., None] * k[i]
    return u, g


def _elements(case, seed):
    nd, p, n, visc, tdep = case["nd"], case["p"], case["n"], case["visc"], bool(case.get("tdep"))
    gen = torch.Generator("cuda").manual_seed(seed)
    r = np.random.default_rng(seed)
    m, dg, bf = _grid(nd, p, n, gen)
    app = make_app(nd, gam=GAM, re=float(r.uniform(200, 2000)) if visc else np.inf, minf=float(r.uniform(0.3, 0.8)))
    if tdep:
        app.tdep, app.fc_u = 1, float(r.uniform(10, 100))
    base = torch.tensor(freestream(nd, GAM, app.param[4]), device="cuda")
    x = dg.transpose(1, 2)
    u, g = _field(x, base, 0.04, gen)
    udg = torch.cat([u, -g.transpose(-1, -2).flatten(-2)], -1).transpose(1, 2).contiguous()   # [ne, nc, npv]
    nodes = torch.tensor(m.perm.T.reshape(-1) - 1, device="cuda")
    off, _ = _field(x[:, nodes], torch.zeros_like(base), 0.01, gen)
    uh = (u[:, nodes] + off).contiguous()                                                  # [ne, ndf, ncu]
    sh = torch.zeros_like(udg)
    if tdep:
        sh[:, :app.ncu] = app.fc_u * (udg[:, :app.ncu] * (1 + 0.001 * torch.rand(
            udg[:, :app.ncu].shape, generator=gen, dtype=udg.dtype, device="cuda")))
    return m, app, dg, bf, udg, uh, sh


def _dev(t):
    return DArray(t.reshape(-1), tuple(reversed(t.shape)))


def _problem(case, seed):
    nd, p, n = case["nd"], case["p"], case["n"]
    r = np.random.default_rng(seed)
    minf, re = float(r.uniform(0.3, 0.8)), float(r.uniform(200, 2000)) if case["visc"] else np.inf
    mesh = mkmesh_square(n + 1, n + 1, p) if nd == 2 else mkmesh_cube(n + 1, n + 1, n + 1, p)
    master, app = mkmaster(nd, p, 2 * p), make_app(nd, gam=GAM, re=re, minf=minf)
    u = state_fourier(mesh.dgnodes, nd, GAM, minf, seed, 4, 0.01, "velocity")
    udg = init_udg(u, app.nc)
    return Problem("case", master, mesh, app, udg, inituhat(master.perm, mesh.elcon, udg, app.ncu, mesh.nsiz),
                   np.zeros_like(udg))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "newton":
        return dict(case=case, P=_problem(case, seed))
    if kind == "linear":
        P = _problem(case, seed)
        s = HDGSolver(P.master, P.mesh, P.app)
        s.assemble(DArray.from_numpy(P.UDG), DArray.from_numpy(P.UH), DArray.from_numpy(P.SH))
        return dict(case=case, solver=s)
    m, app, dg, bf, udg, uh, sh = _elements(case, seed)
    if kind == "schur_uq":
        # a caller's blocks, column-major with the element index last
        blocks = {}
        for part in _chunks(m, app, dg, bf, udg, uh, sh):
            for k, v in part.items():
                blocks.setdefault(k, []).append(v.permute(0, *range(v.dim() - 1, 0, -1)).contiguous())
        return dict(case=case, blocks=[_dev(torch.cat(blocks[k])) for k in
                                       ("M", "C", "E", "BD", "F", "GK", "H", "Rq", "Ru", "Rh")])
    return dict(case=case, master=m, app=app, dm=DeviceMaster(m), dg=_dev(dg), bf=_dev(bf), udg=_dev(udg), uh=_dev(uh),
                sh=_dev(sh), out=alloc_elemental_outputs(m, app, dg.shape[0]) if kind == "elemental" else None)


# ------------------------------------------------------------------------------- the pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "elemental":
        o = hdg_elemental(s["master"], s["app"], s["dg"], s["bf"], s["udg"], s["uh"], s["sh"], out=s["out"],
                          dmaster=s["dm"])
        return dict(AE=o.AE.t, FE=o.FE.t, DUDG=o.DUDG.t, DUDG_DUH=o.DUDG_DUH.t, status=o.status.t)
    if kind == "residual":
        ru, st = residual(s["master"], s["app"], s["dg"], s["bf"], s["udg"], s["uh"], s["sh"], dmaster=s["dm"])
        return dict(RU=ru.t, status=st.t)
    if kind == "schur_uq":
        dudg, dd, ae, fe, st = schur_uq(*s["blocks"])
        return dict(AE=ae.t, FE=fe.t, DUDG=dudg.t, DUDG_DUH=dd.t, status=st.t)
    if kind == "linear":
        s["solver"].linear_solve()
        return dict(factors=s["solver"].Mg.t, x=s["solver"].DUH.t)
    P = s["P"]
    U, H, _ = hdgx_solve(P.master, P.mesh, P.app, P.UDG, P.UH, P.SH, mixed=s["case"]["mixed"])
    return dict(UDG=U, UH=H)


def work(case):
    nd, p, n = case["nd"], case["p"], case["n"]
    m = mkmaster(nd, p, 2 * p)
    ncu, ndf = nd + 2, m.npf * m.nfe
    nc, nh, nu = ncu * (nd + 1), ncu * ndf, m.npv * ncu
    ne = 2 * n ** 2 if nd == 2 else 6 * n ** 3
    w = element_counts(nd, m.npv, m.npf, m.ngv, m.ngf)
    if case["kind"] == "elemental":
        return dict(bytes=ne * w["bytes"], flops=ne * w["flops"])
    if case["kind"] == "residual":
        return dict(bytes=ne * (w["bytes_in"] + 8 * nu), flops=ne * (
            2 * m.npv ** 2 * (nd + 1) * m.ngv + 2 * m.npv * ncu * (nd + 1) * (2 * m.ngv + m.npv) +
            4 * m.npf * m.ngf * m.nfe * ncu * (nd + 1)))
    if case["kind"] == "schur_uq":
        into = (m.npv ** 2 * (1 + nd) + m.npv * ndf * nd + nu * m.npv * nc + nu * nh + nh * m.npv * nc + nh * nh +
                nu * nd + nu + nh)
        return dict(bytes=ne * (8 * into + w["bytes_out"]), flops=ne * w["schur_flops"])
    nf = 3 * n * n + 2 * n if nd == 2 else 12 * n ** 3 + 6 * n * n
    bs = ncu * m.npf
    nnzb = nf + ne * m.nfe * nd                       # the diagonal, and each element's face pairs
    # the system read once, the factors and the solution written once; the factorisation's products
    sys_ = dict(bytes=8 * (2 * nnzb * bs * bs + 2 * nf * bs), flops=2 * bs ** 3 * (nf + 2 * ne * m.nfe))
    if case["kind"] == "linear":
        return sys_
    return dict(bytes=sys_["bytes"] + ne * w["bytes"], flops=sys_["flops"] + ne * w["flops"])


# ------------------------------------------------------------------------- the same in 64 bits
def _flux(app, w):
    """The compressible Navier-Stokes flux [..., ncu, nd] of w [..., nc] = (u, q by direction)."""
    nd, ncu = app.nd, app.ncu
    gam, _, re, pr = (float(v) for v in app.param[:4])
    u, q = w[..., :ncu], w[..., ncu:].unflatten(-1, (nd, ncu))
    rho, v = u[..., 0], u[..., 1:-1] / u[..., :1]
    p = (gam - 1) * (u[..., -1] - 0.5 * (v * u[..., 1:-1]).sum(-1))
    eye = torch.eye(nd, dtype=w.dtype, device=w.device)
    mom = u[..., 1:-1, None] * v[..., None, :] + p[..., None, None] * eye
    en = ((u[..., -1] + p) / rho)[..., None] * u[..., 1:-1]
    if math.isfinite(re):
        qr = q[..., :, 0]
        gv = (q[..., :, 1:-1].transpose(-1, -2) - v[..., :, None] * qr[..., None, :]) / rho[..., None, None]
        tau = (gv + gv.transpose(-1, -2) - 2 / 3 * torch.diagonal(gv, dim1=-2, dim2=-1).sum(-1)[..., None, None] * eye) / re
        px = (gam - 1) * (q[..., :, -1] - 0.5 * (v * v).sum(-1, keepdim=True) * qr -
                          rho[..., None] * (v[..., :, None] * gv).sum(-2))
        T = (px * rho[..., None] - p[..., None] * qr) / (rho * rho)[..., None]
        mom = mom + tau
        en = en + (v[..., :, None] * tau).sum(-2) + gam / (re * pr * (gam - 1)) * T
    return torch.cat([u[..., None, 1:-1], mom, en[..., None, :]], -2)


def _with_jacobian(f, w):
    """f(w) and its derivatives by the last axis of w, as a last axis."""
    cols, val = [], None
    for c in range(w.shape[-1]):
        t = torch.zeros_like(w)
        t[..., c] = 1.0
        val, d = torch.func.jvp(f, (w,), (t,))
        cols.append(d)
    return val, torch.stack(cols, -1)


def _blocks(m, app, dg, bf, udg, uh, sh, jacobian=True):
    """The element blocks of the HDG discretisation (volume and face integrals) of some elements."""
    nd, ncu = app.nd, app.ncu
    T = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dg.device)  # noqa: E731
    vt, vg, mv, ft, fg, mf = (T(getattr(m, k)) for k in ("shapvt", "shapvg", "shapmv", "shapft", "shapfg", "shapmf"))
    ngf, npf, nfe, npv = m.ngf, m.npf, m.nfe, m.npv
    ngt, ndf = ngf * nfe, npf * nfe
    perm = m.perm - 1
    FT, FG, TT, TG = (torch.zeros(s, dtype=dg.dtype, device=dg.device) for s in ((ngt, npv), (npv, ngt), (ngt, ndf), (ndf, ngt)))
    for j in range(nfe):
        g = slice(j * ngf, (j + 1) * ngf)
        at = torch.tensor(perm[:, j], device=dg.device)
        FT[g, at], FG[at, g] = ft[:, :, 0], fg[:, :, 0]
        TT[g, j * npf:(j + 1) * npf], TG[j * npf:(j + 1) * npf, g] = ft[:, :, 0], fg[:, :, 0]
    E = torch.einsum
    J = E("gnk,emn->egkm", mv[:, :, 1:], dg)
    jac = torch.linalg.det(J)
    X = torch.linalg.inv(J) * jac[..., None, None]                                  # adjugate
    xf = dg[:, :, torch.tensor(perm.T.reshape(-1), device=dg.device)].unflatten(-1, (nfe, npf))
    D = E("gnk,emjn->ejgmk", mf[:, :, 1:], xf).flatten(1, 2)                        # [e, gg, nd, nd - 1]
    nv = torch.stack([D[:, :, 1, 0], -D[:, :, 0, 0]], -1) if nd == 2 else torch.linalg.cross(D[..., 0], D[..., 1])
    fj = nv.norm(dim=-1)
    nl = nv / fj[..., None]
    u = udg.transpose(1, 2)                                                          # [e, node, component]
    B = dict(M=app.fc_q * E("rg,gs,eg->ers", vg[:, :, 0], vt[:, :, 0], jac),
             C=E("rgj,egij,gs->ersi", vg[:, :, 1:], X, vt[:, :, 0]),
             E=E("rg,gf,egd->erfd", FG, TT, nv))
    qs = u[..., ncu:].unflatten(-1, (nd, ncu))
    shq = sh.transpose(1, 2)[..., ncu:].unflatten(-1, (nd, ncu)) / app.fc_q
    no_q = E("ersd,esa->erad", B["C"], u[..., :ncu]) - E("erfd,efa->erad", B["E"], uh) + E("ers,esda->erad", B["M"], shq)
    if not jacobian:                                       # the residual alone: q solves its equation
        q = torch.linalg.solve(B["M"], no_q.flatten(2)).unflatten(-1, (ncu, nd))
        u = torch.cat([u[..., :ncu], q.transpose(-1, -2).flatten(-2)], -1)
    else:
        B["Rq"] = no_q - E("ers,esda->erad", B["M"], qs)
    ug, fu, fh = E("gn,enc->egc", vt[:, :, 0], u), E("gn,enc->egc", FT, u), E("gf,efa->ega", TT, uh)
    tau = float(app.param[5])
    wf = torch.cat([fh, fu[..., ncu:]], -1)
    normal = lambda f: E("ega...,eg->ega...", f, fj)  # noqa: E731
    f = _flux(app, ug)
    w = E("egaj,egji->egai", f, X)
    fhat = E("egaj,egj->ega", _flux(app, wf), nl) + tau * (fu[..., :ncu] - fh)
    B["Ru"] = E("rgi,egai->era", vg[:, :, 1:], w) - E("rg,ega->era", FG, normal(fhat))
    if app.tdep:
        st = E("gn,ean->ega", vt[:, :, 0], sh[:, :ncu])
        B["Ru"] = B["Ru"] + E("rg,ega,eg->era", vg[:, :, 0], st - app.fc_u * ug[..., :ncu], jac)
    if not jacobian:
        return B
    _, fc = _with_jacobian(lambda x: _flux(app, x), ug)
    fc = E("egajc,egji->egaic", fc, X)
    B["BD"] = -E("ergac,gs->erasc", E("rgi,egaic->ergac", vg[:, :, 1:], fc), vt[:, :, 0])
    if app.tdep:
        mu = app.fc_u * E("rg,gs,eg->ers", vg[:, :, 0], vt[:, :, 0], jac)
        for a in range(ncu):
            B["BD"][:, :, a, :, a] += mu
    _, hc = _with_jacobian(lambda x: _flux(app, x), wf)
    hc = E("egajc,egj->egac", hc, nl)
    eye = tau * torch.eye(ncu, dtype=dg.dtype, device=dg.device)
    hu = torch.cat([eye.expand(hc[..., :ncu].shape), hc[..., ncu:]], -1)             # by (u, q)
    hh = hc[..., :ncu] - eye                                                         # by the trace
    # Dirichlet faces: the boundary flux is the trace less the boundary state
    edge = (bf < 0).repeat_interleave(ngf, 1)
    state = torch.tensor(np.asarray(app.bcs), dtype=dg.dtype, device=dg.device)[(-bf.long() - 1).clamp_min(0)]
    bh = torch.where(edge[..., None], fh - state.repeat_interleave(ngf, 1), fhat)
    bu = torch.where(edge[..., None, None], torch.zeros_like(hu), hu)
    bb = torch.where(edge[..., None, None], eye / tau, hh)
    B["BD"] += E("rg,gs,egac->erasc", FG, FT, normal(hu))
    B["F"] = E("rg,gf,egab->erabf", FG, TT, normal(hh))
    B["GK"] = E("fg,gs,egac->eafsc", TG, FT, normal(bu))
    B["H"] = E("fg,gh,egab->eafbh", TG, TT, normal(bb))
    B["Rh"] = -E("fg,ega->eaf", TG, normal(bh))
    return B


def _chunks(m, app, dg, bf, udg, uh, sh, jacobian=True):
    step = 512 if app.nd == 3 else 2048
    for e in range(0, dg.shape[0], step):
        part = slice(e, e + step)
        yield _blocks(m, app, dg[part], bf[part], udg[part], uh[part], sh[part], jacobian)


def _schur(B, nd):
    """AE, FE, DUDG, DUDG_DUH of the blocks, in the outputs' layout."""
    E = torch.einsum
    ne, npv, ncu = B["Ru"].shape
    ndf = B["Rh"].shape[2]
    nu, nh = npv * ncu, ncu * ndf
    Mi = torch.linalg.inv(B["M"])
    MiC, MiE, MiR = (E("ers,es...->er...", Mi, B[k]) for k in ("C", "E", "Rq"))
    Bq = B["BD"][..., ncu:].unflatten(-1, (nd, ncu))                                 # [e, r, a, s, d, b]
    SD = B["BD"][..., :ncu] + E("erasdb,eskd->erakb", Bq, MiC)
    rhs0 = B["Ru"] - E("erasdb,esbd->era", Bq, MiR)
    rhs = E("erasdb,esfd->erabf", Bq, MiE) - B["F"]
    A = SD.permute(0, 2, 1, 4, 3).reshape(ne, nu, nu)
    R = torch.cat([rhs0.transpose(1, 2).reshape(ne, nu, 1), rhs.permute(0, 2, 1, 4, 3).reshape(ne, nu, nh)], 2)
    Z = torch.linalg.solve(A, R).reshape(ne, ncu, npv, 1 + nh)
    du, dl = Z[..., 0], Z[..., 1:].unflatten(-1, (ndf, ncu))                         # [e, a, r, f, b]
    dudg = torch.cat([du] + [MiR[..., d].transpose(1, 2) + E("ers,eas->ear", MiC[..., d], du) for d in range(nd)], 1)
    eye = torch.eye(ncu, dtype=du.dtype, device=du.device)
    dd = torch.cat([dl] + [E("ers,easfb->earfb", MiC[..., d], dl) - E("erf,ab->earfb", MiE[..., d], eye)
                           for d in range(nd)], 1)                                   # [e, c, r, f, b]
    fe = B["Rh"] - E("eafsc,ecs->eaf", B["GK"], dudg)
    ae = E("eafsc,ecsgb->eafgb", B["GK"], dd) + B["H"].permute(0, 1, 2, 4, 3)        # [e, a, f, g, b]
    return dict(AE=ae.permute(0, 3, 4, 2, 1).reshape(-1), FE=fe.transpose(1, 2).reshape(-1), DUDG=dudg.reshape(-1),
                DUDG_DUH=dd.permute(0, 3, 4, 1, 2).reshape(-1))


def exact(case, seed):
    if case["kind"] in ("linear", "newton"):     # the end of an iteration, to its tolerance
        return None
    m, app, *arrays = _elements(case, seed)
    if case["kind"] == "residual":
        return dict(RU=torch.cat([b["Ru"].transpose(1, 2).reshape(-1) for b in _chunks(m, app, *arrays, jacobian=False)]),
                    status=None)
    parts = [_schur(b, app.nd) for b in _chunks(m, app, *arrays)]
    return dict({k: torch.cat([q[k] for q in parts]) for k in parts[0]}, status=None)
