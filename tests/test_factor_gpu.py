"""The row kernel of the level-scheduled BILU(0) factorisation at its edges, against the oracle's
computeBILU0 in the same order; 1e-12 of the largest entry, the bound of the other factor tests.
Patterns: chains, stars and complete graphs of up to seven block rows (every pair of neighbours
coupled: up to six updates per elimination, more than the four that are staged together), several
copies side by side so that a level holds many rows, all block sizes; a diagonal block that needs
pivoting; and a singular one, reported in status."""
import ctypes as ct
from types import SimpleNamespace

import numpy as np
import pytest

SIZES = [8, 12, 15, 16, 20, 30]


def _pattern(kind, copies):
    n = 7
    edges = {"chain": [(i, i + 1) for i in range(n - 1)], "star": [(0, i) for i in range(1, n)],
             "complete": [(i, j) for i in range(n) for j in range(i + 1, n)]}[kind]
    adj = [[] for _ in range(n)]
    for i, j in edges:
        adj[i].append(j)
        adj[j].append(i)
    rowpts, colind = [0], []
    for c in range(copies):
        for i in range(n):
            colind += [c * n + i + 1] + [c * n + j + 1 for j in adj[i]]
            rowpts.append(len(colind))
    return SimpleNamespace(nf=n * copies, cbsr_rowpts=np.array(rowpts, dtype=np.int64), cbsr_colind=np.array(colind, dtype=np.int64))


def _factor(mesh, H, o2u):
    import torch
    from hdg_b200._lib import HdgxBsr, check, lib
    from hdg_b200.elemental import DArray
    from hdg_b200.ordering import levels_of_order, sweep_plan
    u2o = np.argsort(o2u).astype(np.int32)
    lv = levels_of_order(mesh.cbsr_rowpts, mesh.cbsr_colind, o2u, u2o)
    plan, maxd = sweep_plan(lv, mesh.cbsr_rowpts, mesh.cbsr_colind)
    keep = [DArray.from_numpy(mesh.cbsr_rowpts, dtype=torch.int64)] + [
        DArray.from_numpy(a, dtype=torch.int32) for a in (mesh.cbsr_colind, lv.color_rows, lv.pos, plan)]
    ptr = np.ascontiguousarray(lv.color_ptr, dtype=np.int32)
    bsr = HdgxBsr(mesh.nf, H.shape[0], len(mesh.cbsr_colind), keep[0].ptr, keep[1].ptr, lv.ncolors, ptr.ctypes.data,
                  keep[2].ptr, keep[3].ptr, None, keep[4].ptr, maxd)
    M, st = DArray.from_numpy(H), DArray.zeros((mesh.nf,), dtype=torch.int32)
    check(lib().hdgx_bilu0_factor(ct.byref(bsr), M.ptr, st.ptr, None), "hdgx_bilu0_factor")
    torch.cuda.synchronize()
    return M.numpy(), st.numpy()


def _system(kind, copies, bs):
    r = np.random.default_rng(bs)
    mesh = _pattern(kind, copies)
    H = np.asfortranarray(r.standard_normal((bs, bs, len(mesh.cbsr_colind))) / bs)
    diag = mesh.cbsr_rowpts[:-1]
    H[np.arange(bs), np.arange(bs), diag[:, None]] += 4.0
    return mesh, H, r.permutation(mesh.nf).astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("bs", SIZES)
@pytest.mark.parametrize("kind,copies", [("chain", 1), ("star", 3), ("complete", 1), ("complete", 120)])
def test_factors_match_oracle(oracle, kind, copies, bs):
    mesh, H, o2u = _system(kind, copies, bs)
    ref, rc = oracle.bilu0(mesh, H, o2u, np.argsort(o2u).astype(np.int32))
    assert rc == 0
    M, st = _factor(mesh, H, o2u)
    assert not st.any()
    assert np.abs(M - ref).max() / np.abs(ref).max() < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("bs", SIZES)
def test_pivoted_and_singular_diagonal_blocks(oracle, bs):
    mesh, H, o2u = _system("chain", 4, bs)
    first, last = int(o2u[0]), int(o2u[1])
    k = int(mesh.cbsr_rowpts[first])
    H[:, :, k] = H[::-1, :, k]                           # no pivots on the diagonal
    ref, rc = oracle.bilu0(mesh, H, o2u, np.argsort(o2u).astype(np.int32))
    assert rc == 0
    M, st = _factor(mesh, H, o2u)
    assert not st.any() and np.abs(M - ref).max() / np.abs(ref).max() < 1e-12
    H[:, :, int(mesh.cbsr_rowpts[last])] = 0.0
    mesh1 = SimpleNamespace(nf=1, cbsr_rowpts=np.array([0, 1]), cbsr_colind=np.array([1]))
    _, st = _factor(mesh1, np.zeros((bs, bs, 1), order="F"), np.array([0], dtype=np.int32))
    assert st[0] == 1
