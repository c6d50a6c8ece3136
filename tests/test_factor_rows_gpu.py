"""Rows of one level of the BILU(0) factorisation do not affect one another: a level of more rows than CTAs
(graphs of four rows, all coupled, each with an order of its own, side by side), some graphs with a singular diagonal
block.  Those rows are reported; the rows of every other graph are the oracle's to 1e-12 of the largest entry,
with status 0."""
from types import SimpleNamespace

import numpy as np
import pytest

from test_factor_gpu import SIZES, _factor


@pytest.mark.gpu
@pytest.mark.parametrize("bs", SIZES)
def test_singular_row_leaves_the_others_alone(oracle, bs):
    r = np.random.default_rng(bs)
    n, copies = 4, 1300                                  # a CTA takes two or three rows of a level
    rows = np.arange(n * copies).reshape(copies, n)
    others = np.array([[j for j in range(n) if j != i] for i in range(n)])
    colind = np.concatenate([rows[:, :, None], rows[:, others]], 2).astype(np.int32) + 1
    mesh = SimpleNamespace(nf=n * copies, cbsr_rowpts=np.arange(0, n * n * copies + 1, n, dtype=np.int64), cbsr_colind=colind.ravel())
    H = np.asfortranarray(r.standard_normal((bs, bs, n * n * copies)) / bs)
    H[np.arange(bs), np.arange(bs), mesh.cbsr_rowpts[:-1, None]] += 4.0
    order = np.argsort(r.random((copies, n)), 1)
    o2u = (rows[:, :1] + order).astype(np.int32).ravel()
    ref, rc = oracle.bilu0(mesh, H, o2u, np.argsort(o2u).astype(np.int32))
    assert rc == 0
    bad = np.arange(0, copies, 40)
    first = n * bad + order[bad, 0]
    H[:, :, mesh.cbsr_rowpts[first]] = 0.0
    M, st = _factor(mesh, H, o2u)
    good = np.setdiff1d(np.arange(copies), bad)
    assert (st[first] == 1).all() and not st.reshape(copies, n)[good].any()
    keep = (n * n * good[:, None] + np.arange(n * n)).ravel()
    assert np.abs(M[..., keep] - ref[..., keep]).max() / np.abs(ref).max() < 1e-12
