"""Diagonal blocks of the BILU(0) factorisation that an elimination without pivoting gets wrong and the first
column of the inverse does not show: two neighbouring unknowns whose 2 x 2 block is nearly singular, coupled
to two others, at every place of the block, the rest of it the identity or a part that couples to them.

Reference: numpy's inverse (partial pivoting).  1e-12 of the largest entry, the bound of the other factor
tests; the condition numbers are 5 to 400.  One row a block, no neighbours, all in one launch."""
from types import SimpleNamespace

import numpy as np
import pytest

from test_factor_gpu import SIZES, _factor


def _blocks(bs):
    """All blocks [bs, bs, n] of a size: pair (i, i + 1) nearly singular, its partner the pair (j, j + 1)."""
    r = np.random.default_rng(bs)
    out = []
    for i in range(0, bs - 3, 2):
        for j in {i + 2, bs - 2 - bs % 2}:
            if j <= i + 1:
                continue
            for eps in (1e-6, 1e-10, 1e-13):
                for coupled in (False, True):
                    A = np.eye(bs)
                    if coupled:
                        A += r.standard_normal((bs, bs)) / (3 * bs)
                    A[np.ix_([i, i + 1], [i, i + 1])] = [[1.0, 1.0], [1.0, 1.0 + eps]]
                    A[np.ix_([i, i + 1], [j, j + 1])] = [[1.0, 0.3], [-0.2, 1.1]]
                    A[np.ix_([j, j + 1], [i, i + 1])] = [[0.9, -0.4], [0.5, 1.2]]
                    if not coupled or i == 0:
                        out.append(A)
                        continue
                    A[i:, :i] = 0.0                      # block upper triangular: the first columns see nothing
                    out.append(A)
    return np.asfortranarray(np.stack(out, -1))


@pytest.mark.gpu
@pytest.mark.parametrize("bs", SIZES)
def test_nearly_singular_pairs(bs):
    H = _blocks(bs)
    n = H.shape[-1]
    mesh = SimpleNamespace(nf=n, cbsr_rowpts=np.arange(n + 1, dtype=np.int64), cbsr_colind=np.arange(1, n + 1, dtype=np.int32))
    M, st = _factor(mesh, H, np.arange(n, dtype=np.int32))
    assert not st.any()
    for k in range(n):
        assert np.linalg.cond(H[..., k]) < 1e3
        ref = np.linalg.inv(H[..., k])
        assert np.abs(M[..., k] - ref).max() / np.abs(ref).max() < 1e-12, k
