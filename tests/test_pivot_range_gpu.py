"""The pivoted elimination that the unpivoted ones fall back to, on entries that no single-precision number
holds: block systems scaled by powers of two, to the sizes at which the 2 x 2 determinants of the unpivoted
elimination are no normal numbers.

Reference: the oracle on the same blocks; 1e-12 of the largest entry, as tests/test_factor_gpu.py and
tests/test_schur_mma_gpu.py (a power of two changes no rounding)."""
import numpy as np
import pytest

from test_factor_gpu import SIZES, _factor, _system
from test_schur_mma_gpu import SHAPES, _blocks, _check


@pytest.mark.gpu
@pytest.mark.parametrize("bs", SIZES)
@pytest.mark.parametrize("k", [-800, -520, -150, 150, 520, 800])
def test_factorisation(oracle, bs, k):
    mesh, H, o2u = _system("complete", 3, bs)
    first = int(mesh.cbsr_rowpts[int(o2u[0])])
    H[:, :, first] = H[::-1, :, first]                   # one that needs pivoting
    H = np.asfortranarray(np.ldexp(H, k))
    ref, rc = oracle.bilu0(mesh, H, o2u, np.argsort(o2u).astype(np.int32))
    assert rc == 0
    M, st = _factor(mesh, H, o2u)
    assert not st.any()
    diag = np.zeros(M.shape[-1], bool)
    diag[mesh.cbsr_rowpts[:-1]] = True
    pos = np.argsort(o2u)
    row = np.repeat(np.arange(mesh.nf), np.diff(mesh.cbsr_rowpts))
    lower = ~diag & (pos[mesh.cbsr_colind - 1] < pos[row])
    for part in (diag, lower, ~diag & ~lower):           # of the order of 2^-k, 1 and 2^k
        assert np.abs(M[..., part] - ref[..., part]).max() / np.abs(ref[..., part]).max() < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", SHAPES)
@pytest.mark.parametrize("k", [-520, 520])
def test_schur_uq(oracle, nd, p, k):
    blk = _blocks(oracle, nd, p, True)
    for name in ("BD", "F", "Ru"):                       # the u equations
        blk[name] = np.asfortranarray(np.ldexp(blk[name], k))
    _check(oracle, nd, blk)


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", SHAPES)
@pytest.mark.parametrize("k", [-520, 480])
def test_schur_uq_mass(oracle, nd, p, k):
    blk = _blocks(oracle, nd, p, True)
    for name in ("M", "C", "E", "Rq"):                   # the q equations
        blk[name] = np.asfortranarray(np.ldexp(blk[name], k))
    _check(oracle, nd, blk)
