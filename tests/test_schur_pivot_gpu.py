"""hdgx_schur_uq on a caller's blocks whose local matrix or mass matrix needs pivoting where the residual column, or
the first column of C, does not show it: the 2 x 2 blocks of some nodes' momenta are nearly singular (not exactly),
and Ru and Rq are zero (only AE and DUDG_DUH are wanted), or the residual does not reach them.

Reference: the oracle's schur_uq (partial pivoting); 1e-12 of the largest entry, as tests/test_schur_mma_gpu.py."""
import numpy as np
import pytest

from test_schur_mma_gpu import KEYS, SHAPES, _blocks


def _swapped(n, pairs, eps, rng):
    """n x n, condition number below 100: the rows of each pair exchanged with their partners', the pair's own block eps."""
    A = 4 * np.eye(n) + 0.5 * rng.standard_normal((n, n)) / np.sqrt(n)
    for (i, j), (k, l) in pairs:
        A[[i, j, k, l]] = A[[k, l, i, j]]
        A[np.ix_([i, j], [i, j])] = eps * np.array([[1.0, 0.5], [0.3, 1.0]])
    return A


def _run(oracle, nd, blk, zero_residual):
    from hdg_b200 import elemental as E
    blk = {k: np.asfortranarray(blk[k]) for k in KEYS}
    out = E.schur_uq(*[blk[k] for k in KEYS])
    ref = oracle.schur_uq(nd, blk)
    assert ref["nbad"] == 0 and int(out[4].numpy().max()) == 0
    for k, v in zip(("DUDG", "DUDG_DUH", "AE", "FE"), out):
        scale = np.abs(ref[k]).max()
        if zero_residual and k in ("DUDG", "FE"):        # exactly zero, and Rh
            scale = 1.0
        err = float(np.abs(v.numpy() - ref[k]).max() / scale)
        assert err < 1e-12, f"{k} {err:.2e}"


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", SHAPES)
@pytest.mark.parametrize("eps", [1e-6, 1e-10, 1e-13])
@pytest.mark.parametrize("residual", ["zero", "elsewhere"])
def test_local_matrix(oracle, nd, p, eps, residual):
    blk = _blocks(oracle, nd, p, True)
    rng = np.random.default_rng(nd + p)
    npv, ncu, _ = blk["Ru"].shape
    ne = blk["Ru"].shape[-1]
    # B = 0: the local matrix is D itself.  The momenta of two nodes against their density and energy
    blk["BD"] = np.zeros_like(blk["BD"])
    for e in range(ne):
        pairs = [((r + npv, r + 2 * npv), (r, r + (ncu - 1) * npv)) for r in (e % npv, (e + 2) % npv)]
        A = _swapped(npv * ncu, pairs, eps, rng)
        if residual == "elsewhere":                      # an equation of its own, all that the residual reaches
            r = (e + 1) % npv
            A[r, :] = A[:, r] = 0.0
            A[r, r] = 3.0
        blk["BD"][:, :, :, :ncu, e] = A.reshape((npv, ncu, npv, ncu), order="F")
    blk["Rq"] = np.zeros_like(blk["Rq"])
    Ru = np.zeros_like(blk["Ru"])
    if residual == "elsewhere":
        Ru[(np.arange(ne) + 1) % npv, 0, np.arange(ne)] = 1.0
    blk["Ru"] = Ru
    _run(oracle, nd, blk, residual == "zero")


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", [s for s in SHAPES if s != (2, 1)])      # three nodes have no two pairs
@pytest.mark.parametrize("eps", [1e-6, 1e-10, 1e-13])
def test_mass_matrix(oracle, nd, p, eps):
    blk = _blocks(oracle, nd, p, True)
    rng = np.random.default_rng(nd + p)
    npv, _, ne = blk["M"].shape
    scale = np.abs(blk["M"]).max()
    blk["M"] = scale * np.stack([_swapped(npv, [((0, 1), (2, 3))], eps, rng) for _ in range(ne)], -1)
    blk["C"][:, 0, 0] = 0.0                              # the first column says nothing
    _run(oracle, nd, blk, False)
