"""hdgx_schur_uq at the compiled element shapes and beside them.

Reference: the oracle's schur_uq on the oracle's own blocks of a mid-Newton state; AE, FE, DUDG and
DUDG_DUH within 1e-12 of their largest entry (the bound of the fixture tests; the blocks are the
inputs, so DUDG is no more sensitive than the rest).  An odd number of elements, outputs only 8-byte
aligned, blocks whose local matrix needs pivoting (two block rows exchanged), and sizes without a
compiled shape (a face node left out)."""
import numpy as np
import pytest

from test_element_mma_gpu import _state

SHAPES = [(2, 1), (2, 2), (2, 3), (2, 4), (3, 1), (3, 2)]
KEYS = ("M", "C", "E", "BD", "F", "GK", "H", "Rq", "Ru", "Rh")


def _blocks(oracle, nd, p, visc):
    P = _state(nd, p, visc)
    return oracle.hdg_elemental(P.master, P.app, P.mesh.dgnodes, P.mesh.bf, P.UDG, P.UH, P.SH, intermediates=True)


def _check(oracle, nd, blk, shift=False):
    import torch
    from hdg_b200 import elemental as E
    empty = E.DArray.empty

    def odd(shape, dtype=torch.float64, device="cuda"):
        a = empty(shape, dtype, device)
        return E.DArray(torch.empty(a.t.numel() + 1, dtype=dtype, device=device)[1:], a.shape)
    if shift:
        E.DArray.empty = staticmethod(odd)
    try:
        out = E.schur_uq(*[blk[k] for k in KEYS])
    finally:
        E.DArray.empty = staticmethod(empty)
    ref = oracle.schur_uq(nd, blk)
    assert ref["nbad"] == 0 and int(out[4].numpy().max()) == 0
    for k, v in zip(("DUDG", "DUDG_DUH", "AE", "FE"), out):
        err = float(np.abs(v.numpy() - ref[k]).max() / np.abs(ref[k]).max())
        assert err < 1e-12, f"{k} {err:.2e}"


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", SHAPES)
@pytest.mark.parametrize("visc,shift", [(False, False), (True, False), (True, True)])
def test_shapes_match_oracle(oracle, nd, p, visc, shift):
    _check(oracle, nd, _blocks(oracle, nd, p, visc), shift)


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", SHAPES)
def test_local_matrix_that_needs_pivoting(oracle, nd, p):
    """The u equations of two nodes exchanged: the same solution, zero or foreign pivots without pivoting."""
    blk = _blocks(oracle, nd, p, True)
    swap = np.arange(blk["Ru"].shape[0])
    swap[[0, -1]] = swap[[-1, 0]]
    for k in ("BD", "F", "Ru"):
        blk[k] = np.asfortranarray(blk[k][swap])
    blk["BD"][0, :, 0, :blk["Ru"].shape[1]] = 0.0          # and no diagonal block at the first node
    _check(oracle, nd, blk)


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", [(2, 2), (3, 1)])
def test_other_sizes_match_oracle(oracle, nd, p):
    blk = _blocks(oracle, nd, p, True)
    n = blk["E"].shape[1] - 1
    cut = {"E": (slice(None), slice(n)), "F": (Ellipsis, slice(n), slice(None)), "GK": (slice(None), slice(n)),
           "H": (slice(None), slice(n), slice(None), slice(n)), "Rh": (slice(None), slice(n))}
    for k, at in cut.items():
        blk[k] = np.asfortranarray(blk[k][at])
    _check(oracle, nd, blk)
