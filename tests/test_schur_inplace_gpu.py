"""hdgx_schur_uq with AE written over H (as the general kernel allows), with and without an elimination that is
repeated with pivoting; bounds of test_schur_mma_gpu.py."""
import numpy as np
import pytest

from test_schur_mma_gpu import KEYS, SHAPES, _blocks


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p", SHAPES)
@pytest.mark.parametrize("pivoted", [False, True])
def test_trace_jacobian_over_h(oracle, nd, p, pivoted):
    import torch
    from hdg_b200._lib import check, lib
    from hdg_b200.elemental import DArray
    blk = _blocks(oracle, nd, p, True)
    if pivoted:
        swap = np.arange(blk["Ru"].shape[0])
        swap[[0, -1]] = swap[[-1, 0]]
        for k in ("BD", "F", "Ru"):
            blk[k] = np.asfortranarray(blk[k][swap])
        blk["BD"][0, :, 0, :blk["Ru"].shape[1]] = 0.0
    npv, ncu, _, nc, ne = blk["BD"].shape
    ndf = blk["E"].shape[1]
    d = {k: DArray.from_numpy(np.asfortranarray(blk[k])) for k in KEYS}
    DUDG, DD, FE = DArray.empty((npv, nc, ne)), DArray.empty((npv, nc, ncu, ndf, ne)), DArray.empty((ncu, ndf, ne))
    check(lib().hdgx_schur_uq(nd, npv, ncu, ndf, ne, *[d[k].ptr for k in KEYS], DUDG.ptr, DD.ptr, d["H"].ptr, FE.ptr,
                              None, None), "hdgx_schur_uq")
    torch.cuda.synchronize()
    ref = oracle.schur_uq(nd, blk)
    for k, v in (("DUDG", DUDG), ("DUDG_DUH", DD), ("AE", d["H"]), ("FE", FE)):
        assert np.abs(v.numpy() - ref[k]).max() / np.abs(ref[k]).max() < 1e-12, k
