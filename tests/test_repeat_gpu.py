"""An application of the BILU(0) factors and a whole linear solve give the same bits every time, whatever else
runs on the GPU: every block size, sums of several neighbours per row, with copies on a second stream beside them."""
import pytest

from test_sweep_gpu import CASES, _system


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", CASES + [("c4", dict(n=8, porder=2)), ("c2", dict(n=40, porder=3))])
def test_same_bits_every_time(oracle, name, kw):
    import torch
    P, ts, dM, DArray = _system(oracle, name, kw)
    gen = torch.Generator("cuda").manual_seed(5)
    x = DArray(torch.randn(ts.bs * ts.nf, dtype=torch.float64, device="cuda", generator=gen), (ts.bs, ts.nf))
    other, big = torch.cuda.Stream(), torch.zeros(1 << 24, dtype=torch.float64, device="cuda")
    first = None
    for rep in range(40):
        v, w = ts.empty_vec(), ts.empty_vec()
        if rep % 2:
            with torch.cuda.stream(other):
                big.add_(1.0)
        ts.bilu0_apply(dM, x, v, w)
        torch.cuda.synchronize()
        bits = v.t.view(torch.int64).clone()
        first = bits if first is None else first
        assert torch.equal(bits, first), f"application {rep}: {int((bits != first).sum())} values differ"


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
def test_same_solve_every_time(mixed):
    import numpy as np
    from hdg_b200 import configs
    from hdg_b200.solve import hdgx_solve
    P = configs.by_name("c4", n=3, porder=2)
    first = None
    for _ in range(4):
        U, H, _ = hdgx_solve(P.master, P.mesh, P.app, P.UDG, P.UH, P.SH, tol=1e-10, maxiter=2, mixed=mixed)
        first = U if first is None else first
        assert np.array_equal(U.view(np.int64), first.view(np.int64))
