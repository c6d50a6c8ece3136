"""An application of the BILU(0) factors with vectors that share storage: the solution over the right-hand side, the work
vector over either, all three in one place, and each of them shifted against another by some rows.  The same
sweeps run, so the solution has the bits of the call on three separate vectors (one launch per level sums in
another order); also captured into a graph."""
import ctypes as ct

import pytest

from test_sweep_gpu import CASES, _system

# offsets in rows of x, v and work in one array of four vectors' length
PLACES = {"v=x": (0, 0, 2), "work=x": (0, 2, 0), "work=v": (0, 2, 2), "all": (0, 0, 0), "v~x": (0, .4, 2), "x~v": (.4, 0, 2),
          "work~x": (0, 2, .4), "work~v": (0, 2, 2.4), "chain": (0, .4, .8)}


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [CASES[k] for k in (1, 2, 3, 4, 6, 8)])
@pytest.mark.parametrize("place", list(PLACES))
def test_same_bits_as_apart(oracle, name, kw, place):
    import torch
    from hdg_b200._lib import check, lib
    P, ts, dM, DArray = _system(oracle, name, kw)
    n = ts.bs * ts.nf
    gen = torch.Generator("cuda").manual_seed(3)
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    ref, w = ts.empty_vec(), ts.empty_vec()
    ts.bilu0_apply(dM, DArray(b.clone(), (ts.bs, ts.nf)), ref, w)
    mem = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
    x, v, wk = (mem[int(o * ts.nf) * ts.bs:][:n] for o in PLACES[place])

    def apply():
        x.copy_(b)
        check(lib().hdgx_bilu0_apply(ct.byref(ts.bsr), dM.ptr, x.data_ptr(), v.data_ptr(), wk.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream), "hdgx_bilu0_apply")
    for _ in range(2):
        apply()
        torch.cuda.synchronize()
        assert torch.equal(v.view(torch.int64), ref.t.view(torch.int64))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            apply()
        for _ in range(2):
            mem.zero_()
            g.replay()
            side.synchronize()
            assert torch.equal(v.view(torch.int64), ref.t.view(torch.int64))
