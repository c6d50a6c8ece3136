"""getq and the element residual (their own kernel) over every compiled shape, for launches of few elements
(four warps each) and of many, on the noisy states of test_element_mma_gpu.py.

Reference: the oracle.  Bound as in tests/test_dirk_gpu.py: max(1e-12, 10 x the oracle's own change when
dgnodes, UDG and UH move by one ulp)."""
import numpy as np
import pytest

from test_element_mma_gpu import SHAPES, _state


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def _jitter(seed):
    r = np.random.default_rng(seed)
    return lambda x: x * (1.0 + 2.2e-16 * r.standard_normal(x.shape))


def _times(a, copies):
    return np.asfortranarray(np.tile(a, (1,) * (a.ndim - 1) + (copies,)))


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,visc", SHAPES)
@pytest.mark.parametrize("copies", [1, 150])
@pytest.mark.parametrize("tdep", [False, True])
def test_residual_every_shape(oracle, nd, p, visc, copies, tdep):
    from hdg_b200.elemental import residual
    P = _state(nd, p, visc, tdep)
    m, jit = P.mesh, _jitter(1)
    if tdep:
        P.SH[:, P.app.ncu:] = np.random.default_rng(2).standard_normal(P.SH[:, P.app.ncu:].shape)
    ref = oracle.residual(P.master, P.app, m.dgnodes, m.bf, P.UDG, P.UH, P.SH)
    ref1 = oracle.residual(P.master, P.app, jit(m.dgnodes), m.bf, jit(P.UDG), jit(P.UH), P.SH)
    Ru, st = residual(P.master, P.app, *(_times(x, copies) for x in (m.dgnodes, m.bf, P.UDG, P.UH, P.SH)))
    assert int(st.numpy().max()) == 0
    assert _rel(Ru.numpy(), _times(ref, copies)) < max(1e-12, 10 * _rel(ref1, ref))


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,visc", SHAPES)
@pytest.mark.parametrize("copies", [1, 150])
def test_getq_every_shape(oracle, nd, p, visc, copies):
    from hdg_b200.elemental import getq
    P = _state(nd, p, visc)
    m, jit = P.mesh, _jitter(3)
    sh = np.zeros_like(P.UDG)
    sh[:, P.app.ncu:] = np.random.default_rng(4).standard_normal(sh[:, P.app.ncu:].shape)
    for s, fc_q in ((sh, 0.7), (None, 1.0)):
        ref = oracle.getq(P.master, P.app, m.dgnodes, m.bf, P.UDG, P.UH, s, fc_q)
        ref1 = oracle.getq(P.master, P.app, jit(m.dgnodes), m.bf, jit(P.UDG), jit(P.UH), s, fc_q)
        big = [_times(x, copies) for x in (m.dgnodes, m.bf, P.UDG, P.UH)]
        Q, st = getq(P.master, P.app, *big, None if s is None else _times(s, copies), fc_q=fc_q)
        assert int(st.numpy().max()) == 0
        assert _rel(Q.numpy(), _times(ref, copies)) < max(1e-12, 10 * _rel(ref1, ref))


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,visc", [(2, 3, True), (3, 1, False)])
def test_status_is_that_of_the_elemental_kernel(nd, p, visc):
    """Faces of a boundary type that no flux is known for, elements collapsed to a point and nearly so."""
    from hdg_b200.elemental import hdg_elemental, residual
    P = _state(nd, p, visc)
    P.app.bcm = [9] * len(P.app.bcm)
    m = P.mesh
    m.dgnodes[:, :, 2] = m.dgnodes[:1, :, 2]
    m.dgnodes[:, :, 4] = 0.0
    _, st = residual(P.master, P.app, m.dgnodes, m.bf, P.UDG, P.UH, P.SH)
    out = hdg_elemental(P.master, P.app, m.dgnodes, m.bf, P.UDG, P.UH, P.SH)
    assert np.array_equal(st.numpy(), out.status.numpy())
    assert int(st.numpy().ravel()[4]) != 0
