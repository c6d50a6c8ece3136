"""The reciprocal inside the tensor-core eliminations, and small and large elements.

A diagonal block with the pairs (d, 1) on its diagonal has the determinants d, so the factorisation returns that
reciprocal itself: within 2 ulp of 1 / d over 80,000 mantissas and all exponents at which d and 1 / d are
normal numbers (an approximation good to 2^-20 or better, e^3 < 2^-59 after the step, and two roundings: below 2 ulp).

Elements scaled by powers of two: the mass matrix is of the order of the volume, so its 2 x 2 determinants leave
the range of normal numbers long before anything else does.  Reference: the oracle on the same elements; bounds of
test_element_mma_gpu.py and test_residual_gpu.py."""
import copy
from types import SimpleNamespace

import numpy as np
import pytest

from test_element_mma_gpu import _check, _state
from test_factor_gpu import _factor


def _reciprocals(d):
    n = d.size // 4
    H = np.zeros((8, 8, n), order="F")
    for i in range(4):
        H[2 * i, 2 * i], H[2 * i + 1, 2 * i + 1] = d[i * n:(i + 1) * n], 1.0
    mesh = SimpleNamespace(nf=n, cbsr_rowpts=np.arange(n + 1, dtype=np.int64), cbsr_colind=np.arange(1, n + 1, dtype=np.int32))
    M, st = _factor(mesh, H, np.arange(n, dtype=np.int32))
    assert not st.any()
    return np.concatenate([M[2 * i, 2 * i] for i in range(4)])


@pytest.mark.gpu
def test_reciprocal_within_two_ulp():
    r = np.random.default_rng(0)
    m = np.concatenate([1 + r.random(80000 - 8), [1.0, 1.5, 2 - 2.0 ** -52, 1 + 2.0 ** -52, 1 + 2.0 ** -20, 2 - 2.0 ** -20, 1.25, 1.75]])
    e = np.concatenate([np.zeros(20000, int), np.arange(60000) % 2043 - 1021])
    d = np.ldexp(m, e) * r.choice([-1.0, 1.0], m.size)
    with np.errstate(over="ignore"):
        ref = 1.0 / d
    got = _reciprocals(d)
    ulp = np.abs(got - ref) / np.spacing(np.abs(ref))
    assert ulp.max() < 2.0, (d[ulp.argmax()], got[ulp.argmax()])


SCALES = [(2, 1, -270), (2, 3, -270), (2, 3, 250), (3, 1, -175), (3, 2, -175), (3, 2, 165), (3, 3, -175)]


def _scaled(nd, p, k):
    P = _state(nd, p, False)
    P.mesh = copy.copy(P.mesh)
    P.mesh.dgnodes = np.asfortranarray(np.ldexp(P.mesh.dgnodes, k))
    P.UDG[:, P.app.ncu:] = np.ldexp(P.UDG[:, P.app.ncu:], -k)
    return P


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,k", SCALES)
def test_elements_of_extreme_size(oracle, nd, p, k):
    from hdg_b200.elemental import hdg_elemental
    P = _scaled(nd, p, k)
    _check(oracle, P, hdg_elemental(P.master, P.app, P.mesh.dgnodes, P.mesh.bf, P.UDG, P.UH, P.SH))


@pytest.mark.gpu
@pytest.mark.parametrize("nd,p,k", SCALES)
def test_gradients_of_elements_of_extreme_size(oracle, nd, p, k):
    from hdg_b200.elemental import getq
    P, P1 = _scaled(nd, p, k), _state(nd, p, False)
    run = lambda Q: getq(Q.master, Q.app, Q.mesh.dgnodes, Q.mesh.bf, Q.UDG, Q.UH, Q.SH)
    (Q, st), (Q1, _) = run(P), run(P1)
    assert int(st.numpy().max()) == 0
    # a power of two through and through: the same bits
    assert np.array_equal(np.ldexp(Q.numpy(), k), Q1.numpy())
