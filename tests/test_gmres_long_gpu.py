"""GMRES on vectors too long for the fused Gram-Schmidt step (1,700,000 unknowns): the separate products, on the
systems and with the bounds of test_gmres_step_gpu.py; just below and above the line."""
import pytest

from test_gmres_step_gpu import _solve


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [8000, 8200])
def test_long_vectors(copies):
    assert _solve(copies, 7, 30, lambda r, eye: r / 30, 4.0, 20, True) > 1
