"""GPU: A \\ u for upwind operators of high order, whose interior columns hold 9 to
14 entries of U and at most one multiplier: counts of two digits, which must not
be taken for one of the solve kernel's short patterns.

Tolerance: 16 cond(A_l) eps relative in the 2-norm, the bar of the other solve
tests (cond up to 1.6e10 here)."""
import numpy as np
import pytest

import deo
import oracle as O
from test_gpu_solve import EPS, _dev, _host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1.0, -1.0])
@pytest.mark.parametrize("off,a", [(0, 9), (0, 10), (0, 11), (1, 11), (1, 12), (1, 13), (1, 14)])
def test_wide_upwind_bands(cuda, off, a, c):
    n = 40
    h = 1.0 / (n + 1)
    u = np.random.default_rng(a).standard_normal(n)
    x = _host(deo.ldiv(deo.UpwindDifference(1, a, h, n, c, offside=off) * deo.Dirichlet0BC(), _dev(u)))
    ref, cond = O.ghost_solve(O.upwind(1, a, h, n, c, offside=off), O.dirichlet0(), u)
    assert np.linalg.norm(x - ref) <= 16 * cond * EPS * np.linalg.norm(ref)
