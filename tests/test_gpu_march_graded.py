"""GPU: 3-D Float64 Laplacians with an odd first size on grids that are uniform only in
part: against the oracle, and on the kernel that is the faster one there (the marching
kernel where it holds two thirds of the points, the generic one elsewhere)."""
import numpy as np
import pytest

import deo
import oracle as O
from cases import to_device, to_host

pytestmark = pytest.mark.gpu
SHAPE = (75, 70, 66)


def _steps(kind, n):
    if kind == "halves":
        return np.r_[np.full(n // 2, 1.0 / n), np.full(n + 1 - n // 2, 2.0 / n)]
    if kind == "ends":
        return np.r_[np.full(4, 0.5 / n), np.full(n - 7, 1.0 / n), np.full(4, 0.5 / n)]
    return 1.0 / (n + 1)


@pytest.mark.parametrize("kinds,kernel", [("u/u/u", "k_lap_fx"), ("u/u/ends", "k_lap_fx"), ("u/u/halves", "k_apply"),
                                          ("halves/u/u", "k_apply"), ("halves/halves/halves", "k_apply")])
@pytest.mark.parametrize("a", [2, 4])
def test_partly_uniform_grids(cuda, kinds, kernel, a):
    dx = [_steps(k, n) for k, n in zip(kinds.split("/"), SHAPE)]
    A = deo.DiffEqOperatorCombination([deo.CenteredDifference(2, a, dx[k], SHAPE[k], axis=k + 1) * deo.MultiDimDirectionalBC(
        deo.Dirichlet0BC(), k + 1, SHAPE) for k in range(3)])
    terms = [(O.centered(2, a, dx[k], SHAPE[k], axis=k + 1), O.dirichlet0(), None) for k in range(3)]
    u = np.asfortranarray(np.random.default_rng(3).standard_normal(SHAPE))
    p, out = deo.Plan(A.terms(), SHAPE, 0), deo.julia_array(SHAPE, fill=np.nan)
    p.apply(to_device(u), out)
    assert p.kernels[0] == kernel
    err = np.abs(to_host(out) - O.apply(terms, u)) / np.spacing(O.abs_scale(terms, u))
    assert (err <= 4).all(), float(err.max())
