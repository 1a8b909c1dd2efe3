"""GPU: A \\ u for line lengths around the solve kernel's 8-step blocks, where its
plain columns (one pattern of interchanges, multipliers and entries of U) begin
and end: tridiagonal and 4-diagonal bands, with and without interchanges, with
A_b zero and not, Float64 and Float32, in place and out of place.

Tolerance: 16 cond(A_l) eps relative in the 2-norm, the bar of the other solve
tests; Float32 adds the rounding of its input and result."""
import numpy as np
import pytest

import deo
import oracle as O
from test_gpu_solve import EPS, _dev, _host

pytestmark = pytest.mark.gpu
BCS = {"dirichlet0": (lambda h, a: deo.Dirichlet0BC(), lambda h, a: O.dirichlet0()),
       "dirichlet": (lambda h, a: deo.DirichletBC(1.5, -0.5), lambda h, a: O.dirichlet(1.5, -0.5)),
       "robin": (lambda h, a: deo.RobinBC((1.0, 0.5, 0.1), (1.0, 0.5, -0.2), h, a),
                 lambda h, a: O.robin((1.0, 0.5, 0.1), (1.0, 0.5, -0.2), h, a))}


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("bc", list(BCS))
@pytest.mark.parametrize("a", [2, 4])
def test_line_lengths(cuda, a, bc, dtype):
    rng = np.random.default_rng(4)
    for n in (9, 12, 15, 16, 17, 24, 31, 40, 41, 100):
        h = 1.0 / (n + 1)
        A = deo.CenteredDifference(2, a, h, n, axis=2) * deo.MultiDimBC(BCS[bc][0](h, a), (5, n, 3), 2)
        u = rng.standard_normal((5, n, 3))
        if dtype == "f32":
            u = u.astype(np.float32).astype(np.float64)
        ud = _dev(u, dtype)
        x = _host(deo.ldiv(A, ud))
        deo.ldiv_(ud, A, ud)
        assert np.array_equal(_host(ud), x)
        op, q = O.centered(2, a, h, n), BCS[bc][1](h, a)
        for i in range(5):
            for k in range(3):
                ref, cond = O.ghost_solve(op, q, u[i, :, k])
                tol = 16 * cond * EPS + (2.0 ** -23 if dtype == "f32" else 0.0)
                assert np.linalg.norm(x[i, :, k] - ref) <= tol * np.linalg.norm(ref), (n, i, k)
