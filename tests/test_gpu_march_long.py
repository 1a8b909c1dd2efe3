"""GPU: the marching kernel on arrays long in axis 3: against the generic kernel (4 ulp of
sum |c_k u_k|, from its response to |u|'s bound: the largest weights), and the host's
share of a call, which does not grow with the length."""
import time

import numpy as np
import pytest

import deo

pytestmark = pytest.mark.gpu


def _plan(n):
    A = deo.DiffEqOperatorCombination([deo.CenteredDifference(2, 2, 1.0, n[k], axis=k + 1) * deo.MultiDimDirectionalBC(
        deo.Dirichlet0BC(), k + 1, n) for k in range(3)])
    return deo.Plan(A.terms(), n, 0)


@pytest.mark.parametrize("nz", [5, 257, 1021, 20000])
def test_chunks_of_any_length(cuda, nz):
    import torch
    n = (24, 18, nz)
    p, g = _plan(n), _plan(n)
    g.set_option(deo.DEO_OPT_FAST_PATH, 0)
    torch.manual_seed(nz)
    u, out, ref = deo.julia_array(n), deo.julia_array(n, fill=np.nan), deo.julia_array(n)
    u.copy_(torch.randn(n, dtype=torch.float64, device="cuda"))
    for f, h in ((p.apply, g.apply), (p.adjoint, g.adjoint)):
        out.fill_(float("nan"))
        f(u, out)
        h(u, ref)
        # sum |c_k u_k| <= 12 max|u| < 64
        assert float((out - ref).abs().max()) <= 4 * np.spacing(32.0)


def test_host_share_of_a_call(cuda):
    import torch
    n = (16, 16, 400_000)
    p, u, out = _plan(n), deo.julia_array(n, fill=1.0), deo.julia_array(n)
    best = 1.0
    for _ in range(20):
        torch.cuda.synchronize()
        t = time.perf_counter()
        p.apply(u, out)
        best = min(best, time.perf_counter() - t)
    torch.cuda.synchronize()
    assert best < 150e-6, best
