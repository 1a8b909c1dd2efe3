"""GPU: Gradient, Divergence, Curl and nonlinear_diffusion! in the reference's order where
it is asked for, at sizes that are evaluated in block fixed point by default: bit for bit
the values of the same points in an array or line below those sizes."""
import numpy as np
import pytest

import deo
from deo import _lib as L

pytestmark = pytest.mark.gpu
NEVER = 2 ** 63 - 1


@pytest.mark.parametrize("kind,n,m", [("Gradient", 104, 40), ("Curl", 164, 40)])
def test_vector_calculus(cuda, kind, n, m):
    import torch
    torch.manual_seed(1)
    ext = () if kind == "Gradient" else (3,)
    M = deo.julia_array((n + 2,) * 3 + ext)
    M.copy_(torch.randn(M.shape, dtype=M.dtype, device="cuda"))
    part = deo.julia_array((m + 2,) * 3 + ext)
    part.copy_(M[: m + 2, : m + 2, : m + 2])
    make = lambda k: getattr(deo, kind)(4, (0.1,) * 3, (k,) * 3)
    big, small = make(n), make(m)
    want = (small * part)[4:m - 4, 4:m - 4, 4:m - 4]
    by_default = (big * M)[4:m - 4, 4:m - 4, 4:m - 4].clone()
    L.lib().deo_vector_calculus_march_min(big._plan(0), NEVER)
    assert torch.equal((big * M)[4:m - 4, 4:m - 4, 4:m - 4], want) and not torch.equal(by_default, want)


def test_nonlinear_diffusion(cuda):
    import torch
    from deo.nonlinear import _plan
    torch.manual_seed(2)
    n, m = 1 << 17, 1000
    p, q = (torch.randn(n + 2, dtype=torch.float64, device="cuda") for _ in range(2))
    want = deo.nonlinear_diffusion(2, 1, 4, p[: m + 2].clone(), q[: m + 2].clone(), 0.1, m)[8:-8]
    by_default = deo.nonlinear_diffusion(2, 1, 4, p, q, 0.1, n)[8:m - 8]
    plan = _plan(2, 1, 4, 0.1, n, 0)
    try:
        L.lib().deo_nonlinear_diffusion_march_min(plan._h, NEVER)
        assert torch.equal(deo.nonlinear_diffusion(2, 1, 4, p, q, 0.1, n)[8:m - 8], want) and not torch.equal(by_default, want)
    finally:
        L.lib().deo_nonlinear_diffusion_march_min(plan._h, 0)
