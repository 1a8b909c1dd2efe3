"""GPU: nonlinear_diffusion! on long Float64 lines whose steps differ -- of two sizes, by
a rounding, in one place -- against the oracle (the bound of the uniform lines' test: 16
EPS of the products of sums of moduli), and in the row-table kernel's time: a line of
2^17 points, where the block fixed-point kernel begins, against one a point shorter."""
import numpy as np
import pytest

import deo
import oracle as O
from test_gpu_nld_fx import EPS, MIN

pytestmark = pytest.mark.gpu


def _steps(kind, n):
    if kind == "halves":
        return np.r_[np.full(n // 2, 1e-5), np.full(n + 1 - n // 2, 2e-5)]
    if kind == "linspace":
        return np.diff(np.linspace(0.0, 1.0, n + 2))
    dx = np.full(n + 1, 1.0 / n)
    dx[n // 3] *= 1.5
    return dx


@pytest.mark.parametrize("kind", ["halves", "linspace", "one"])
def test_steps_that_differ(cuda, kind):
    import torch

    def run(n):
        rng = np.random.default_rng(2)
        p, q, dx = rng.uniform(0.5, 1.5, n + 2), rng.uniform(0.5, 1.5, n + 2), _steps(kind, n)
        du, pd, qd = torch.full((n,), 7.0, device="cuda", dtype=torch.float64), torch.from_numpy(p).cuda(), torch.from_numpy(q).cuda()
        times = []
        for _ in range(8):
            e = torch.cuda.Event(True), torch.cuda.Event(True)
            e[0].record()
            for _ in range(4):
                deo.nonlinear_diffusion_(du, 2, 1, 2, pd, qd, dx, n)
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        return min(times), du.cpu().numpy(), (2, 1, 2, p, q, dx, n)

    t, got, args = run(MIN)
    ref, scale = O.nonlinear_diffusion(*args), O.nonlinear_diffusion(*args, absolute=True)
    assert (np.abs(got - ref) <= 16 * EPS * scale).all()
    assert t < 2 * run(MIN - 1)[0]
