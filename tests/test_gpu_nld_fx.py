"""GPU: nonlinear_diffusion! on long uniform lines (Float64, block fixed point)
against the oracle.

Bound: a derivative is within 2 ulp of its own sum |w u|, the oracle's within
3.5 EPS of it (7 taps), so a product of two of them within 11 EPS of the product
of the sums and 2 EPS for the product's and the sum's rounding: 13 EPS < 16."""
import numpy as np
import pytest

import deo
import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
TILE, MIN = 512, 1 << 17  # points of a tile; shortest line that takes the kernel


def _field(kind, n, rng):
    x = rng.standard_normal(n)
    if kind == "smooth":
        return np.sin(np.linspace(0, 9, n)) + 1e-3 * x
    if kind == "scales":  # most points far below their tile's largest
        return x * 10.0 ** rng.integers(-30, 3, n)
    if kind == "sparse":
        return np.where(rng.random(n) < 0.01, x, 0.0)
    if kind == "extreme":  # the ends of the exponent range, tile by tile
        return x * np.resize(np.repeat([1e-305, 1e140, 1e-320, 1e-8], TILE), n)
    x[[0, 700, n - 1]] = [np.inf, np.nan, -np.inf]
    return x


@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("m", [0, 1])
@pytest.mark.parametrize("a", [2, 4])
@pytest.mark.parametrize("size,kind", [(MIN, "smooth"), (MIN + 1, "sparse"), (MIN + TILE - 1, "scales"),
                                       (MIN + 77, "extreme"), (MIN + 2, "special"), (MIN + TILE - 2, "zeros")])
def test_long_lines(cuda, n, m, a, size, kind):
    import torch
    rng = np.random.default_rng(size + 10 * n + m + 100 * a)
    h = 1.0 / (size + 1)
    if kind == "zeros":
        p, q = np.zeros(size + 2), rng.standard_normal(size + 2)
    else:
        q = _field(kind, size + 2, rng)
        p = rng.uniform(0.5, 2.0, size + 2) if kind in ("extreme", "special") else _field(kind, size + 2, rng)
    du = torch.full((size,), 7.0, device="cuda", dtype=torch.float64)
    deo.nonlinear_diffusion_(du, n, m, a, torch.from_numpy(p).cuda(), torch.from_numpy(q).cuda(), h, size)
    got = du.cpu().numpy()
    with np.errstate(all="ignore"):
        ref = O.nonlinear_diffusion(n, m, a, p, q, h, size)
        scale = O.nonlinear_diffusion(n, m, a, p, q, h, size, absolute=True)
    if kind == "extreme":
        # sums that reach the subnormal range round to 2^-1074, which the bound does not
        # count: those tiles are in the reference's order, bit for bit a short line's
        for t in range(2 * TILE, size - TILE, 64 * TILE):
            s = slice(t, t + TILE + 2)
            short = deo.nonlinear_diffusion(n, m, a, torch.from_numpy(p[s]).cuda(), torch.from_numpy(q[s]).cuda(), h, TILE)
            assert np.array_equal(got[t + 8:t + TILE - 8], short.cpu().numpy()[8:-8])
        scale[(np.arange(size) // TILE) % 4 == 2] = np.inf
        got[~np.isfinite(scale)] = ref[~np.isfinite(scale)]
    fin = np.isfinite(scale)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert (np.abs(got - ref)[fin] <= 16 * EPS * scale[fin] + 5e-324).all(), np.nanmax(np.abs(got - ref)[fin])
    assert np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
