"""GPU: the transposed apply of 3-D Float64 plans on the marching kernel, point by
point: symmetric bands, and bands of a diffusion and an advection term merged into
one, whose weights at -1 and +1 differ (up to a weight of zero at cell Peclet number
2).  Fields: noise, a front with values many binades below it behind it, isolated
values, values of all scales.

The reference is the sum over the stencil's own weights (read off the generic
kernel's response to a unit impulse) in extended precision, at the points whose
columns are read by interior rows alone.

Tolerance: 2 ulp of sum |w d| (the kernel's bound) + 0.5 of its rounding, or, for
points in the reference's order, 1.5 for sums of 7 rounded products: below 4."""
import numpy as np
import pytest

import deo
from cases import build, to_device, to_host
from test_gpu_parity import T

pytestmark = pytest.mark.gpu
SHAPE = (70, 22, 26)


def _field(kind):
    rng = np.random.default_rng(7)
    v = rng.standard_normal(SHAPE)
    if kind == "front":
        x = np.arange(SHAPE[0])[:, None, None]
        v = np.where(x < 30, 1.0 + 0.1 * v, v * np.exp2(-20.0 - 0.3 * (x - 30)))
    elif kind == "sparse":
        v = np.where(rng.random(SHAPE) < 0.03, np.round(4 * v), 0.0)
    elif kind == "spikes":  # one large value among small ones
        v = np.where(rng.random(SHAPE) < 0.01, v, 2.0 ** -30 * v)
    elif kind == "wide":
        v = v * np.exp2(rng.integers(-40, 41, size=SHAPE).astype(np.float64))
    return np.asfortranarray(v)


@pytest.mark.parametrize("field", ["normal", "front", "sparse", "spikes", "wide"])
@pytest.mark.parametrize("a,peclet", [(2, 0.0), (4, 0.0), (2, 1.0), (2, 1.9), (2, -1.9), (2, 1.99), (2, 2.0), (2, -2.0), (4, 1.3)])
def test_transposed_against_its_stencil(cuda, a, peclet, field):
    h, bc = 1.0 / 71, ("dirichlet0",)
    terms = [T("centered", 2, a, axis=k, h=h, bc=bc) for k in (1, 2, 3)]
    if peclet:
        terms += [T("centered", 1, a, axis=k, h=h, bc=bc, coeff=peclet / h) for k in (1, 2, 3)]
    A, _, _ = build(dict(shape=SHAPE, terms=terms, seed=1))
    p, g = (deo.Plan(A.terms(), SHAPE, 0, merge_terms=True) for _ in range(2))
    g.set_option(deo.DEO_OPT_FAST_PATH, 0)
    c = tuple(n // 2 for n in SHAPE)
    one, resp = np.zeros(SHAPE, order="F"), deo.julia_array(SHAPE)
    one[c] = 1.0
    g.apply(to_device(one), resp)  # resp[c + o] = w[-o], the transpose's weight of d[x - o]
    r = to_host(resp)
    d = _field(field)
    H = a // 2
    ref, scale = np.zeros(SHAPE, np.longdouble), np.zeros(SHAPE)
    for axis in range(3):
        for o in range(-H, H + 1):
            at = list(c)
            at[axis] += o
            w = r[tuple(at)] if o or axis == 0 else 0.0  # (the centre weights come added)
            # out[x] = sum over rows i of A[i, x] d[i]; row i = x + o reads x at -o with w[-o] = resp[c + o]
            ref += np.longdouble(w) * np.roll(d, -o, axis)
            scale += np.abs(w * np.roll(d, -o, axis))
    out = deo.julia_array(SHAPE, fill=np.nan)
    p.adjoint(to_device(d), out)
    assert p.kernels[0] == "k_lap_fx"
    m = (slice(3 * H + 1, -3 * H - 1),) * 3
    err = np.abs(to_host(out).astype(np.longdouble) - ref)[m] / np.spacing(scale)[m]
    assert (err <= 4).all(), float(err.max())
