"""GPU: the marching block fixed-point Laplacian on values that are small against their
block's largest, where the rest of a unit is evaluated on exponents of its points' own or in
the reference's order: pulses of a few cells, values that fall by many binades a cell (in
every direction, so that the block's exponent rises and falls), a pulse behind ordinary
values, small regions among zeros and subnormals, Inf and NaN in a pulse's foot.  Band radii
1-3, one band for the axes and three, forward and transposed, more than one tile and chunk.

Tolerance: 4 ulp of sum |c_k u_k|: the kernel's bound is 2 ulp and half an ulp of its rounding,
the oracle's sums of 5 to 7 rounded products and 2 additions stay below 1.5."""
import numpy as np
import pytest

import deo
import oracle as O
from cases import build, to_device, to_host
from test_gpu_parity import T

pytestmark = pytest.mark.gpu
SHAPE = (70, 19, 61)


def _field(kind):
    rng = np.random.default_rng(3)
    x, y, z = np.meshgrid(*(np.arange(n, dtype=np.float64) for n in SHAPE), indexing="ij")
    r2 = (x - 30.3) ** 2 + (y - 9.1) ** 2 + (z - 33.7) ** 2
    if kind == "pulse":
        v = np.exp(-r2 / 18.0)
    elif kind == "steep":
        v = np.exp2(-6.5 * np.sqrt(r2)) * (1 + rng.random(SHAPE))
    elif kind == "late":
        v = np.where(z < 25, rng.standard_normal(SHAPE), -np.exp(-r2 / 18.0))
    elif kind == "island":
        v = np.where(r2 < 60, np.exp2(-np.round(r2)) * rng.standard_normal(SHAPE), 0.0)
        v[50:55] = 2.0 ** -1060
        v[x < 2] = -0.0
        v[10, 9, 33] = 1.0
    else:  # "special"
        v = np.exp(-r2 / 18.0)
        v[55, 10, 30], v[12, 5, 40] = np.inf, np.nan
    return np.asfortranarray(v)


@pytest.mark.parametrize("field", ["pulse", "steep", "late", "island", "special"])
@pytest.mark.parametrize("a,one_band", [(2, True), (4, True), (6, True), (2, False), (4, False), (6, False)])
def test_small_values(cuda, a, one_band, field):
    h = [1 / 65.0] * 3 if one_band else [0.1, 0.07, 0.2]
    A, oterms, _ = build(dict(shape=SHAPE, terms=[T("centered", 2, a, axis=k + 1, h=h[k], bc=("dirichlet0",)) for k in range(3)],
                              seed=1))
    u = _field(field)
    p, g = deo.Plan(A.terms(), SHAPE, 0), deo.Plan(A.terms(), SHAPE, 0)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)  # the kernel at every size
    g.set_option(deo.DEO_OPT_FAST_PATH, 0)
    scale = O.abs_scale(oterms, u)
    base = np.asfortranarray(np.random.default_rng(6).standard_normal(SHAPE))
    out, acc, other = deo.julia_array(SHAPE, fill=np.nan), to_device(base), deo.julia_array(SHAPE, fill=np.nan)
    p.apply(to_device(u), out)
    assert p.kernels[0] == "k_lap_fx"
    p.apply(to_device(u), acc, overwrite=False)

    def close(got, ref, where):
        fin = np.isfinite(ref) & where
        assert np.array_equal(np.isnan(got)[where], np.isnan(ref)[where])
        inf = np.isinf(ref) & where
        assert np.array_equal(got[inf], ref[inf])
        err = np.abs(got - ref)[fin] / np.spacing(np.where(np.isfinite(scale), scale, 1.0))[fin]
        assert (err <= 4).all(), float(err.max())

    got = to_host(out)
    close(got, O.apply(oterms, u), np.ones(SHAPE, bool))
    fin = np.isfinite(got)
    assert np.array_equal(to_host(acc)[fin], (got + base)[fin])
    # transposed: the columns read by interior rows alone have the forward weights (symmetric bands)
    p.adjoint(to_device(u), out)
    assert p.kernels[0] == "k_lap_fx"
    g.adjoint(to_device(u), other)
    inner = np.zeros(SHAPE, bool)
    inner[(slice(a + 2, -a - 2),) * 3] = True
    close(to_host(out), to_host(other), inner)
