"""GPU: 2-D Float64 plans in block fixed point on tiles whose values are small against their
largest, evaluated on the exponents of each row's own taps: pulses of a few points, values that
fall by many binades a point, a pulse beside ordinary values in one tile, small regions among
zeros and subnormals, Inf and NaN in a pulse's foot.

Tolerance: 4 ulp of sum|c_k u_k|, as for the kernel's other fields: each axis's sum is within 2
ulp of its own scale and half an ulp of its rounding; the oracle's sums stay below 1.5."""
import numpy as np
import pytest

import deo
import oracle as O
from cases import build, to_device, to_host
from test_gpu_rows_fx import PLANS

pytestmark = pytest.mark.gpu
SHAPE = (100, 71)


def _field(kind):
    rng = np.random.default_rng(3)
    x, y = np.meshgrid(*(np.arange(n, dtype=np.float64) for n in SHAPE), indexing="ij")
    r2 = (x - 30.3) ** 2 + (y - 40.1) ** 2
    if kind == "pulse":
        v = np.exp(-r2 / 18.0)
    elif kind == "steep":
        v = np.exp2(-6.5 * np.sqrt(r2)) * (1 + rng.random(SHAPE))
    elif kind == "beside":
        v = np.where(y < 45, rng.standard_normal(SHAPE), -np.exp(-((x - 30) ** 2 + (y - 45) ** 2) / 9.0))
    elif kind == "island":
        v = np.where(r2 < 60, np.exp2(-np.round(r2)) * rng.standard_normal(SHAPE), 0.0)
        v[50:55] = 2.0 ** -1060
        v[55] = -0.0
    else:  # "special"
        v = np.exp(-r2 / 18.0)
        v[55, 10], v[12, 60] = np.inf, np.nan
    return np.asfortranarray(v)


@pytest.mark.parametrize("field", ["pulse", "steep", "beside", "island", "special"])
@pytest.mark.parametrize("name", list(PLANS))
def test_small_values(cuda, name, field):
    A, oterms, _ = build(dict(shape=SHAPE, terms=PLANS[name], seed=3))
    u = _field(field)
    p = deo.Plan(A.terms(), SHAPE, 0)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)  # the kernel at every size
    base = np.asfortranarray(np.random.default_rng(6).standard_normal(SHAPE))
    out, acc = deo.julia_array(SHAPE, fill=np.nan), to_device(base)
    p.apply(to_device(u), out)
    assert p.kernels == ("k_rows_fx",)
    p.apply(to_device(u), acc, overwrite=False)
    got = to_host(out)
    with np.errstate(all="ignore"):
        ref, scale = O.apply(oterms, u), O.abs_scale(oterms, u)
        fin = np.isfinite(ref)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
        err = np.abs(got - ref)[fin] / np.spacing(np.where(np.isfinite(scale), scale, 1.0))[fin]
    assert (err <= 4).all(), float(err.max())
    assert np.array_equal(to_host(acc)[fin], (got + base)[fin])
