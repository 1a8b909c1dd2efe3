"""GPU: Gradient / Divergence / Curl in block fixed point on values that are small against their
block's largest, where the rest of a unit is evaluated on the exponents of each derivative's own
taps: pulses of a few cells, values that fall by many binades a cell in every direction, a pulse
behind ordinary values, small regions among zeros and subnormals, one component of another scale,
Inf and NaN in a pulse's foot.  Orders 2, 4, 6, more than one tile and chunk; overwriting and
adding.

Tolerance: 4 ulp of sum |c_k u_k|, as for the kernel's other fields: its bound is 2 ulp and half
an ulp of each rounding, the oracle's sums of 3 to 7 products stay below 1.5."""
import numpy as np
import pytest

import deo
import oracle as O
from deo import _lib as L
from test_gpu_vector_march import KINDS, _dev, _host, _in_shape, _pair

pytestmark = pytest.mark.gpu


def _field(kind, shape):
    rng = np.random.default_rng(3)
    g = np.meshgrid(*(np.arange(n, dtype=np.float64) for n in shape), indexing="ij")
    x, y, z = g[:3]
    c = g[3] if len(g) > 3 else 0.0
    r2 = (x - 30.3) ** 2 + (y - 9.1 - c) ** 2 + (z - 23.7) ** 2
    if kind == "pulse":
        v = np.exp(-r2 / 18.0)
    elif kind == "steep":
        v = np.exp2(-6.5 * np.sqrt(r2)) * (1 + rng.random(shape))
    elif kind == "late":
        v = np.where(z < 15, rng.standard_normal(shape), -np.exp(-r2 / 18.0))
    elif kind == "island":
        v = np.where(r2 < 60, np.exp2(-np.round(r2)) * rng.standard_normal(shape), 0.0)
        v = np.where((x >= 50) & (x < 55), 2.0 ** -1060, v)
    elif kind == "scales":
        v = np.exp(-r2 / 18.0) * np.exp2(-200.0 * c)
        v = np.where(c == 2, 0.0, v)
    else:  # "special"
        v = np.exp(-r2 / 18.0)
        v[(45, 10, 30) + (0,) * (len(shape) - 3)], v[(12, 5, 40) + (0,) * (len(shape) - 3)] = np.inf, np.nan
    return np.asfortranarray(v)


@pytest.mark.parametrize("field", ["pulse", "steep", "late", "island", "scales", "special"])
@pytest.mark.parametrize("kind,lens,a", [("gradient", (70, 19, 61), 2), ("gradient", (70, 19, 61), 4), ("gradient", (70, 19, 61), 6),
                                         ("divergence", (70, 19, 61), 2), ("divergence", (70, 19, 61), 4),
                                         ("divergence", (70, 19, 61), 6), ("curl", (67, 67, 67), 2), ("curl", (67, 67, 67), 4),
                                         ("curl", (67, 67, 67), 6)])
def test_small_values(cuda, kind, lens, a, field):
    M = _field(field, _in_shape(kind, lens))
    A, ops = _pair(kind, a, [1.0, 0.5, 2.0] if kind != "curl" else [0.5] * 3, lens)
    k = KINDS[kind][0]
    base = np.asfortranarray(np.random.default_rng(7).standard_normal(A.out_shape()))
    out, acc, Md = deo.julia_array(A.out_shape(), fill=np.nan), _dev(base), _dev(M)
    L.lib().deo_vector_calculus_march_min(A._plan(0), 0)  # the kernel itself, below the sizes that choose it
    A.mul_(out, Md, overwrite=True)
    A.mul_(acc, Md)
    for got, init in ((_host(out), None), (_host(acc), base)):
        ref = O.vector_calculus(k, ops, M, out=None if init is None else np.asfortranarray(init.copy()), overwrite=init is None)
        scale = O.vector_calculus(k, ops, M, absolute=True) + (0 if init is None else np.abs(init))
        fin = np.isfinite(ref)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
        ulp = np.spacing(np.where(np.isfinite(scale), scale, 1.0))[fin]
        err = np.abs(got[fin] - ref[fin])
        assert (err <= 4 * ulp).all(), float((err / ulp).max())
