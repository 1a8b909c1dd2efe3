"""GPU: the marching block fixed-point Float64 kernel of Gradient / Divergence /
Curl (3-D, uniform grids) against the oracle at the edges of its 64 x 8 tiles,
below them and at odd sizes, orders 2 to 6, on fields that meet its branches:
exponents that rise and fall, zeros beside values, values far below their
block's largest, Inf/NaN, and scales near the ends of the Float64 range.

Tolerance: 4 ulp of sum |c_k u_k| per output entry, the bar of the Float64
vector operators: each derivative is within 2 ulp of its own sum plus its
rounding, added as the reference adds them; the oracle's sums of up to 7 rounded
products stay below 1.5."""
import numpy as np
import pytest

import deo
import oracle as O
from deo import _lib as L
from test_gpu_vector import _dev, _host, _in_shape, _pair, KINDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["normal", "waves", "zeros", "sparse", "wide", "special", "tiny", "huge"])
@pytest.mark.parametrize("kind,lens,a", [("gradient", (64, 8, 12), 4), ("gradient", (67, 17, 30), 2),
                                         ("gradient", (131, 9, 9), 6), ("divergence", (66, 10, 21), 4),
                                         ("divergence", (33, 19, 8), 2), ("curl", (20, 20, 20), 4),
                                         ("curl", (67, 67, 67), 2), ("curl", (9, 9, 9), 6)])
def test_vector_march_against_oracle(cuda, kind, lens, a, field):
    rng = np.random.default_rng(11)
    shape = _in_shape(kind, lens)
    M = rng.standard_normal(shape)
    if field == "waves":
        z = np.arange(shape[2]).reshape((1, 1, -1) + (1,) * (len(shape) - 3))
        M = np.exp2(6 * np.sin(z / 2.0)) + 1e-3 * M
    elif field == "zeros":
        M[:, :, shape[2] // 2:] = 0.0
        M[: shape[0] // 3] = 0.0
    elif field == "sparse":  # points that see one small-weight tap, or nothing
        M = np.where(rng.random(shape) < 0.03, np.round(4 * M), 0.0)
    elif field == "wide":
        M = M * np.exp2(rng.integers(-40, 41, size=shape).astype(np.float64))
    elif field == "special":
        M[(shape[0] // 2, shape[1] // 2, shape[2] // 2) + (0,) * (len(shape) - 3)] = np.inf
        M[(3, 4, 5) + (0,) * (len(shape) - 3)] = np.nan
    elif field == "tiny":
        M = M * 2.0 ** -1015
    elif field == "huge":
        M = M * 2.0 ** 1000
    M = np.asfortranarray(M)
    A, ops = _pair(kind, a, [1.0, 0.5, 2.0] if kind != "curl" else [0.5] * 3, lens)
    k = KINDS[kind][0]
    base = np.asfortranarray(rng.standard_normal(A.out_shape()))
    out, acc = deo.julia_array(A.out_shape(), fill=np.nan), _dev(base)
    Md = _dev(M)
    L.lib().deo_vector_calculus_march_min(A._plan(0), 0)  # the kernel itself, below the sizes that choose it
    A.mul_(out, Md, overwrite=True)
    A.mul_(acc, Md)
    for got, init in ((_host(out), None), (_host(acc), base)):
        ref = O.vector_calculus(k, ops, M, out=None if init is None else np.asfortranarray(init.copy()),
                                overwrite=init is None)
        scale = O.vector_calculus(k, ops, M, absolute=True) + (0 if init is None else np.abs(init))
        fin = np.isfinite(ref)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
        ulp = np.spacing(np.where(np.isfinite(scale), scale, 1.0))[fin]
        err = np.abs(got[fin] - ref[fin])
        assert (err <= 4 * ulp).all(), float((err / ulp).max())
