"""GPU: the marching block fixed-point Float64 interior (3-D Laplacian-type
plans, default options) against the oracle: band radii 1-3, one band for the
axes and three, sizes at the edges of its 64 x 8 tiles and below them, odd row
lengths, and fields that meet each of its branches -- exponents that rise and
fall along axis 3, zeros beside values, values far below their block's largest,
Inf/NaN, and scales at the ends of the Float64 range.

Tolerance: 4 ulp of sum|c_k u_k|, the bar of every Float64 path: the kernel's
own bound is 2 ulp plus half an ulp of its rounding, the oracle's sums of 5 to
7 rounded products and 2 additions stay below 1.5."""
import numpy as np
import pytest

import deo
import oracle as O
from cases import build, to_device, to_host
from test_gpu_parity import T

pytestmark = pytest.mark.gpu
ROBIN = ("robin", (1.0, 0.5, 0.0), (1.0, 0.5, 0.0), 1)


def _field(kind, shape):
    rng = np.random.default_rng(5)
    v = rng.standard_normal(shape)
    z = np.arange(shape[2])[None, None, :]
    if kind == "waves":  # the block's exponent rises and falls by several along axis 3; zero crossings
        v = np.sin(0.3 * np.arange(shape[0]))[:, None, None] * np.exp2(6 * np.sin(z / 2.0)) + 1e-3 * v
    elif kind == "zeros":  # a compact support: exact zeros beside values
        v[:, :, shape[2] // 2:] = 0.0
        v[: shape[0] // 3] = 0.0
    elif kind == "sparse":  # points that see one small-weight tap, or nothing
        v = np.where(rng.random(shape) < 0.03, np.round(4 * v), 0.0)
    elif kind == "wide":
        v = v * np.exp2(rng.integers(-40, 41, size=shape).astype(np.float64))
    elif kind == "special":
        v[shape[0] // 2, shape[1] // 2, shape[2] // 2] = np.inf
        v[3, 4, 5] = np.nan
    elif kind == "tiny":  # results near and below the smallest normal
        v = v * 2.0 ** -1015
    elif kind == "huge":
        v = v * 2.0 ** 1005
    return np.asfortranarray(v)


@pytest.mark.parametrize("field", ["normal", "waves", "zeros", "sparse", "wide", "special", "tiny", "huge"])
@pytest.mark.parametrize("shape,a,one_band", [((64, 16, 20), 4, True), ((65, 17, 13), 4, False), ((131, 9, 40), 2, True),
                                              ((33, 24, 11), 6, False), ((130, 31, 12), 6, True), ((12, 11, 9), 2, False)])
def test_march_against_oracle(cuda, shape, a, one_band, field):
    h = [1 / 65.0] * 3 if one_band else [0.1, 0.07, 0.2]
    if field in ("tiny", "huge"):
        h = [1.0] * 3 if one_band else [1.0, 0.5, 2.0]
    case = dict(shape=shape, terms=[T("centered", 2, a, axis=k + 1, h=h[k], bc=ROBIN) for k in range(3)], seed=1)
    A, oterms, _ = build(case)
    u = _field(field, shape)
    p = deo.Plan(A.terms(), shape, 0)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)  # the kernel at every size
    base = np.asfortranarray(np.random.default_rng(6).standard_normal(shape))
    out, acc = deo.julia_array(shape, fill=np.nan), to_device(base)
    p.apply(to_device(u), out)
    assert p.kernels[0] == "k_lap_fx" and p.get_option(deo.DEO_OPT_FX_FP64_ROWS) == 0
    p.apply(to_device(u), acc, overwrite=False)
    got = to_host(out)
    ref, scale = O.apply(oterms, u), O.abs_scale(oterms, u)
    fin = np.isfinite(ref)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
    ulp = np.spacing(np.where(np.isfinite(scale), scale, 1.0))
    assert (np.abs(got - ref)[fin] <= 4 * ulp[fin]).all(), float((np.abs(got - ref)[fin] / ulp[fin]).max())
    assert np.array_equal(to_host(acc)[fin], (got + base)[fin])
    # the same values whatever else runs: a second apply, and one on another stream
    import torch
    s, again = torch.cuda.Stream(), deo.julia_array(shape, fill=np.nan)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        p.apply(to_device(u), again)
    torch.cuda.synchronize()
    assert np.array_equal(to_host(again), got, equal_nan=True)
