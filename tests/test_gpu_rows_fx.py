"""GPU: 2-D Float64 plans in block fixed point (rows folded to windows with
integer weights) against the oracle at the edges of the 32 x 32 tiles and at
sizes whose last tile overlaps the one before, windows of 3 to 9 points, terms
along one axis or both, an upwind term with a field of both signs and zeros,
every kind of boundary condition, and fields that meet each branch.

Tolerance: 4 ulp of sum|c_k u_k|, the bar of every Float64 path: each axis's sum
is within 2 ulp of its own scale plus a rounding, added as the reference adds its
terms; the oracle's own sums stay below 1.5."""
import numpy as np
import pytest

import deo
import oracle as O
from cases import build, to_device, to_host
from test_gpu_parity import T

pytestmark = pytest.mark.gpu
GEN = ("general", (0.3, 1.0, 0.4), (-0.2, 1.0, 0.6), 1)
ROBIN = ("robin", (1.0, 0.5, 0.0), (1.0, 0.5, 0.0), 1)
NU = dict(grid="nonuniform")
PLANS = {
    "graded-field": [T("centered", 1, 6, axis=1, bc=GEN, **NU), T("centered", 2, 6, axis=2, bc=GEN, **NU),
                     T("upwind", 1, 3, axis=1, coeff="field", bc=GEN, **NU)],
    "x-only": [T("centered", 2, 4, axis=1, bc=ROBIN, **NU)],
    "y-only-wide": [T("centered", 4, 4, axis=2, bc=("dirichlet", 0.5, -0.25), **NU)],
    "field-one-axis": [T("centered", 2, 2, axis=1, bc=("dirichlet0",)),
                       T("upwind", 1, 2, axis=1, coeff="field", bc=("dirichlet0",))],
    "uniform-mixed": [T("centered", 2, 2, axis=1, bc=("periodic",)), T("centered", 1, 2, axis=1, bc=("periodic",)),
                      T("centered", 2, 4, axis=2, bc=("neumann", 0.2, 0.1, 1))],
    "upwind": [T("upwind", 1, 1, axis=2, coeff=-0.7, bc=("dirichlet0",)), T("centered", 2, 2, axis=1, bc=ROBIN)],
}


@pytest.mark.parametrize("field", ["normal", "waves", "zeros", "sparse", "wide", "special", "tiny", "huge"])
@pytest.mark.parametrize("shape", [(32, 32), (33, 40), (65, 100), (100, 63)])
@pytest.mark.parametrize("name", list(PLANS))
def test_rows_against_oracle(cuda, name, shape, field):
    case = dict(shape=shape, terms=PLANS[name], seed=3)
    A, oterms, u = build(case)
    rng = np.random.default_rng(9)
    if field == "waves":
        u = np.sin(0.2 * np.arange(shape[0]))[:, None] * np.exp2(5 * np.sin(np.arange(shape[1]) / 9.0))[None, :] + 1e-4 * u
    elif field == "zeros":
        u[:, shape[1] // 2:] = 0.0
        u[: shape[0] // 3] = 0.0
    elif field == "sparse":  # points that see one small-weight tap, or nothing
        u = np.where(rng.random(shape) < 0.03, np.round(4 * u), 0.0)
    elif field == "wide":
        u = u * np.exp2(rng.integers(-40, 41, size=shape).astype(np.float64))
    elif field == "special":
        u[shape[0] // 2, shape[1] // 2] = np.inf
        u[3, 4] = np.nan
    elif field == "tiny":
        u = u * 2.0 ** -1010
    elif field == "huge":
        u = u * 2.0 ** 960
    u = np.asfortranarray(u)
    p = deo.Plan(A.terms(), shape, 0)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)  # the kernel at every size
    base = np.asfortranarray(rng.standard_normal(shape))
    out, acc = deo.julia_array(shape, fill=np.nan), to_device(base)
    p.apply(to_device(u), out)
    assert p.kernels == ("k_rows_fx",)
    p.apply(to_device(u), acc, overwrite=False)
    got = to_host(out)
    with np.errstate(all="ignore"):
        ref, scale = O.apply(oterms, u), O.abs_scale(oterms, u)
        fin = np.isfinite(ref)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
        ulp = np.spacing(np.where(np.isfinite(scale), scale, 1.0))[fin]
        err = np.abs(got[fin] - ref[fin])
        assert (err <= 4 * ulp).all(), float((err / ulp).max())
        assert np.array_equal(to_host(acc)[fin], (got + base)[fin])
    # the reference's order where it is asked for
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 0)
    p.apply(to_device(u), out)
    assert p.kernels == ("k_apply",)


@pytest.mark.parametrize("a", [2, 4])
@pytest.mark.parametrize("h", [(1 / 1025, 1 / 1025), (1 / 1025, 1 / 513)])
@pytest.mark.parametrize("shape,kernel", [((1024, 512), "k_rows_fx"), ((1023, 512), "k_apply"), ((1025, 513), "k_rows_fx")])
def test_default_2d_laplacian(cuda, shape, kernel, h, a):
    """Laplacian-type plans on each side of the size from which the default apply takes this kernel."""
    case = dict(shape=shape, terms=[T("centered", 2, a, axis=k + 1, h=h[k], bc=ROBIN) for k in range(2)], seed=2)
    A, oterms, u = build(case)
    p = deo.Plan(A.terms(), shape, 0)
    out = deo.julia_array(shape, fill=np.nan)
    p.apply(to_device(u), out)
    assert p.kernels == (kernel,)
    ref, scale = O.apply(oterms, u), O.abs_scale(oterms, u)
    assert (np.abs(to_host(out) - ref) <= 4 * np.spacing(scale)).all()
