"""GPU: when the rows of the 2-D block fixed-point kernel are built: with plans that take
it by themselves (also with more rows than are kept while building), and on request with
smaller ones, whose operators may be gone by then; not before."""
import gc

import numpy as np
import pytest

import deo
import oracle as O
from cases import build, to_device, to_host
from test_gpu_rows_fx import PLANS
from test_gpu_parity import T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(PLANS))
def test_built_on_request(cuda, name):
    A, oterms, u = build(dict(shape=(65, 100), terms=PLANS[name], seed=3))
    p = deo.Plan(A.terms(), (65, 100), 0)
    before = p.table_bytes()
    del A
    gc.collect()
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)
    assert p.table_bytes() > before
    out = deo.julia_array((65, 100), fill=np.nan)
    p.apply(to_device(u), out)
    assert p.kernels == ("k_rows_fx",)
    assert (np.abs(to_host(out) - O.apply(oterms, u)) <= 4 * np.spacing(O.abs_scale(oterms, u))).all()


@pytest.mark.parametrize("shape", [(65600, 33), (33, 65601)])
def test_long_axes(cuda, shape):
    terms = [T("centered", 1, 4, axis=1, bc=("robin", (1.0, 0.5, 0.0), (1.0, 0.5, 0.0), 1), grid="nonuniform"),
             T("centered", 2, 2, axis=2, bc=("dirichlet0",)), T("upwind", 1, 2, axis=1, coeff="field", bc=("dirichlet0",))]
    A, oterms, u = build(dict(shape=shape, terms=terms, seed=4))
    p, out = deo.Plan(A.terms(), shape, 0), deo.julia_array(shape, fill=np.nan)
    p.apply(to_device(u), out)
    assert p.kernels == ("k_rows_fx",)
    assert (np.abs(to_host(out) - O.apply(oterms, u)) <= 4 * np.spacing(O.abs_scale(oterms, u))).all()
