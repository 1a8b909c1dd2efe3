"""GPU: the straight tap loops and the single-instance stage, at lines around the
block sizes and barely longer than their boundary rows: applies against the oracle
(4 ulp of sum|w u|, the bar of every Float64 path; the oracle's own sums stay below
1.5), and batches and stages of one and two instances bit for bit against them."""
import numpy as np
import pytest

import deo
import oracle as O
from cases import build
from test_gpu_parity import T

pytestmark = pytest.mark.gpu
GEN = ("general", (0.3, 1.0, 0.4), (-0.2, 1.0, 0.6), 1)
NU = dict(grid="nonuniform")
LINES = {
    "short": lambda ax: T("centered", 1, 2, axis=ax, bc=GEN),
    "long": lambda ax: T("centered", 4, 6, axis=ax, bc=GEN),
    "graded": lambda ax: T("centered", 2, 4, axis=ax, bc=GEN, **NU),
    "graded-long": lambda ax: T("centered", 4, 6, axis=ax, bc=("periodic",), **NU),
    "field": lambda ax: T("upwind", 1, 2, axis=ax, coeff="field", bc=("dirichlet0",)),
    "graded-field": lambda ax: T("centered", 2, 2, axis=ax, coeff="field", bc=GEN, **NU),
}


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(25,), (511,), (513,), (1537,), (24, 25), (40, 33), (24, 25, 26)])
@pytest.mark.parametrize("name", list(LINES))
def test_straight_rows(cuda, name, shape, dtype):
    import torch
    from deo.batch import Batch, StageBatch
    A, oterms, u = build(dict(shape=shape, terms=[LINES[name](ax + 1) for ax in range(len(shape))], seed=5), dtype)
    p = deo.Plan(A.terms(), shape, 0 if dtype == "f64" else 1)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 0)
    p.set_option(deo.DEO_OPT_FAST_PATH, 0)
    td = torch.float64 if dtype == "f64" else torch.float32
    new = lambda: deo.julia_array(shape, td)  # noqa: E731
    c = new().copy_(torch.from_numpy(u))
    a, b = c.flip(0).clone(), torch.ones_like(c)
    a, b = new().copy_(a), new().copy_(b)
    f = new()
    p.apply(c, f)
    if dtype == "f64":
        ref = O.apply(oterms, u)
        tol = O.ulp_tolerance(oterms, u)
        assert (np.abs(f.cpu().numpy() - ref) <= tol).all()
    for adj in (False, True):
        g = new()
        (p.adjoint if adj else p.apply)(c, f)
        Batch([(p, c, g)], adjoint=adj).run(False)
        assert torch.equal(f, g)
        for kw in (dict(gamma=1.0), dict(a=a, alpha=0.75, gamma=0.25), dict(a=a, alpha=0.3, b=b, beta=0.5, gamma=0.2)):
            one, two, three = new(), new(), new()
            st = dict(plan=p, c=c, dt=1e-3, adjoint=adj, **kw)
            StageBatch([dict(st, out=one)]).run(False)
            StageBatch([dict(st, out=two), dict(st, out=three)]).run(False)
            assert torch.equal(one, two) and torch.equal(one, three)
