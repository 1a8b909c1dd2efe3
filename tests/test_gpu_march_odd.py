"""GPU: sums of first or third derivatives over three axes (no centre weight) on the
marching kernel, orders 2 to 6, against the oracle at the 4-ulp bar and on the fields
of the Laplacian's tests; and that their points are accepted there: the sum of three
first derivatives takes about the Laplacian's time (nearly four times that while
every point was evaluated again in the reference's order)."""
import numpy as np
import pytest

import deo
import oracle as O
from cases import build, to_device, to_host
from test_gpu_march import ROBIN, _field
from test_gpu_parity import T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["normal", "waves", "sparse", "wide", "special", "tiny", "huge"])
@pytest.mark.parametrize("shape,d,a,one_band", [((64, 16, 20), 1, 4, True), ((65, 17, 13), 1, 2, False), ((33, 24, 11), 1, 6, False),
                                                ((131, 9, 14), 3, 2, True), ((66, 20, 12), 3, 4, False)])
def test_odd_derivatives_against_oracle(cuda, shape, d, a, one_band, field):
    h = [1 / 65.0] * 3 if one_band else [0.1, 0.07, 0.2]
    if field in ("tiny", "huge"):
        h = [1.0] * 3 if one_band else [1.0, 0.5, 2.0]
    A, oterms, _ = build(dict(shape=shape, terms=[T("centered", d, a, axis=k + 1, h=h[k], bc=ROBIN) for k in range(3)], seed=1))
    u = _field(field, shape)
    p = deo.Plan(A.terms(), shape, 0)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)  # the kernel at every size
    out = deo.julia_array(shape, fill=np.nan)
    p.apply(to_device(u), out)
    assert p.kernels[0] == "k_lap_fx"
    got, ref, scale = to_host(out), O.apply(oterms, u), O.abs_scale(oterms, u)
    fin = np.isfinite(ref)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
    err = np.abs(got[fin] - ref[fin]) / np.spacing(scale[fin])
    assert (err <= 4).all(), float(err.max())


def test_first_derivatives_take_the_laplacians_time(cuda):
    import torch
    n = (192,) * 3
    u, out = deo.julia_array(n), deo.julia_array(n)
    u.copy_(torch.sin(torch.arange(192 ** 3, device="cuda", dtype=torch.float64).reshape(n) * 1e-3) + 2)

    def best(d):
        p = deo.Plan(deo.DiffEqOperatorCombination([deo.CenteredDifference(d, 2, 1 / 193, 192, axis=k) * deo.MultiDimDirectionalBC(
            deo.Dirichlet0BC(), k, n) for k in (1, 2, 3)]).terms(), n, 0)
        times = []
        for _ in range(12):
            e = torch.cuda.Event(True), torch.cuda.Event(True)
            e[0].record()
            for _ in range(4):
                p.apply(u, out)
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        return min(times)

    assert best(1) < 2 * best(2)
