"""GPU: what a plan's options report is what its applies do."""
import pytest

import deo
from cases import build, to_device
from test_gpu_parity import T

pytestmark = pytest.mark.gpu
ROBIN = ("robin", (1.0, 0.5, 0.0), (1.0, 0.5, 0.0), 1)


def _lap(shape, h):
    return build(dict(shape=shape, terms=[T("centered", 2, 2, axis=k + 1, h=h[k], bc=ROBIN) for k in range(len(shape))], seed=1))


@pytest.mark.parametrize("shape,h,sums,concurrent,kernel", [
    ((64, 40, 32), (0.1, 0.1, 0.1), 1, 1, "k_lap_fx"), ((64, 40, 32), (0.1, 0.2, 0.3), 1, 1, "k_lap_fx"),
    ((65, 40, 32), (0.1, 0.2, 0.3), 0, 0, "k_apply"), ((1024, 512), (0.001, 0.002), 1, 0, "k_rows_fx"),
    ((1024, 512), (0.001, 0.001), 1, 0, "k_rows_fx"), ((100, 60), (0.01, 0.02), 0, 0, "k_apply")])
def test_what_applies_is_reported(cuda, shape, h, sums, concurrent, kernel):
    A, _, u = _lap(shape, h)
    p, out = deo.Plan(A.terms(), shape, 0), deo.julia_array(shape)
    ud = to_device(u)
    p.apply(ud, out)
    assert p.kernels[0] == kernel
    assert p.get_option(deo.DEO_OPT_EXACT_SUMS) == sums and p.get_option(deo.DEO_OPT_CONCURRENT_SHELL) == concurrent
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 0)
    assert p.get_option(deo.DEO_OPT_EXACT_SUMS) == 0
