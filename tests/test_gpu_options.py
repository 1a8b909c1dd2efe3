"""GPU: what a plan's options report is what its applies do, and the exact-sums option
returned from another variant is the default again."""
import numpy as np
import pytest

import deo
from cases import build, to_device, to_host
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
    want = to_host(out)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)
    p.apply(ud, out)
    assert p.kernels[0] == kernel and np.array_equal(to_host(out), want)


def test_rows_option_given_back(cuda):
    A, _, u = _lap((64, 40, 32), (0.1, 0.1, 0.1))
    p, out = deo.Plan(A.terms(), (64, 40, 32), 0), deo.julia_array((64, 40, 32))
    p.set_option(deo.DEO_OPT_FX_FP64_ROWS, 2)
    assert p.get_option(deo.DEO_OPT_FX_FP64_ROWS) == 2
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 0)
    p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)
    assert p.get_option(deo.DEO_OPT_FX_FP64_ROWS) == 0


def test_tuned_choices_belong_to_the_kernel_they_were_timed_with(cuda, tmp_path):
    A, _, u = _lap((64, 40, 32), (0.1, 0.1, 0.1))
    path = tmp_path / "tuned"
    # a choice stored for the per-point kernel under the key that both kernels once shared
    path.write_text("lap/f64/64x40x32/t3/H1/es1/bc000 0 0 2 0\n")
    p, out, ud = deo.Plan(A.terms(), (64, 40, 32), 0), deo.julia_array((64, 40, 32)), to_device(u)
    p.autotune(ud, out, cache_path=str(path))
    assert any(line.startswith("lap/f64/64x40x32/t3/H1/es1/bc000/march ") for line in path.read_text().splitlines())
