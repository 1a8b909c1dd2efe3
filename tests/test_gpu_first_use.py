"""GPU: the first use of a plan or batch on a stream of its own while the default stream
is busy: what the plan puts on the device at creation has to be there.  The result is
compared, bit for bit, with that of the same call when nothing else runs."""
import numpy as np
import pytest

import deo

pytestmark = pytest.mark.gpu


def _busy(torch):
    a = torch.ones(8192, 8192, device="cuda")
    for _ in range(8):
        a = a @ a * 1e-4  # tens of milliseconds on the default stream
    return a


@pytest.mark.parametrize("kind", ["gradient", "laplacian", "batch"])
def test_first_call_on_a_side_stream(cuda, kind):
    import torch
    n = (110, 101, 97)
    torch.manual_seed(3)
    if kind == "gradient":
        M, make = deo.julia_array(tuple(x + 2 for x in n)), lambda: deo.Gradient(2, (0.1, 0.2, 0.3), n)
        out, again = (deo.julia_array(n + (3,), fill=np.nan) for _ in range(2))
        call = lambda A, o: A.mul_(o, M, overwrite=True)
    else:
        M, out, again = deo.julia_array(n), deo.julia_array(n, fill=np.nan), deo.julia_array(n, fill=np.nan)

        def make():
            A = deo.DiffEqOperatorCombination([deo.CenteredDifference(2, 2, 0.1, n[k], axis=k + 1) * deo.MultiDimDirectionalBC(
                deo.Dirichlet0BC(), k + 1, n) for k in range(3)])
            return deo.Plan(A.terms(), n, 0)

        def call(p, o):
            if kind == "laplacian":
                p.apply(M, o)
            else:
                p.batch = deo.Batch([(p, M, o)])
                p.batch.run(use_graph=False)

    M.copy_(torch.randn(M.shape, dtype=M.dtype, device="cuda"))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    keep = _busy(torch)
    with torch.cuda.stream(side):
        A = make()
        call(A, out)
    torch.cuda.synchronize()
    call(A, again)
    torch.cuda.synchronize()
    assert torch.equal(out, again) and torch.isfinite(keep).all()
