"""GPU: launches that share a plan's or a batch's claim counters: a captured call
replayed on one stream beside direct calls on another, as many captured calls as there
are counters, and a batch run directly on two streams at once.  Every output is complete,
then and in every later call."""
import gc

import numpy as np
import pytest

import deo

pytestmark = pytest.mark.gpu


def _calls(kind, N=(130, 60, 33)):
    """call(out), its expected result, further outputs"""
    import torch
    torch.manual_seed(1)
    if kind == "gradient":
        A = deo.Gradient(2, (0.1, 0.2, 0.3), N)
        deo._lib.lib().deo_vector_calculus_march_min(A._plan(0), 0)
        M, shape = deo.julia_array(tuple(x + 2 for x in N)), N + (3,)
        run = lambda o: A.mul_(o, M, overwrite=True)
    else:
        G = deo.DiffEqOperatorCombination([deo.CenteredDifference(2, 2, 0.1 * (k + 1), N[k], axis=k + 1) * deo.MultiDimDirectionalBC(
            deo.Dirichlet0BC(), k + 1, N) for k in range(3)])
        p, M, shape = deo.Plan(G.terms(), N, 0), deo.julia_array(N), N
        p.set_option(deo.DEO_OPT_EXACT_SUMS, 1)
        run = {"laplacian": p.apply, "transposed": p.adjoint}.get(kind)
        run = (lambda f: lambda o: f(M, o))(run) if run else None
    M.copy_(torch.randn(M.shape, dtype=M.dtype, device="cuda"))
    outs = [deo.julia_array(shape, fill=np.nan) for _ in range(3)]
    if kind == "batch":
        b = deo.Batch([(p, M, outs[0]), (p, M, outs[1])])  # (both outputs by every run)
        run = lambda o: b.run(use_graph=False)
    return run, outs


@pytest.mark.parametrize("kind", ["laplacian", "transposed", "gradient", "batch"])
def test_replays_beside_direct_calls(cuda, kind):
    import torch
    run, (want, a, b) = _calls(kind)
    torch.cuda.synchronize()
    run(want)
    torch.cuda.synchronize()
    want = want.clone()
    gc.collect()  # (a plan of an earlier test freed during the capture would end it)
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        for _ in range(1024):
            run(a)
    t = torch.cuda.Stream()
    for _ in range(5):
        for o in (a, b):
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            for _ in range(2):
                graph.replay()
        with torch.cuda.stream(t):
            for _ in range(500):
                run(b)
        torch.cuda.synchronize()
        assert torch.equal(a, want) and (kind == "batch" or torch.equal(b, want))
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    o = a if kind == "batch" else b
    for _ in range(1100):
        o.fill_(float("nan"))
        run(o)
        bad += (o != want).any()
    assert int(bad) == 0


def test_one_batch_on_two_streams(cuda):
    import torch
    run, (want, a, _) = _calls("batch", (256, 128, 100))
    torch.cuda.synchronize()
    run(None)
    torch.cuda.synchronize()
    expect = want.clone()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(200):
        for s in streams:
            with torch.cuda.stream(s):
                run(None)
    torch.cuda.synchronize()
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(40):
        for o in (want, a):
            o.fill_(float("nan"))
        run(None)
        bad += (want != expect).any() + (a != expect).any()
    assert int(bad) == 0
