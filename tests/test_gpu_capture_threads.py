"""GPU: a plan whose applies use its side stream, called directly on one thread while
another thread captures calls of it: both are complete, and so is the graph."""
import gc
import threading

import numpy as np
import pytest

import deo

pytestmark = pytest.mark.gpu
N = (96, 50, 40)


@pytest.mark.parametrize("kind", ["f64", "f64-three-bands", "f32"])
@pytest.mark.parametrize("call", ["apply", "adjoint"])
def test_direct_calls_during_a_capture(cuda, kind, call):
    import torch
    dt = torch.float32 if kind == "f32" else torch.float64
    h = (0.1, 0.2, 0.3) if kind == "f64-three-bands" else (0.1,) * 3
    A = deo.DiffEqOperatorCombination([deo.CenteredDifference(2, 2, h[k], N[k], axis=k + 1) * deo.MultiDimDirectionalBC(
        deo.Dirichlet0BC(), k + 1, N) for k in range(3)])
    p = deo.Plan(A.terms(), N, 1 if kind == "f32" else 0)
    f = getattr(p, call)
    u, want, a, b = (deo.julia_array(N, dt, fill=np.nan) for _ in range(4))
    torch.manual_seed(4)
    u.copy_(torch.randn(N, dtype=dt, device="cuda"))
    f(u, want)
    torch.cuda.synchronize()
    errors, s, t = [], torch.cuda.Stream(), torch.cuda.Stream()

    def direct():
        try:
            with torch.cuda.stream(t):
                f(u, b)
            t.synchronize()
        except Exception as e:  # (reported by the assertion below)
            errors.append(e)

    gc.collect()  # (a plan of an earlier test freed during the capture would end it)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        f(u, a)
        other = threading.Thread(target=direct)
        other.start()
        other.join()
        f(u, a)
    assert not errors and torch.equal(b, want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(a, want)
    a.fill_(float("nan"))
    f(u, a)
    assert torch.equal(a, want)
