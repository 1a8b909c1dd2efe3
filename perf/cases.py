"""The performance cases: calls that a user of the framework makes, each through its public entry
points, with the sizes of the benchmark's configurations, of the tests, and of the odd grids between them.

  line     du = (L*Q)*u on a vector (method-of-lines right-hand sides of 1-D problems)
  lap      mul!(du, Dxx + Dyy [+ Dzz], u) with a boundary condition on every face
  grad     the same apply under reverse-mode differentiation: the value and the pullback
  graded   the sum of first and second derivatives on a graded 2-D grid with an upwind term whose
           coefficient is a field
  batch    many small independent problems, one pass forward and one transposed
  mol      fixed SSP-RK3 steps of an advection-diffusion problem
  solve    A \\ u along one axis (an implicit step)
  vector   gradient, divergence or curl of a padded array
  nld      nonlinear_diffusion! on a long line

`exact` restates the operators (finite-difference weights, boundary rows, ghost maps) in numpy and
applies them with torch in Float64.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "diffeqoperators.jl_gb300"))
import deo  # noqa: E402


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the right-hand side of a small 1-D heat equation: one short launch, called in a time loop
        dict(name="line_1024_f64", kind="line", n=1024, d=2, a=2, graded=False, dtype="f64"),
        # the headline: the 3-D Laplacian of the benchmark, RobinBC on every face
        dict(name="lap_256_f64", kind="lap", nx=256, ny=256, nz=256, a=4, bc="robin", dtype="f64"),
        # a 3-D grid whose sides are odd (2^k + 1 nodes and the like)
        dict(name="lap_ragged_f64", kind="lap", nx=193, ny=129, nz=101, a=4, bc="robin", dtype="f64"),
        # the same Laplacian in Float32
        dict(name="lap_256_f32", kind="lap", nx=256, ny=256, nz=256, a=4, bc="robin", dtype="f32"),
        # a loss gradient through the right-hand side, on an ordinary grid
        dict(name="grad_lap_f64", kind="grad", nx=160, ny=128, nz=96, a=4, bc="robin", dtype="f64"),
        # the benchmark's graded grid: four centred operators and an upwind one with a field
        dict(name="graded_2048_f64", kind="graded", nx=2048, ny=2048, dtype="f64"),
        # the benchmark's mixed batch (1-D and 2-D, orders 1-4 and 2-8), forward and transposed
        dict(name="batch_256_f64", kind="batch", count=256, scale=1.0),
        # a method-of-lines solve of the serving workload's 2-D kind
        dict(name="mol_768x500_f64", kind="mol", nx=768, ny=500, nz=1, steps=12),
        # an implicit step along the slowest axis: tridiagonal lines
        dict(name="solve_256_f64", kind="solve", nx=256, ny=256, nz=256, axis=3, a=2, dtype="f64"),
        # the gradient of a scalar field, and the curl of a Float32 field with an odd side
        dict(name="gradient_256_f64", kind="vector", op="gradient", nx=256, ny=256, nz=256, a=4, dtype="f64"),
        dict(name="curl_127_f32", kind="vector", op="curl", nx=127, ny=127, nz=127, a=4, dtype="f32"),
        # nonlinear diffusion on a long line
        dict(name="nld_4m_f64", kind="nld", n=(1 << 22) - 5, a=4, dtype="f64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, nd, lo, hi, cap):
    while True:
        s = [_log(rng, lo, hi) for _ in range(nd)]
        if math.prod(s) <= cap:
            return s + [1] * (3 - nd)


def draw(rng):
    kind = rng.choice(["line", "lap", "lap", "lap", "grad", "graded", "batch", "mol", "solve", "vector", "vector", "nld"])
    dtype = rng.choice(["f64", "f64", "f32"])
    if kind == "line":
        return dict(kind=kind, n=_log(rng, 256, 1 << 20), d=rng.randint(1, 4), a=rng.choice([2, 4, 6, 8]),
                    graded=rng.random() < 0.5, dtype=dtype)
    if kind in ("lap", "grad"):
        nd = rng.choice([2, 3, 3])
        nx, ny, nz = _sides(rng, nd, 32 if nd == 3 else 100, 300 if nd == 3 else 4096, 1 << 24)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, a=rng.choice([2, 4]),
                    bc=rng.choice(["robin", "dirichlet0", "periodic"]), dtype=dtype if kind == "lap" else "f64")
    if kind == "graded":
        nx, ny, _ = _sides(rng, 2, 200, 2500, 1 << 22)
        return dict(kind=kind, nx=nx, ny=ny, dtype="f64")
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(32, 256), scale=rng.choice([0.25, 0.5, 1.0]))
    if kind == "mol":
        nd = rng.choice([1, 2, 3])
        nx, ny, nz = _sides(rng, nd, {1: 1000, 2: 100, 3: 32}[nd], {1: 200000, 2: 900, 3: 90}[nd], 400000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randint(4, 12))
    if kind == "solve":
        nx, ny, nz = _sides(rng, 3, 32, 300, 1 << 24)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, axis=rng.choice([2, 3]), a=rng.choice([2, 4]), dtype=dtype)
    if kind == "vector":
        op = rng.choice(["gradient", "divergence", "curl"])
        nx, ny, nz = _sides(rng, 3, 32, 300, 1 << 23)
        if op == "curl":
            nx = ny = nz = _log(rng, 32, 190)
        return dict(kind=kind, op=op, nx=nx, ny=ny, nz=nz, a=rng.choice([2, 4, 6]), dtype=dtype)
    return dict(kind=kind, n=_log(rng, 1 << 14, 1 << 22), a=rng.choice([2, 4]), dtype=dtype)


# ---------------------------------------------------------------------------
# inputs and plans
# ---------------------------------------------------------------------------
ROBIN = ((1.0, 0.5, 0.0), (1.0, 0.5, 0.0))
BATCH_ROBIN, BATCH_DIRICHLET = ((1.0, 0.5, 0.1), (1.0, 0.5, -0.1)), (0.1, -0.2)


def _shape(c):
    s = (c["nx"], c["ny"]) + ((c["nz"],) if c.get("nz", 1) > 1 else ())
    return s[:1] if len(s) == 2 and s[1] == 1 else s


def _dtype(c):
    return torch.float32 if c.get("dtype") == "f32" else torch.float64


def _julia(x, dtype=None):
    """A column-major (axis 1 contiguous) copy of x."""
    t = deo.julia_array(tuple(x.shape), dtype or x.dtype, x.device)
    return t.copy_(x)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _smooth(shape, seed, noise=1e-3):
    """A sum of 8 Fourier modes per axis with amplitudes in (-1, 1), and white noise."""
    g = _gen(seed)
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for ax, n in enumerate(shape):
        x = torch.arange(1, n + 1, device="cuda", dtype=torch.float64) / (n + 1)
        k = torch.arange(1, 9, device="cuda", dtype=torch.float64) * math.pi
        ab = torch.rand((2, 8), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        f = (ab[0] * torch.sin(k * x[:, None]) + ab[1] * torch.cos(k * x[:, None])).sum(1)
        out += f.reshape([n if a == ax else 1 for a in range(len(shape))])
    return out + noise * torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def _graded_dx(n):
    """Grid spacings h(1 + 0.5 sin(2 pi i / (n + 1))) of the unit interval."""
    dx = 1.0 + 0.5 * np.sin(2 * np.pi * np.arange(n + 1) / (n + 1))
    return dx / dx.sum()


def _deo_bc(kind, dx):
    return {"robin": lambda: deo.RobinBC(*ROBIN, dx, 1), "dirichlet0": deo.Dirichlet0BC, "periodic": deo.PeriodicBC}[kind]()


def _laplacian(shape, a, bc):
    ops = []
    for ax, n in enumerate(shape):
        h = 1.0 / (n + 1)
        ops.append(deo.CenteredDifference(2, a, h, n, axis=ax + 1) *
                   deo.MultiDimDirectionalBC(_deo_bc(bc, h), ax + 1, shape))
    return deo.DiffEqOperatorCombination(ops)


def _graded_inputs(c, seed):
    """u: normal values smoothed by 5 Jacobi passes; the field cos(2 pi x) sin(2 pi y); the ghost coefficients."""
    nx, ny = c["nx"], c["ny"]
    u = torch.randn((nx, ny), generator=_gen(seed), device="cuda", dtype=torch.float64)
    for _ in range(5):
        v = u.clone()
        v[1:-1, 1:-1] = 0.25 * (u[:-2, 1:-1] + u[2:, 1:-1] + u[1:-1, :-2] + u[1:-1, 2:])
        u = v
    dxs = [_graded_dx(n) for n in (nx, ny)]
    x, y = (torch.from_numpy(np.cumsum(d)[:-1]).cuda() for d in dxs)
    f = torch.cos(2 * math.pi * x)[:, None] * torch.sin(2 * math.pi * y)[None, :]
    rng = np.random.default_rng(20251210)
    al, ar = rng.uniform(-1, 1, 3), rng.uniform(-1, 1, 3)
    al[1], ar[1] = abs(al[1]) + 0.5, abs(ar[1]) + 0.5
    return u, f, dxs, al, ar


def _batch_specs(c):
    """(shape, d, a, graded, robin): 70 % lines of 64 to 65536 points, 30 % planes of sides 32 to 1024."""
    rng = np.random.default_rng(20251203)
    out = []
    for _ in range(c["count"]):
        d, a = int(rng.integers(1, 5)), int(rng.choice([2, 4, 6, 8]))
        graded, robin = rng.random() < 0.5, rng.random() < 0.5
        side = lambda lo, hi: max(16, int(np.exp(rng.uniform(np.log(lo), np.log(hi))) * c["scale"]))  # noqa: E731
        shape = (side(64, 65536),) if rng.random() < 0.7 else (side(32, 1024), side(32, 1024))
        out.append((shape, d, a, graded, robin))
    return out


def _mol_params(c):
    nu, adv = 0.05, 0.6
    shape = _shape(c)
    h = 1.0 / (shape[0] + 1)
    hm = 1.0 / (max(shape) + 1)
    return nu, adv, 0.4 * min(h / adv, hm * hm / (2.0 * nu * len(shape)))


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "line":
        n = c["n"]
        dx = _graded_dx(n) if c["graded"] else 1.0 / (n + 1)
        x = torch.arange(1, n + 1, device="cuda", dtype=torch.float64) / (n + 1)
        u = (torch.sin(2 * math.pi * x) + 0.01 * torch.randn(n, generator=_gen(seed), device="cuda", dtype=torch.float64))
        u = u.to(_dtype(c))
        A = deo.CenteredDifference(c["d"], c["a"], dx, n) * deo.Dirichlet0BC(np.float64)
        deo.plan_for(A.terms(), (n,), 0 if c["dtype"] == "f64" else 1)
        return dict(kind=k, A=A, u=u, du=torch.empty_like(u))
    if k in ("lap", "grad"):
        shape = _shape(c)
        u = _julia(_smooth(shape, seed), _dtype(c))
        A = _laplacian(shape, c["a"], c["bc"])
        deo.plan_for(A.terms(), shape, 0 if c["dtype"] == "f64" else 1)
        s = dict(kind=k, A=A, u=u, du=deo.julia_array(shape, _dtype(c)))
        if k == "grad":
            s["u"].requires_grad_(True)
            s["v"] = _julia(torch.randn(shape, generator=_gen(seed + 1), device="cuda", dtype=torch.float64), _dtype(c))
        return s
    if k == "graded":
        u, f, dxs, al, ar = _graded_inputs(c, seed)
        shape = (c["nx"], c["ny"])
        q = [deo.MultiDimDirectionalBC(deo.GeneralBC(al, ar, dxs[i], 1), i + 1, shape) for i in range(2)]
        ops = [deo.CenteredDifference(d, 6, dxs[i], shape[i], axis=i + 1) * q[i] for d in (1, 2) for i in range(2)]
        ops.append(deo.with_field(deo.UpwindDifference(1, 3, dxs[0], shape[0], axis=1), _julia(f)) * q[0])
        A = deo.DiffEqOperatorCombination(ops)
        deo.plan_for(A.terms(), shape, 0)
        return dict(kind=k, A=A, u=_julia(u), du=deo.julia_array(shape))
    if k == "batch":
        specs = _batch_specs(c)
        sizes = [math.prod(s[0]) for s in specs]
        offs = np.concatenate([[0], np.cumsum([(n + 1) // 2 * 2 for n in sizes])])
        u = torch.randn(int(offs[-1]), generator=_gen(seed), device="cuda", dtype=torch.float64)
        f, b = torch.zeros_like(u), torch.zeros_like(u)
        fwd, adj = [], []
        for (shape, d, a, graded, robin), o, n in zip(specs, offs, sizes):
            terms = []
            for ax, m in enumerate(shape):
                dx = _graded_dx(m) if graded else 1.0 / (m + 1)
                bc = deo.RobinBC(*BATCH_ROBIN, dx, 1) if robin else deo.DirichletBC(*BATCH_DIRICHLET)
                L = deo.CenteredDifference(d, a, dx, m, axis=ax + 1)
                terms.append(L * (bc if len(shape) == 1 else deo.MultiDimDirectionalBC(bc, ax + 1, shape)))
            p = deo.Plan(terms, shape, 0)
            view = lambda t: t[int(o):int(o) + n].as_strided(shape, deo.fortran_strides(shape))  # noqa: E731
            fwd.append((p, view(u), view(f)))
            adj.append((p, view(f), view(b)))
        return dict(kind=k, fwd=deo.Batch(fwd), adj=deo.Batch(adj, adjoint=True), u=u, f=f, b=b)
    if k == "mol":
        shape = _shape(c)
        nu, adv, dt = _mol_params(c)
        u = _julia(_smooth(shape, seed, 0.0)) if len(shape) > 1 else _smooth(shape, seed, 0.0)
        bc = deo.Dirichlet0BC()
        ops = [nu * deo.CenteredDifference(2, 2, 1.0 / (n + 1), n, axis=i + 1) for i, n in enumerate(shape)]
        ops.append(deo.UpwindDifference(1, 2, 1.0 / (shape[0] + 1), shape[0], -adv, axis=1))
        A = deo.DiffEqOperatorCombination(
            [L * (bc if len(shape) == 1 else deo.MultiDimDirectionalBC(bc, L.axis, shape)) for L in ops])
        deo.plan_for(A.terms(), shape, 0)
        return dict(kind=k, A=A, u=u, dt=dt, steps=c["steps"])
    if k == "solve":
        shape = _shape(c)
        n, ax = shape[c["axis"] - 1], c["axis"]
        h = 1.0 / (n + 1)
        A = deo.CenteredDifference(2, c["a"], h, n, axis=ax) * deo.MultiDimBC(deo.RobinBC(*ROBIN, h, c["a"]), shape, ax)
        u = _julia(torch.randn(shape, generator=_gen(seed), device="cuda", dtype=torch.float64), _dtype(c))
        deo.solve_plan_for(A, shape, 0 if c["dtype"] == "f64" else 1)
        return dict(kind=k, A=A, u=u, x=deo.julia_array(shape, _dtype(c)))
    if k == "vector":
        shape = _shape(c)
        A = {"gradient": deo.Gradient, "divergence": deo.Divergence, "curl": deo.Curl}[c["op"]](
            c["a"], tuple(1.0 / (n + 1) for n in shape), shape)
        M = deo.julia_array(A.in_shape(), _dtype(c))
        M.copy_(_vector_input(c, seed))
        out = deo.julia_array(A.out_shape(), _dtype(c))
        A.mul_(out, M, overwrite=True)  # builds the operator's plan
        return dict(kind=k, A=A, M=M, out=out)
    if k == "nld":
        p, q = (t.to(_dtype(c)) for t in _nld_input(c, seed))
        du = torch.empty(c["n"], device="cuda", dtype=_dtype(c))
        deo.nonlinear_diffusion_(du, 2, 1, c["a"], p, q, 1.0 / (c["n"] + 1), c["n"])  # builds the plan
        return dict(kind=k, p=p, q=q, du=du, n=c["n"], a=c["a"])
    raise ValueError(k)


def _vector_input(c, seed):
    padded = tuple(n + 2 for n in _shape(c))
    if c["op"] == "gradient":
        return _smooth(padded, seed)
    return torch.stack([_smooth(padded, 3 * seed + i) for i in range(3)], dim=-1)


def _nld_input(c, seed):
    x = torch.linspace(0, 1, c["n"] + 2, device="cuda", dtype=torch.float64)
    g = _gen(seed)
    ph = torch.rand(2, generator=g, device="cuda", dtype=torch.float64)
    q = torch.sin(2 * math.pi * (x + ph[0])) + 1e-3 * torch.randn(c["n"] + 2, generator=g, device="cuda",
                                                                 dtype=torch.float64)
    return 1.0 + 0.5 * torch.cos(2 * math.pi * (x + ph[1])), q


def run(s):
    k = s["kind"]
    if k in ("line", "lap", "graded"):
        return deo.mul_(s["du"], s["A"], s["u"])
    if k == "grad":
        y = deo.autodiff.apply(s["A"], s["u"])
        (g,) = torch.autograd.grad(y, s["u"], s["v"])
        return [y.detach(), g]
    if k == "batch":
        s["fwd"].run(True)
        s["adj"].run(True)
        return [s["f"], s["b"]]
    if k == "mol":
        return deo.autodiff.ssprk3_solve(s["A"], s["u"], s["dt"], s["steps"])
    if k == "solve":
        return deo.ldiv_(s["x"], s["A"], s["u"])
    if k == "vector":
        return s["A"].mul_(s["out"], s["M"], overwrite=True)
    return deo.nonlinear_diffusion_(s["du"], 2, 1, s["a"], s["p"], s["q"], 1.0 / (s["n"] + 1), s["n"])


def work(case):
    c, k = case, case["kind"]
    es = 4 if c.get("dtype") == "f32" else 8
    if k == "line":
        return {"bytes": 2 * es * c["n"], "flops": 2 * (c["d"] + c["a"]) * c["n"]}
    if k == "batch":
        specs = _batch_specs(c)
        pts = sum(math.prod(s[0]) for s in specs)
        fl = sum(4 * (s[1] + s[2]) * len(s[0]) * math.prod(s[0]) for s in specs)
        return {"bytes": 4 * es * pts, "flops": fl}
    if k == "nld":
        return {"bytes": 3 * es * c["n"], "flops": 2 * (5 * c["a"] + 10) * c["n"]}
    shape = _shape(c)
    pts, nd = math.prod(shape), len(shape)
    if k == "lap":
        return {"bytes": 2 * es * pts, "flops": 2 * nd * (c["a"] + 1) * pts}
    if k == "grad":
        return {"bytes": 4 * es * pts, "flops": 4 * nd * (c["a"] + 1) * pts}
    if k == "graded":
        return {"bytes": 3 * es * pts, "flops": 2 * 34 * pts}
    if k == "mol":  # the state in and out once
        return {"bytes": 2 * es * pts, "flops": 3 * c["steps"] * (6 * nd + 12) * pts}
    if k == "solve":
        return {"bytes": 2 * es * pts, "flops": 4 * c["a"] * pts}
    nin, nout, nder = {"gradient": (1, 3, 3), "divergence": (3, 1, 3), "curl": (3, 3, 6)}[c["op"]]
    return {"bytes": es * (nin * math.prod(n + 2 for n in shape) + nout * pts), "flops": 2 * nder * (c["a"] + 1) * pts}


# ---------------------------------------------------------------------------
# the same results in plain numpy / torch, Float64
# ---------------------------------------------------------------------------
def _weights(m, x0, x):
    """Finite-difference weights of the m-th derivative at x0 on the points x (Fornberg 1988), the
    middle weight corrected by the residue of their sum."""
    n = len(x)
    C = np.zeros((n, m + 1))
    C[0, 0] = 1.0
    c1, c4 = 1.0, x[0] - x0
    for i in range(1, n):
        mn = min(i, m)
        c2, c5 = 1.0, c4
        c4 = x[i] - x0
        for j in range(i):
            c3 = x[i] - x[j]
            c2 *= c3
            if j == i - 1:
                for s in range(mn, 0, -1):
                    C[i, s] = c1 * (s * C[i - 1, s - 1] - c5 * C[i - 1, s]) / c2
                C[i, 0] = -c1 * c5 * C[i - 1, 0] / c2
            for s in range(mn, 0, -1):
                C[j, s] = (c4 * C[j, s] - s * C[j, s - 1]) / c3
            C[j, 0] = c4 * C[j, 0] / c3
        c1 = c2
    w = C[:, m].copy()
    if m:
        w[n // 2] -= w.sum()
    return w


def _weight_rows(m, x0, X):
    """_weights for many rows at once: X (rows, points), x0 (rows)."""
    R, n = X.shape
    C = np.zeros((R, n, m + 1))
    C[:, 0, 0] = 1.0
    c1, c4 = np.ones(R), X[:, 0] - x0
    for i in range(1, n):
        mn = min(i, m)
        c2, c5 = np.ones(R), c4
        c4 = X[:, i] - x0
        for j in range(i):
            c3 = X[:, i] - X[:, j]
            c2 = c2 * c3
            if j == i - 1:
                for s in range(mn, 0, -1):
                    C[:, i, s] = c1 * (s * C[:, i - 1, s - 1] - c5 * C[:, i - 1, s]) / c2
                C[:, i, 0] = -c1 * c5 * C[:, i - 1, 0] / c2
            for s in range(mn, 0, -1):
                C[:, j, s] = (c4 * C[:, j, s] - s * C[:, j, s - 1]) / c3
            C[:, j, 0] = c4 * C[:, j, 0] / c3
        c1 = c2
    w = C[:, :, m].copy()
    if m:
        w[:, n // 2] -= w.sum(1)
    return w


def _centered(d, a, dx, n):
    """(first padded position, weights) of every row of CenteredDifference(d, a, dx, n) over the padded line."""
    st, bs = d + a - 1 + (d + a) % 2, d + a
    bpc = st // 2 - 1
    K = max(st, bs)
    i = np.arange(n)
    p0 = np.where(i < bpc, 0, np.where(i < n - bpc, i + 1 - st // 2, n + 2 - bs))
    W = np.zeros((n, K))
    inner = (i >= bpc) & (i < n - bpc)
    x = np.arange(n + 2) / (n + 1.0) if np.isscalar(dx) else np.concatenate([[0.0], np.cumsum(dx)])
    if np.isscalar(dx):
        s = float(dx) ** -d
        W[inner, :st] = s * _weights(d, 0.0, np.arange(-(st // 2), st // 2 + 1.0))
        for r in range(bpc):
            low = s * _weights(d, r + 1.0, np.arange(float(bs)))
            W[r, :bs] = low
            W[n - 1 - r, :bs] = (-1) ** d * low[::-1]
    else:
        rows = i[inner]
        X = x[(p0[inner])[:, None] + np.arange(st)] - x[rows + 1][:, None]
        W[inner, :st] = _weight_rows(d, np.zeros(len(rows)), X)
        for r in range(bpc):
            W[r, :bs] = _weights(d, x[r + 1], x[:bs])
            hx = x[n + 2 - bs:] - x[n + 2 - bs]
            W[n - 1 - r, :bs] = _weights(d, hx[bs - 2 - r], hx)
    return p0, W


def _upwind_rows(d, a, dx, n, sign):
    """The rows of UpwindDifference(d, a, dx, n) for coefficients of one sign (no offside points)."""
    st = d + a
    bpc = st - 2
    x = np.arange(n + 2) * float(dx) if np.isscalar(dx) else np.concatenate([[0.0], np.cumsum(dx)])
    i = np.arange(n)
    if sign > 0:
        p0 = np.where(i + 1 + st <= n + 2, i + 1, n + 2 - st)
    else:
        p0 = np.where(i < bpc, 0, i + 2 - st)
    p0 = np.clip(p0, 0, n + 2 - st)
    X = x[p0[:, None] + np.arange(st)]
    return p0, _weight_rows(d, x[i + 1], X)


def _ghosts(bc, dx, n):
    """(a_l, b_l, a_r, b_r): the ghost values a . u + b from the points nearest each end; None: the edge planes."""
    if bc == "periodic":
        return None
    if bc == "dirichlet0":
        return np.zeros(1), 0.0, np.zeros(1), 0.0
    if bc[0] == "dirichlet":
        return np.zeros(1), bc[1], np.zeros(1), bc[2]
    dl, dr = (dx, dx) if np.isscalar(dx) else (dx, dx[::-1])
    if bc[0] == "robin":
        (l0, l1, l2), (r0, r1, r2), order = bc[1], bc[2], bc[3]
        s = _weights(1, 1.0, np.arange(1.0, order + 2))
        at = lambda v, k: v if np.isscalar(v) else v[k]  # noqa: E731
        den_l, den_r = l0 + l1 * s[0] / at(dl, 0), r0 - r1 * s[0] / at(dr, 0)
        a_l = np.array([-l1 * s[1 + k] / (den_l * at(dl, 1 + k)) for k in range(order)])
        a_r = np.array([r1 * s[1 + k] / (den_r * at(dr, 1 + k)) for k in range(order)])[::-1]
        return a_l, l2 / den_l, a_r, r2 / den_r
    al, ar = bc[1], bc[2]  # ("general", al, ar): three coefficients a side, order 1
    w = _weights(1, 1.0, np.array([1.0, 2.0]))
    sl = w / dl[:2]
    wr = _weights(1, 2.0, np.array([1.0, 2.0]))
    sr = wr / np.array([dr[0], dr[1]])
    den_l, den_r = al[1] + al[2] * sl[0], ar[1] + ar[2] * sr[1]
    return np.array([-al[2] * sl[1] / den_l]), -al[0] / den_l, np.array([-ar[2] * sr[0] / den_r]), -ar[0] / den_r


def _pad(u, ax, g):
    n = u.shape[ax]
    if g is None:
        if u.dim() == 1:
            return torch.cat([u[-1:], u, u[:1]])
        return torch.cat([u.narrow(ax, 0, 1), u, u.narrow(ax, n - 1, 1)], dim=ax)
    a_l, b_l, a_r, b_r = g
    lo = sum(float(w) * u.narrow(ax, k, 1) for k, w in enumerate(a_l)) + b_l
    hi = sum(float(w) * u.narrow(ax, n - len(a_r) + k, 1) for k, w in enumerate(a_r)) + b_r
    return torch.cat([lo, u, hi], dim=ax)


def _rows_apply(x, ax, p0, W):
    """sum_k W[i, k] x[p0[i] + k] along axis ax of the padded array x."""
    n, K = W.shape
    at = torch.from_numpy(np.ascontiguousarray(p0)).cuda()
    Wd = torch.from_numpy(np.ascontiguousarray(W)).cuda()
    shape = [n if a == ax else 1 for a in range(x.dim())]
    out = None
    for k in range(K):
        t = Wd[:, k].reshape(shape) * x.index_select(ax, torch.clamp(at + k, max=x.shape[ax] - 1))
        out = t if out is None else out + t
    return out


def _term(u, ax, rows, g):
    return _rows_apply(_pad(u, ax, g), ax, *rows)


def _lap_exact(u, c):
    out = 0.0
    for ax, n in enumerate(u.shape):
        h = 1.0 / (n + 1)
        bc = ("robin", *ROBIN, 1) if c["bc"] == "robin" else c["bc"]
        out = out + _term(u, ax, _centered(2, c["a"], h, n), _ghosts(bc, h, n))
    return out


def exact(case, seed):
    c, k = case, case["kind"]
    s = prepare(case, seed) if k not in ("batch",) else None
    if k == "line":
        n = c["n"]
        dx = _graded_dx(n) if c["graded"] else 1.0 / (n + 1)
        return _term(s["u"].double(), 0, _centered(c["d"], c["a"], dx, n), _ghosts("dirichlet0", dx, n))
    if k == "lap":
        return _lap_exact(s["u"].double(), c)
    if k == "grad":
        u = s["u"].detach().double().requires_grad_(True)
        y = _lap_exact(u, c)
        (g,) = torch.autograd.grad(y, u, s["v"].double())
        return [y.detach(), g]
    if k == "graded":
        u, f, dxs, al, ar = _graded_inputs(c, seed)
        g = [_ghosts(("general", al, ar), dxs[i], u.shape[i]) for i in range(2)]
        out = 0.0
        for d in (1, 2):
            for i in range(2):
                out = out + _term(u, i, _centered(d, 6, dxs[i], u.shape[i]), g[i])
        up, dn = (_term(u, 0, _upwind_rows(1, 3, dxs[0], u.shape[0], sg), g[0]) for sg in (1, -1))
        return out + f * torch.where(f >= 0, up, dn)
    if k == "batch":
        specs = _batch_specs(c)
        sizes = [math.prod(sp[0]) for sp in specs]
        offs = np.concatenate([[0], np.cumsum([(n + 1) // 2 * 2 for n in sizes])])
        uf = torch.randn(int(offs[-1]), generator=_gen(seed), device="cuda", dtype=torch.float64)
        f, b = torch.zeros_like(uf), torch.zeros_like(uf)
        for (shape, d, a, graded, robin), o, n in zip(specs, offs, sizes):
            flat = uf[int(o):int(o) + n].clone().requires_grad_(True)
            u = flat.reshape(tuple(reversed(shape))).permute(*reversed(range(len(shape))))
            y = 0.0
            for ax, m in enumerate(shape):
                dx = _graded_dx(m) if graded else 1.0 / (m + 1)
                bc = ("robin", *BATCH_ROBIN, 1) if robin else ("dirichlet", *BATCH_DIRICHLET)
                y = y + _term(u, ax, _centered(d, a, dx, m), _ghosts(bc, dx, m))
            (g,) = torch.autograd.grad(y, flat, y.detach())
            f[int(o):int(o) + n] = y.detach().permute(*reversed(range(len(shape)))).reshape(-1)
            b[int(o):int(o) + n] = g
        return [f, b]
    if k == "mol":
        nu, adv, dt = _mol_params(c)
        u = s["u"]
        terms = [(i, (lambda r: (r[0], nu * r[1]))(_centered(2, 2, 1.0 / (n + 1), n)), _ghosts("dirichlet0", 0.0, n))
                 for i, n in enumerate(u.shape)]
        n = u.shape[0]
        p0, W = _upwind_rows(1, 2, 1.0 / (n + 1), n, -1)
        terms.append((0, (p0, -adv * W), _ghosts("dirichlet0", 0.0, n)))
        F = lambda v: sum(_term(v, *t) for t in terms)  # noqa: E731
        for _ in range(c["steps"]):
            u1 = u + dt * F(u)
            u2 = 0.75 * u + 0.25 * (u1 + dt * F(u1))
            u = u / 3.0 + (2.0 / 3.0) * (u2 + dt * F(u2))
        return u
    if k == "solve":
        ax, u = c["axis"] - 1, s["u"].double()
        n = u.shape[ax]
        h = 1.0 / (n + 1)
        rows, g = _centered(2, c["a"], h, n), _ghosts(("robin", *ROBIN, c["a"]), h, n)
        off = _term(torch.zeros(n, dtype=torch.float64, device="cuda"), 0, rows, g)
        eye = torch.eye(n, dtype=torch.float64, device="cuda")
        Al = _term(eye, 0, rows, g) - off[:, None]
        b = u.movedim(ax, 0)
        x = torch.linalg.solve(Al, b.reshape(n, -1) - off[:, None])
        return x.reshape(b.shape).movedim(0, ax)
    if k == "vector":
        M, shape = s["M"].double(), _shape(c)
        rows = [_centered(1, c["a"], 1.0 / (n + 1), n) for n in shape]

        def D(x, a):  # along a on the padded line, the other axes at the output's own index
            for b in range(3):
                if b != a:
                    x = x.narrow(b, 0, shape[b])
            return _rows_apply(x, a, *rows[a])
        if c["op"] == "gradient":
            return torch.stack([D(M, a) for a in range(3)], dim=-1)
        if c["op"] == "divergence":
            return sum(D(M[..., a], a) for a in range(3))
        return torch.stack([D(M[..., 2], 1) - D(M[..., 1], 2), D(M[..., 0], 2) - D(M[..., 2], 0),
                            D(M[..., 1], 0) - D(M[..., 0], 1)], dim=-1)
    n, h = c["n"], 1.0 / (c["n"] + 1)
    p, q = s["p"].double(), s["q"].double()
    D = lambda o, x: _rows_apply(x, 0, *_centered(o, c["a"], h, n))  # noqa: E731
    return D(1, q) * D(2, p) + 2.0 * D(2, q) * D(1, p) + D(3, q) * p[1:-1]
