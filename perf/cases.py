"""The workloads that the performance of this framework is judged on.

Every case goes through the package's public Python entry points as a program
would call them.  Designs are synthetic, drawn on the GPU from a seed, with
the shapes of ``within_b200/workloads.py``:

- ``two_factor``  uniform codes in two factors (500 x 200 levels at n = 100,000)
- ``panel``       worker-sorted worker/firm/year panel: ten observations per
  worker (geometric), n/100 firms of Pareto(1.5) size, a worker switching firm
  with probability 0.1 per observation, 20 years
- ``fixest``      the reference's wall-clock design: ten observations per
  worker, ten years, firm = i modulo the number of firms
- ``slopes``      firms of Pareto(1.5) size with an intercept and a slope, and
  30 years

``listed`` holds the cases, ``draw`` makes more of the same ranges, ``prepare``
what a program holds before the call, ``run`` the call, ``work`` the bytes and
operations no implementation can do without and ``exact`` the same outputs from
conjugate gradients on the normal equations in plain torch FP64.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import within_b200 as wb


def listed():
    return [
        # the smallest call: a regression on a few thousand rows inside a loop; launches and latency only
        {"name": "solve_2k", "kind": "solve", "design": "two_factor", "n": 2003, "k": 1, "weighted": False,
         "precision": "fp64", "host": False, "tol": 1e-8},
        # the small plain configuration, numpy in and out as most programs call it
        {"name": "solve_100k_host", "kind": "solve", "design": "two_factor", "n": 100000, "k": 1,
         "weighted": False, "precision": "fp64", "host": True, "tol": 1e-8},
        # the reference's wall-clock design with a kept solver: many light iterations on a dense core
        {"name": "fixest_1m", "kind": "solve", "design": "fixest", "n": 1000000, "k": 1, "weighted": False,
         "precision": "fp64", "host": False, "tol": 1e-6},
        # the same design one-shot: set-up and solve, the wall-clock a script sees
        {"name": "oneshot_1m", "kind": "oneshot", "design": "fixest", "n": 1000000, "tol": 1e-6},
        # the headline: one response on the large worker/firm/year panel
        {"name": "panel_10m", "kind": "solve", "design": "panel", "n": 10000000, "k": 1, "weighted": False,
         "precision": "fp64", "host": False, "tol": 1e-8},
        # response and seven covariates of the same panel in one batch
        {"name": "panel_10m_k8", "kind": "solve", "design": "panel", "n": 10000000, "k": 8, "weighted": False,
         "precision": "fp64", "host": False, "tol": 1e-8},
        # a weighted regression with two covariates on an odd number of rows: a batch of three columns
        {"name": "panel_2m_w_k3", "kind": "solve", "design": "panel", "n": 1999993, "k": 3, "weighted": True,
         "precision": "fp64", "host": False, "tol": 1e-8},
        # mixed precision on a weighted panel, four columns, at the tolerance where it equals the FP64 solve
        {"name": "mixed_4m_k4", "kind": "solve", "design": "panel", "n": 4000000, "k": 4, "weighted": True,
         "precision": "mixed", "host": False, "tol": 1e-11},
        # differentiable demeaning with varying slopes and weights: forward and backward
        {"name": "slopes_2m_grad", "kind": "grad", "n": 2000000, "tol": 1e-10},
        # independent designs of uneven size, eight columns each, numpy in and out
        {"name": "many_16_k8", "kind": "many", "designs": 16, "lo": 10000, "hi": 200000, "k": 8, "tol": 1e-8},
        # the plain operator in both directions, for programs that bring their own iteration
        {"name": "operator_10m", "kind": "operator", "n": 10000000, "weighted": False},
        # the preconditioner alone, for the same programs
        {"name": "precond_4m", "kind": "precond", "n": 4000000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.choice(["two_factor", "panel", "panel", "panel", "fixest", "oneshot", "mixed", "grad", "many",
                       "operator", "precond"])
    w = rng.random() < 0.5
    if pick == "two_factor":
        return {"kind": "solve", "design": "two_factor", "n": _log_int(rng, 2000, 500000),
                "k": rng.choice([1, 1, 2, 5]), "weighted": w, "precision": "fp64", "host": rng.random() < 0.5,
                "tol": 1e-8}
    if pick == "panel":
        k = rng.randint(1, 8)
        return {"kind": "solve", "design": "panel", "n": _log_int(rng, 20000, 10000000 // (2 * k if k > 1 else 1)),
                "k": k, "weighted": w, "precision": "fp64", "host": False, "tol": 1e-8}
    if pick == "fixest":
        return {"kind": "solve", "design": "fixest", "n": _log_int(rng, 50000, 1000000), "k": rng.choice([1, 2]),
                "weighted": w, "precision": "fp64", "host": False, "tol": 1e-6}
    if pick == "oneshot":
        return {"kind": "oneshot", "design": rng.choice(["two_factor", "fixest"]),
                "n": _log_int(rng, 50000, 600000), "tol": 1e-6}
    if pick == "mixed":
        return {"kind": "solve", "design": "panel", "n": _log_int(rng, 200000, 4000000), "k": rng.randint(1, 4),
                "weighted": True, "precision": "mixed", "host": False, "tol": 1e-11}
    if pick == "grad":
        return {"kind": "grad", "n": _log_int(rng, 100000, 2000000), "tol": 1e-10}
    if pick == "many":
        return {"kind": "many", "designs": rng.randint(4, 16), "lo": 10000, "hi": _log_int(rng, 20000, 150000),
                "k": rng.randint(1, 8), "tol": 1e-8}
    if pick == "operator":
        return {"kind": "operator", "n": _log_int(rng, 20000, 10000000), "weighted": w}
    return {"kind": "precond", "n": _log_int(rng, 20000, 4000000)}


# ---------------------------------------------------------------------------
# inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, n):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g)


def _normal(g, *shape):
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def _pareto_draws(g, levels, count):
    """`count` levels drawn in proportion to Pareto(1.5) sizes."""
    sizes = (1.0 - _uniform(g, levels)).pow(-1.0 / 1.5)
    cdf = torch.cumsum(sizes / sizes.sum(), 0)
    return torch.searchsorted(cdf, _uniform(g, count), right=True).clamp_(max=levels - 1)


def _uniform_codes(g, levels, n):
    c = torch.randint(0, levels, (n,), device="cuda", generator=g)
    c[-1] = levels - 1
    return c


def _codes(design, n, g):
    """The design's code columns as int64 CUDA tensors, in the order a program's table has them.  The last
    row carries the largest level of every factor, so the number of coefficients does not depend on the seed."""
    if design == "two_factor":
        a, b = max(20, n // 200), max(20, n // 500)
        return [_uniform_codes(g, a, n), _uniform_codes(g, b, n)]
    i = torch.arange(n, device="cuda")
    if design == "fixest":
        firms = max(1, round(max(1, round(n / 10)) / 23))
        return [i // 10, i % 10, i % firms]
    workers, firms = max(1, n // 10), max(1, n // 100)
    counts = torch.empty(workers, dtype=torch.float64, device="cuda").geometric_(0.1, generator=g)
    ends = torch.cumsum(counts, 0)
    worker = torch.searchsorted(ends, i.to(torch.float64), right=True).clamp_(max=workers - 1)
    switch = _uniform(g, n) < 0.1
    switch[0] = True
    switch[1:] |= worker[1:] != worker[:-1]
    spell = torch.cumsum(switch, 0) - 1
    firm = _pareto_draws(g, firms, n)[spell]
    worker[-1], firm[-1] = workers - 1, firms - 1
    return [worker, firm, _uniform_codes(g, 20, n)]


def _matrix(cols):
    """uint32 categories matrix in column order, as the package takes it."""
    return torch.stack([c.to(torch.int32) for c in cols]).cpu().numpy().view(np.uint32).T


def _weights(g, n, sigma=1.0):
    return torch.exp(sigma * _normal(g, n))


def _many_shapes(case):
    """Rows and level counts of the designs: rows spread evenly over their logarithm, two or three factors."""
    count, lo, hi = case["designs"], case["lo"], case["hi"]
    out = []
    for i in range(count):
        n = int(lo * (hi / lo) ** ((i + 0.5) / count)) | 1
        r = random.Random(n)
        out.append((n, [_log_int(r, 20, max(21, n // 10)) for _ in range(2 + i % 2)]))
    return out


def _inputs(case, seed):
    """Everything of a case that depends on the seed, on the GPU."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "many":
        return [([_uniform_codes(g, lv, n) for lv in levels],
                 _normal(g, case["k"], n)) for n, levels in _many_shapes(case)]
    n = case["n"]
    if kind == "grad":
        firms = max(2, n // 40)
        firm = _pareto_draws(g, firms, n)
        year = torch.randint(0, 30, (n,), device="cuda", generator=g)
        return {"firm": firm, "year": year, "x": _normal(g, n), "z": _normal(g, n), "w": _weights(g, n, 0.5),
                "v": _normal(g, n)}
    cols = _codes(case.get("design", "panel"), n, g)
    w = _weights(g, n) if case.get("weighted") else None
    if kind == "operator":
        nd = sum(int(c.max()) + 1 for c in cols)
        return {"cols": cols, "w": w, "x": _normal(g, nd), "u": _normal(g, n)}
    if kind == "precond":
        return {"cols": cols, "w": w, "r": _normal(g, sum(int(c.max()) + 1 for c in cols))}
    k = case.get("k", 1)
    if case.get("design") == "fixest":
        return {"cols": cols, "w": w, "Y": 2.0 * torch.rand(k, n, dtype=torch.float64, device="cuda", generator=g) - 1.0}
    return {"cols": cols, "w": w, "Y": _normal(g, k, n)}


def _options(case):
    return wb.LsmrOptions(tol=case["tol"], maxiter=2000)


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "many":
        solver = wb.SolverSet([_matrix(cols) for cols, _ in d])
        return {"kind": kind, "solver": solver, "Ys": [Y.cpu().numpy().T for _, Y in d], "options": _options(case)}
    if kind == "grad":
        effects = [wb.Effect(d["firm"].to(torch.int32).cpu().numpy().view(np.uint32), True, [d["x"].cpu().numpy()]),
                   wb.Effect(d["year"].to(torch.int32).cpu().numpy().view(np.uint32), True)]
        solver = wb.Solver(effects, weights=d["w"].cpu().numpy())
        return {"kind": kind, "solver": solver, "effects": effects, "z": d["z"], "w": d["w"], "v": d["v"],
                "options": _options(case)}
    codes = _matrix(d["cols"])
    w = None if d["w"] is None else d["w"].cpu().numpy()
    if kind == "oneshot":
        return {"kind": kind, "codes": codes, "y": d["Y"][0].cpu().numpy(), "options": _options(case)}
    if kind == "operator":
        solver = wb.Solver(codes, w, wb.PreconditionerConfig.Off)
        return {"kind": kind, "solver": solver, "x": d["x"], "u": d["u"],
                "y": torch.empty(case["n"], dtype=torch.float64, device="cuda"),
                "g": torch.empty(solver.n_dofs, dtype=torch.float64, device="cuda")}
    if kind == "precond":
        solver = wb.Solver(codes, w)
        return {"kind": kind, "solver": solver, "m": solver.preconditioner, "r": d["r"],
                "out": torch.empty_like(d["r"])}
    solver = wb.Solver(codes, w, precision=case["precision"])
    if case["host"]:
        Y = d["Y"].cpu().numpy()
        return {"kind": kind, "solver": solver, "host": True, "options": _options(case),
                "Y": Y[0] if case["k"] == 1 else Y.T}
    # column-major (n, k), the layout the device entry point documents
    return {"kind": kind, "solver": solver, "host": False, "options": _options(case),
            "Y": d["Y"][0] if case["k"] == 1 else d["Y"].t()}


# ---------------------------------------------------------------------------
# the calls

def run(state):
    kind = state["kind"]
    if kind == "many":
        return [(x, dm) for x, dm, _, _ in state["solver"].solve_batch(state["Ys"], state["options"])]
    if kind == "grad":
        z = state["z"].detach().requires_grad_(True)
        w = state["w"].detach().requires_grad_(True)
        out = wb.demean(z, state["effects"], weights=w, options=state["options"], solver=state["solver"])
        gz, gw = torch.autograd.grad(out, (z, w), state["v"])
        return {"out": out.detach(), "gz": gz, "gw": gw}
    if kind == "oneshot":
        r = wb.solve(state["codes"], state["y"], options=state["options"])
        return {"x": r.x, "demeaned": r.demeaned}
    if kind == "operator":
        state["solver"].operator_apply_device(state["x"], state["y"])
        state["solver"].operator_apply_adjoint_device(state["u"], state["g"])
        return {"y": state["y"], "g": state["g"]}
    if kind == "precond":
        state["m"].apply_device(state["r"], state["out"])
        return state["out"]
    if state["host"]:
        if state["Y"].ndim == 1:
            r = state["solver"].solve(state["Y"], state["options"])
        else:
            r = state["solver"].solve_batch(state["Y"], state["options"])
        return {"x": r.x, "demeaned": r.demeaned}
    X, D, _ = state["solver"].solve_device(state["Y"], state["options"])
    return {"x": X, "demeaned": D}


def _solve_work(n, levels, k, weighted, slopes=0):
    q, nd = len(levels), sum(levels) + slopes * levels[0]
    terms = q + slopes
    return (4 * q * n + 8 * n * (int(weighted) + slopes) + k * (16 * n + 8 * nd), 4 * terms * n * k)


def _levels(design, n):
    if design == "two_factor":
        return [max(20, n // 200), max(20, n // 500)]
    if design == "fixest":
        return [-(-n // 10), 10, max(1, round(max(1, round(n / 10)) / 23))]
    return [max(1, n // 10), max(1, n // 100), 20]


def work(case):
    """Inputs read once and outputs written once; one product with the design and one with its transpose."""
    kind = case["kind"]
    if kind == "many":
        each = [_solve_work(n, lv, case["k"], False) for n, lv in _many_shapes(case)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    n = case["n"]
    if kind == "grad":
        # codes, slope, z, w, v in; demeaned and the two gradients out; a solve in each direction
        return {"bytes": 2 * 4 * n + 8 * n * 4 + 8 * n * 3, "flops": 2 * 4 * 3 * n}
    levels = _levels(case.get("design", "panel"), n)
    if kind == "operator":
        nd = sum(levels)
        return {"bytes": 2 * 4 * 3 * n + 8 * n * (2 + int(case["weighted"])) + 16 * nd, "flops": 4 * 3 * n}
    if kind == "precond":
        # the vector in and out, and one value and index per worker/firm spell, worker/year and firm/year pair
        nd = sum(levels)
        return {"bytes": 16 * nd + 12 * (n // 5), "flops": 4 * (n // 5)}
    b, f = _solve_work(n, levels, case.get("k", 1), case.get("weighted", False))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same outputs in plain torch

def _design_matrix(cols, values=None):
    """(codes with offsets, loadings or None per column block, dofs)."""
    off, terms = 0, []
    for t, c in enumerate(cols):
        terms.append((c + off, None if values is None else values[t]))
        off += int(c.max()) + 1
    order = [torch.argsort(c, stable=True) for c, _ in terms]
    ends = torch.cat([torch.bincount(c, minlength=off)[None] for c, _ in terms]).sum(0).cumsum(0)
    n = cols[0].shape[0]
    rows = torch.cat(order)
    vals = torch.cat([torch.ones(n, dtype=torch.float64, device="cuda") if v is None else v[o]
                      for (c, v), o in zip(terms, order)])
    crow = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), ends])
    dt = torch.sparse_csr_tensor(crow.to(torch.int32), rows.to(torch.int32), vals, (off, n))
    return {"terms": terms, "dt": dt, "dofs": off}


def _apply(m, X):
    """D X' for X (k, dofs): (k, n)."""
    out = None
    for c, v in m["terms"]:
        g = X[:, c] if v is None else X[:, c] * v
        out = g if out is None else out.add_(g)
    return out


def _adjoint(m, U):
    """D' U' for U (k, n): (k, dofs)."""
    return torch.stack([torch.mv(m["dt"], u) for u in U])


def _project(m, w, Y):
    """Y minus its weighted least-squares fit on the design, one row per column, by conjugate gradients on
    the normal equations with a diagonal scaling, restarted on the true residual until it stops falling."""
    wf = (lambda U: U) if w is None else (lambda U: U * w)
    sq = _design_matrix_squares(m)
    diag = torch.mv(sq, torch.ones(Y.shape[1], dtype=torch.float64, device="cuda") if w is None else w)
    inv = torch.where(diag > 0, 1.0 / diag, torch.zeros_like(diag))
    R = Y.clone()
    g0 = None
    for restart in range(4):
        g = _adjoint(m, wf(R))
        size = (g * g * inv).sum(1)
        g0 = (_adjoint(m, wf(Y).abs()) ** 2 * inv).sum(1) if g0 is None else g0
        if bool((size <= 1e-31 * g0).all()):
            break
        d = torch.zeros_like(g)
        z = g * inv
        p = z.clone()
        gz = (g * z).sum(1)
        stop = torch.maximum(1e-24 * gz, 1e-32 * g0)
        for it in range(3000):
            live = gz > stop   # a column that has converged stays as it is
            if it % 16 == 15 and not bool(live.any()):
                break
            ap = _adjoint(m, wf(_apply(m, p)))
            a = torch.where(live, gz / (p * ap).sum(1), torch.zeros_like(gz))[:, None]
            d += a * p
            g = g - a * ap
            z = g * inv
            new = torch.where(live, (g * z).sum(1), gz)
            p = torch.where(live[:, None], z + (new / gz)[:, None] * p, p)
            gz = new
        R = R - _apply(m, d)
    return R


def _design_matrix_squares(m):
    dt = m["dt"]
    return torch.sparse_csr_tensor(dt.crow_indices(), dt.col_indices(), dt.values() ** 2, dt.shape)


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind == "many":
        return [(None, _project(_design_matrix(cols), None, Y).t()) for cols, Y in d]
    if kind == "grad":
        one = torch.ones_like(d["x"])
        m = _design_matrix([d["firm"], d["firm"], d["year"]], [one, d["x"], one])
        a = d["v"] / d["w"]
        r, s = _project(m, d["w"], torch.stack([d["z"], a]))
        return {"out": r, "gz": d["w"] * s, "gw": -r * (a - s)}
    if kind == "precond":
        return None
    m = _design_matrix(d["cols"])
    if kind == "operator":
        s = 1.0 if d["w"] is None else d["w"].sqrt()
        return {"y": _apply(m, d["x"][None])[0] * s, "g": _adjoint(m, (d["u"] * s)[None])[0]}
    r = _project(m, d["w"], d["Y"])
    flat = kind == "oneshot" or (case["host"] and case["k"] == 1)
    return {"x": None, "demeaned": r[0] if flat else r.t()}
