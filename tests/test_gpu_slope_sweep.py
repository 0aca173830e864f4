"""The specialised single-column sweep of designs with one slope column against
the generic sweep (staged_sweep 0), at the sizes where its row chunks and
ranges have remainders, for every class of the other terms."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import demeaned_errors

pytestmark = pytest.mark.gpu


def effects(wb, kind, n, rng):
    u32 = lambda a: a.astype(np.uint32)   # noqa: E731
    firm = u32(np.sort(rng.integers(0, max(1, n // 12), n)))
    year = u32(rng.integers(0, 9, n))
    x = rng.standard_normal(n)
    return {"firm_slope_year": [wb.Effect(firm, True, [x]), wb.Effect(year, True)],
            "year_slope": [wb.Effect(firm, True), wb.Effect(year, True, [x])],
            "slope_only": [wb.Effect(firm, True), wb.Effect(year, False, [x])],
            "alone": [wb.Effect(firm, True, [x])],
            "rest": [wb.Effect(firm, True, [x]), wb.Effect(u32(rng.integers(0, max(1, n // 9), n)), True)],
            "three": [wb.Effect(firm, True, [x]), wb.Effect(year, True),
                      wb.Effect(u32(rng.integers(0, max(1, n // 7), n)), True)]}[kind]


# 128 rows per chunk, one chunk per warp up to 303,104 rows (148 x 2 blocks of 8 warps)
@pytest.mark.parametrize("kind,n,weighted", [
    ("firm_slope_year", 127, False), ("firm_slope_year", 128, True), ("firm_slope_year", 1025, True),
    ("firm_slope_year", 303105, True), ("year_slope", 40003, False), ("slope_only", 5001, True),
    ("alone", 20002, True), ("rest", 30001, False), ("three", 60001, True)])
def test_slope_sweep_matches_generic(wb, kind, n, weighted):
    rng = np.random.default_rng(n)
    eff = effects(wb, kind, n, rng)
    w = rng.lognormal(0, 0.5, n) if weighted else None
    y = rng.standard_normal(n)
    opts = wb.LsmrOptions(tol=1e-12, maxiter=20000)
    a = wb.Solver(eff, weights=w, tuning={"staged_sweep": 0})
    b = wb.Solver(eff, weights=w, tuning={}, preconditioner=a.preconditioner)
    ra, rb = a.solve(y, opts), b.solve(y, opts)
    assert rb.converged
    # the same preconditioner, both at tol 1e-12: the contract's 1e-7 at 1e-8, scaled with room
    assert demeaned_errors(rb.demeaned, ra.demeaned, y)["inf_over_inf"] < 1e-8
    np.testing.assert_array_equal(b.solve(y, opts).x, rb.x)


def test_adjoint_matches_generic(wb):
    import torch
    n = 50_021
    rng = np.random.default_rng(4)
    eff = effects(wb, "firm_slope_year", n, rng)
    w = rng.lognormal(0, 0.5, n)
    u = torch.tensor(rng.standard_normal(n), device="cuda")
    out = []
    for tuning in ({"staged_sweep": 0}, {}):
        s = wb.Solver(eff, weights=w, preconditioner=wb.PreconditionerConfig.Off, tuning=tuning)
        g = torch.empty(s.n_dofs, dtype=torch.float64, device="cuda")
        s.operator_apply_adjoint_device(u, g)
        out.append(g)
    # sums of at most n terms of unit size in two orders
    assert float((out[0] - out[1]).abs().max()) <= n * 2.3e-16 * float(out[0].abs().max())
