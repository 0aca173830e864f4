"""The staged single-column sweep against the generic one (staged_sweep 0):
histogram terms whose bins leave room for three, two and no staged blocks per
SM, with and without weights, at remainders of its chunks and ranges."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import demeaned_errors

pytestmark = pytest.mark.gpu


# 454,656 rows: one chunk of 128 rows for each of the 148 x 3 x 8 warps
@pytest.mark.parametrize("n,levels,weighted", [
    (129, 20, False), (40_003, 20, True), (40_003, 33, False), (40_003, 60, True), (454_657, 20, False),
    (454_657, 33, True)])
def test_staged_sweep_matches_generic(wb, n, levels, weighted):
    import torch
    rng = np.random.default_rng(n + levels)
    worker = np.sort(rng.integers(0, max(1, n // 10), n))
    spell = np.repeat(rng.integers(0, max(1, n // 40), n // 5 + 1), 5)[:n]
    codes = np.asfortranarray(np.column_stack([worker, spell, rng.integers(0, levels, n)]).astype(np.uint32))
    w = rng.lognormal(0, 1, n) if weighted else None
    y = rng.standard_normal(n)
    opts = wb.LsmrOptions(tol=1e-12, maxiter=20000)
    a = wb.Solver(codes, weights=w, tuning={"staged_sweep": 0})
    b = wb.Solver(codes, weights=w, tuning={}, preconditioner=a.preconditioner)
    ra, rb = a.solve(y, opts), b.solve(y, opts)
    assert rb.converged
    # the same preconditioner, both at tol 1e-12: the contract's 1e-7 at 1e-8, scaled with room
    assert demeaned_errors(rb.demeaned, ra.demeaned, y)["inf_over_inf"] < 1e-8
    np.testing.assert_array_equal(b.solve(y, opts).x, rb.x)
    u = torch.tensor(rng.standard_normal(n), device="cuda")
    ga, gb = (torch.empty(s.n_dofs, dtype=torch.float64, device="cuda") for s in (a, b))
    a.operator_apply_adjoint_device(u, ga)
    b.operator_apply_adjoint_device(u, gb)
    # sums of at most n terms in two orders
    assert float((ga - gb).abs().max()) <= n * 2.3e-16 * float(ga.abs().max())
