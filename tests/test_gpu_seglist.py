"""The list engine (default) against the block-tile engine of the same
preconditioner, at every column count: long segments cut into pieces, medium
and short ones, many tiny subdomains, and empty segments."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import demeaned_errors

pytestmark = pytest.mark.gpu


def design(kind, rng):
    if kind == "panel":      # long rows of C^T (years, large firms), giant subdomains
        from within_b200 import workloads as WL
        return WL.akm_panel(n=150_000, n_workers=15_000, n_firms=1_500, seed=3)
    if kind == "islands":    # thousands of components of a few levels each
        g = np.repeat(np.arange(6_000), 4)
        return np.asfortranarray(np.column_stack([2 * g + rng.integers(0, 2, g.size),
                                                  2 * g + rng.integers(0, 2, g.size)]).astype(np.uint32))
    if kind == "rounds":     # a deep factor: 30 and more narrow elimination rounds and a dense core
        from within_b200 import workloads as WL
        return WL.fixest_like(n=600_000)[0]
    if kind == "rounds_wide":   # a factor whose first rounds are launches of their own
        return np.asfortranarray(np.column_stack([rng.integers(0, 30_000, 150_000), rng.integers(0, 6_000, 150_000)])
                                 .astype(np.uint32))
    # unused levels: empty segments of the prolongation and of the adjoint's rest
    a, b = 3 * rng.integers(0, 700, 40_000), 2 * rng.integers(0, 900, 40_000)
    return np.asfortranarray(np.column_stack([a, b, rng.integers(0, 4, 40_000)]).astype(np.uint32))


@pytest.mark.parametrize("kind", ["panel", "islands", "gaps", "rounds", "rounds_wide"])
@pytest.mark.parametrize("k", [1, 2, 3, 8])
def test_lists_match_tiles(wb, kind, k):
    rng = np.random.default_rng(11 + k)
    codes = design(kind, rng)
    n = codes.shape[0]
    w = rng.lognormal(0, 1, n) if k != 2 else None
    Y = np.asfortranarray(rng.standard_normal((n, k)))
    opts = wb.LsmrOptions(tol=1e-12, maxiter=5000)
    a = wb.Solver(codes, weights=w, tuning={"warp_ranges": 0})
    b = wb.Solver(codes, weights=w, tuning={}, preconditioner=a.preconditioner)
    ra, rb = a.solve_batch(Y, opts), b.solve_batch(Y, opts)
    for c in range(k):
        assert rb.converged[c]
        # the same preconditioner and both at tol 1e-12: the contract's 1e-7 at 1e-8, scaled with room
        assert demeaned_errors(rb.demeaned[:, c], ra.demeaned[:, c], Y[:, c])["inf_over_inf"] < 1e-8
    again = b.solve_batch(Y, opts)
    np.testing.assert_array_equal(again.x, rb.x)


def test_preconditioner_apply_matches_tiles(wb):
    import torch
    codes = design("panel", np.random.default_rng(1))
    a = wb.Solver(codes, tuning={"warp_ranges": 0})
    b = wb.Solver(codes, tuning={})
    r = torch.randn(a.n_dofs, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    za, zb = torch.empty_like(r), torch.empty_like(r)
    a.preconditioner.apply_device(r, za)
    b.preconditioner.apply_device(r, zb)
    # one apply: sums of at most 1e5 terms in another order
    assert float((za - zb).norm() / za.norm()) < 1e-12
