"""The column-lane sweep where its histogram bins leave room for two blocks per
SM (36 to 53 bins) and for one (54 to 64), on rows that fill that grid, against
the single-column solves."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import demeaned_errors

pytestmark = pytest.mark.gpu


# one row past 16-row ranges on every stream: 148 blocks x 4 warps x 8 (K = 8), 16 (4) or 32 (2) streams, twice with
# two blocks per SM
@pytest.mark.parametrize("levels,k,n,weighted", [
    (64, 8, 148 * 4 * 8 * 16 + 1, True), (54, 8, 148 * 4 * 8 * 16 + 1, False), (53, 8, 2 * 148 * 4 * 8 * 16 + 1, True),
    (36, 8, 2 * 148 * 4 * 8 * 16 + 1, False), (64, 4, 148 * 4 * 16 * 16 + 1, False),
    (50, 3, 2 * 148 * 4 * 16 * 16 + 1, True), (64, 2, 148 * 4 * 32 * 16 + 1, True),
    (50, 2, 2 * 148 * 4 * 32 * 16 + 1, False)])
def test_batch_matches_single_columns(wb, levels, k, n, weighted):
    rng = np.random.default_rng(levels * 8 + k)
    worker = np.sort(rng.integers(0, n // 9, n))
    spell = np.repeat(rng.integers(0, n // 30, n // 4 + 1), 4)[:n]
    third = rng.integers(0, levels, n)
    third[-1] = levels - 1
    codes = np.asfortranarray(np.column_stack([worker, spell, third]).astype(np.uint32))
    w = rng.lognormal(0, 1, n) if weighted else None
    Y = np.asfortranarray(rng.standard_normal((n, k)))
    opts = wb.LsmrOptions(tol=1e-12, maxiter=20000)
    s = wb.Solver(codes, weights=w, tuning={})
    b = s.solve_batch(Y, opts)
    assert all(b.converged)
    for c in range(k):
        one = s.solve(np.ascontiguousarray(Y[:, c]), opts)
        # both solves stop at tol 1e-12: the contract's 1e-7 at tol 1e-8, scaled with room
        assert demeaned_errors(b.demeaned[:, c], one.demeaned, Y[:, c])["inf_over_inf"] < 1e-8
    np.testing.assert_array_equal(s.solve_batch(Y, opts).x, b.x)
