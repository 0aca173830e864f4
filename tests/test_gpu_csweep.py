"""Column-lane row sweep (several right-hand sides): batches against the
single-column solves of the same design, at the sizes where its row ranges,
steps and streams have remainders, for every mix of term classes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import demeaned_errors, normal_equation_residual

pytestmark = pytest.mark.gpu


def design(kind, n, rng):
    worker = np.sort(rng.integers(0, max(1, n // 9), n))
    spell = np.repeat(rng.integers(0, max(1, n // 30), n // 4 + 1), 4)[:n]
    year = rng.integers(0, 20, n)
    cols = {"run_run_hist": [worker, spell, year], "hist_hist": [rng.integers(0, 7, n), rng.integers(0, 50, n)],
            "run_rest": [worker, rng.integers(0, max(1, n // 5), n)], "hist_run": [year, worker],
            "one": [worker]}[kind]
    return np.asfortranarray(np.column_stack(cols).astype(np.uint32))


# 511..513: one block of eight-column ranges of 16 rows; 227329: one row past
# the full grid's 16-row ranges at eight columns
@pytest.mark.parametrize("kind,n,k,weighted", [
    ("run_run_hist", 1, 2, False), ("run_run_hist", 17, 8, True), ("run_run_hist", 511, 8, False),
    ("run_run_hist", 512, 4, True), ("run_run_hist", 513, 8, False), ("run_run_hist", 227329, 8, True),
    ("run_run_hist", 100003, 3, False), ("run_run_hist", 50001, 2, True), ("hist_hist", 4099, 5, True),
    ("run_rest", 30011, 8, False), ("hist_run", 20003, 2, False), ("one", 777, 4, True)])
def test_batch_matches_single_columns(wb, kind, n, k, weighted):
    rng = np.random.default_rng(n * 8 + k)
    codes = design(kind, n, rng)
    w = rng.lognormal(0, 1, n) if weighted else None
    Y = np.asfortranarray(rng.standard_normal((n, k)))
    opts = wb.LsmrOptions(tol=1e-12, maxiter=20000)
    s = wb.Solver(codes, weights=w)
    b = s.solve_batch(Y, opts)
    assert all(b.converged)
    for c in range(k):
        one = s.solve(np.ascontiguousarray(Y[:, c]), opts)
        # both solves stop at tol 1e-12: the contract's 1e-7 at tol 1e-8, scaled with room
        assert demeaned_errors(b.demeaned[:, c], one.demeaned, Y[:, c])["inf_over_inf"] < 1e-8
        if n > 600:
            assert normal_equation_residual(codes.T, Y[:, c], b.demeaned[:, c], w) < 1e-9
    again = s.solve_batch(Y, opts)
    np.testing.assert_array_equal(again.demeaned, b.demeaned)
    np.testing.assert_array_equal(again.x, b.x)


def test_mixed_residual_sweep(wb):
    """The FP64 residual sweep of the mixed-precision refinement (two, four and eight columns)."""
    n = 60013
    rng = np.random.default_rng(7)
    codes = design("run_run_hist", n, rng)
    w = rng.lognormal(0, 1, n)
    s = wb.Solver(codes, weights=w)
    sm = wb.Solver(codes, weights=w, precision="mixed")
    opts = wb.LsmrOptions(tol=1e-11, maxiter=20000)
    for k in (2, 4, 7):
        Y = np.asfortranarray(rng.standard_normal((n, k)))
        a, m = s.solve_batch(Y, opts), sm.solve_batch(Y, opts)
        assert all(m.converged)
        for c in range(k):
            assert demeaned_errors(m.demeaned[:, c], a.demeaned[:, c], Y[:, c])["inf_over_inf"] < 1e-7
