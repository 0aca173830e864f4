"""The times a solve reports: until its right-hand side is loaded, the
iteration, and the rest of the call (demeaning and results)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph_loop", ["1", "0"])
def test_times_divide_the_call(wb, monkeypatch, graph_loop):
    monkeypatch.setenv("WITHIN_GRAPH_LOOP", graph_loop)
    n = 16_000_000
    i = np.arange(n, dtype=np.uint32)
    codes = np.asfortranarray(np.column_stack([i // 160_000, i % 100]))
    s = wb.Solver(codes, preconditioner=wb.PreconditionerConfig.Off, tuning={})
    y = np.random.default_rng(1).standard_normal(n)
    for _ in range(3):
        r = s.solve(y, wb.LsmrOptions(tol=1e-8, maxiter=2))
        # after the loop: demeaning reads 8 bytes of codes and 8 of y per row and writes 8, the store writes 8 (what
        # it reads may still be cached); before it: the load reads 8.  All at 8 TB/s at the most.
        rest = r.time_total - r.time_setup - r.time_solve
        assert rest >= 32 * n / 8e12
        assert r.time_setup >= 8 * n / 8e12
        # the start and at least one iteration: u read and written, codes read
        assert r.time_solve >= 24 * n / 8e12
        assert r.time_solve < r.time_total


def test_times_of_a_zero_response(wb):
    rng = np.random.default_rng(2)
    codes = np.asfortranarray(np.column_stack([rng.integers(0, 50, 3_000), rng.integers(0, 40, 3_000)]).astype(np.uint32))
    r = wb.Solver(codes).solve(np.zeros(3_000))
    assert r.iterations == 0
    assert 0.0 <= r.time_solve < r.time_total and 0.0 <= r.time_setup < r.time_total
