"""What a mixed-precision solver builds and which ranges its sweeps walk: no
FP64 plan that nothing reads, the scan sweep on its own ranges at one column,
and plans for both precisions when a solver changes over."""
from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def panel(n, seed=3):
    rng = np.random.default_rng(seed)
    worker = np.sort(rng.integers(0, n // 10, n))
    spell = np.repeat(rng.integers(0, n // 40, n // 4 + 1), 4)[:n]
    return (np.asfortranarray(np.column_stack([worker, spell, rng.integers(0, 20, n)]).astype(np.uint32)),
            rng.lognormal(0, 1, n), rng)


def test_no_fp64_lists(wb):
    code = ("import sys; sys.path[:0] = [%r, %r]\n"
            "import numpy as np, within_b200 as wb\n"
            "from test_gpu_mixed_plans import panel\n"
            "c, w, rng = panel(60_000)\n"
            "s = wb.Solver(c, w, precision='mixed')\n"
            "for k in (1, 4): s.solve_batch(np.asfortranarray(rng.standard_normal((60_000, k))))\n"
            % (ROOT, os.path.join(ROOT, "tests")))
    err = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, WITHIN_TRACE="1"), check=True,
                         capture_output=True, text=True).stderr
    assert "tile and range plans" in err
    assert "segment lists" not in err


# 606,209: a row past the full ranges of 148 x 3 x 8 warps' chunks, whole for 148 x 2 x 8
@pytest.mark.parametrize("n", [3_001, 606_209])
def test_single_column_keeps_the_scan_ranges(wb, n):
    """Staged or not, the FP32 normal operator and the FP64 residual walk the same ranges: the same bits."""
    codes, w, rng = panel(n)
    y = rng.standard_normal(n)
    opts = wb.LsmrOptions(tol=1e-11, maxiter=2000)
    a = wb.Solver(codes, w, precision="mixed", tuning={"staged_sweep": 0})
    b = wb.Solver(codes, w, precision="mixed", tuning={}, preconditioner=a.preconditioner)
    ra, rb = a.solve(y, opts), b.solve(y, opts)
    np.testing.assert_array_equal(rb.x, ra.x)
    np.testing.assert_array_equal(rb.demeaned, ra.demeaned)


@pytest.mark.parametrize("first", ["fp64", "mixed"])
def test_precision_changes_over(wb, first):
    codes, w, rng = panel(20_011)
    second = "mixed" if first == "fp64" else "fp64"
    opts = wb.LsmrOptions(tol=1e-11, maxiter=2000)
    s = wb.Solver(codes, w, precision=first)
    fresh = {p: wb.Solver(codes, w, precision=p, preconditioner=s.preconditioner) for p in ("fp64", "mixed")}
    for k in (1, 3):
        Y = np.asfortranarray(rng.standard_normal((20_011, k)))
        for p in (first, second, first):
            s.set_precision(p)
            np.testing.assert_array_equal(s.solve_batch(Y, opts).x, fresh[p].solve_batch(Y, opts).x)
