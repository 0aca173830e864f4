"""The adjoint of designs with many full-resolution terms: one launch for a
group of problems, against per-level sums formed in plain numpy."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import demeaned_errors

pytestmark = pytest.mark.gpu


def columns(kind, n, rng):
    """(codes, slopes) per term; none has few levels, so every term but the sorted one keeps its rows."""
    if kind == "eight_long":        # every segment in pieces of blocks
        return [(rng.integers(0, 70 + i, n), 0) for i in range(8)]
    if kind == "eight_short":       # every segment short, fewer blocks than problems at the smallest size
        return [(rng.integers(0, n // 4 + i, n), 0) for i in range(8)]
    if kind == "mixed_lengths":     # short, medium, long and empty segments side by side
        skew = np.minimum((rng.pareto(1.0, n) * 3).astype(np.int64), n // 50)
        return [(rng.integers(0, n // 5, n), 0), (3 * rng.integers(0, max(30, n // 100), n), 0), (skew + 40, 0),
                (rng.integers(0, 90, n), 0)]
    if kind == "wide_short":
        return [(rng.integers(0, n // 4 + i, n), 0) for i in range(3)] + [(rng.integers(0, 90 + i, n), 0) for i in range(2)]
    # twelve problems beside the sorted term's: two launches
    return [(rng.integers(0, m, n), 3) for m in (80, 100, max(81, n // 30), max(82, n // 3))]


@pytest.mark.parametrize("n", [1_003, 60_001])
@pytest.mark.parametrize("kind", ["eight_long", "eight_short", "mixed_lengths", "twelve"])
def test_adjoint_matches_numpy(wb, kind, n):
    import torch
    from within_b200 import _ffi
    rng = np.random.default_rng(n)
    terms = columns(kind, n, rng)
    slopes = [[rng.standard_normal(n) for _ in range(s)] for _, s in terms]
    eff = [wb.Effect(c.astype(np.uint32), True, z) if z else wb.Effect(c.astype(np.uint32), True)
           for (c, _), z in zip(terms, slopes)]
    s = wb.Solver(eff, preconditioner=wb.PreconditionerConfig.Off, tuning={})
    u = rng.standard_normal(n)
    perm = s.obs_perm()   # the operator takes rows in the solver's own order
    ud = torch.tensor(u if perm is None else u[perm], device="cuda")
    g = torch.empty(s.n_dofs, dtype=torch.float64, device="cuda")
    s.operator_apply_adjoint_device(ud, g)   # builds the plans
    L = _ffi.lib()
    L.within_launch_count_reset()
    s.operator_apply_adjoint_device(ud, g)
    # the sweep, its two closing kernels at most, and one launch per eight problems instead of one per problem
    assert L.within_launch_count() <= 4 + (len(terms) + sum(len(z) for z in slopes) + 7) // 8
    if kind == "twelve":   # x is in the whitened basis of the slopes: the solve below covers it
        return
    want = np.concatenate([np.bincount(c, weights=u, minlength=int(c.max()) + 1) for c, _ in terms])
    size = np.concatenate([np.bincount(c, weights=np.abs(u), minlength=int(c.max()) + 1) for c, _ in terms])
    # two orders of a sum of m terms differ by at most 2 m eps times the sum of their sizes; m <= n
    got = g.cpu().numpy()
    assert np.all(np.abs(got - want) <= 2 * n * 2.3e-16 * size)
    assert np.all(got[size == 0] == 0.0)


# wide_short: problems of short segments that fill the GPU run alone beside the grouped ones
@pytest.mark.parametrize("kind,k,n", [(q, k, 20_011) for q in ("eight_long", "mixed_lengths", "twelve")
                                      for k in (1, 2, 4, 8)] + [("wide_short", 8, 200_003)])
def test_solve_matches_tiles(wb, kind, k, n):
    rng = np.random.default_rng(k)
    terms = columns(kind, n, rng)
    eff = [wb.Effect(c.astype(np.uint32), True, [rng.standard_normal(n) for _ in range(q)]) if q
           else wb.Effect(c.astype(np.uint32), True) for c, q in terms]
    w = rng.lognormal(0, 0.5, n)
    Y = np.asfortranarray(rng.standard_normal((n, k)))
    opts = wb.LsmrOptions(tol=1e-12, maxiter=20000)
    a = wb.Solver(eff, weights=w, tuning={"warp_ranges": 0})
    b = wb.Solver(eff, weights=w, tuning={}, preconditioner=a.preconditioner)
    ra, rb = a.solve_batch(Y, opts), b.solve_batch(Y, opts)
    assert all(rb.converged)
    for c in range(k):
        # the same preconditioner and both at tol 1e-12: the contract's 1e-7 at 1e-8, scaled with room
        assert demeaned_errors(rb.demeaned[:, c], ra.demeaned[:, c], Y[:, c])["inf_over_inf"] < 1e-8
    np.testing.assert_array_equal(b.solve_batch(Y, opts).x, rb.x)
