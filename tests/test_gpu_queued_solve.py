"""A solve is queued to its end before the host waits: a non-finite response
is reported, writes nothing, and leaves the solver usable."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_response_writes_nothing(wb, k, bad):
    import torch
    rng = np.random.default_rng(2)
    n = 4_001
    codes = np.asfortranarray(np.column_stack([rng.integers(0, 90, n), rng.integers(0, 40, n)]).astype(np.uint32))
    s = wb.Solver(codes)
    Y = torch.tensor(rng.standard_normal((k, n)), device="cuda").t()
    good = [t.clone() for t in s.solve_device(Y)[:2]]
    Z = Y.clone().t().contiguous().t()
    Z[n // 2, k - 1] = bad
    X = torch.full((k, s.n_dofs), 7.0, dtype=torch.float64, device="cuda").t()
    D = torch.full((k, n), 7.0, dtype=torch.float64, device="cuda").t()
    with pytest.raises(ValueError, match="finite"):
        s.solve_device(Z, X=X, D=D)
    assert bool((X == 7.0).all()) and bool((D == 7.0).all())
    again = s.solve_device(Y)[:2]
    assert torch.equal(again[0], good[0]) and torch.equal(again[1], good[1])


def test_demeaned_over_the_response(wb):
    """The outputs may overwrite the response (D is Y)."""
    import torch
    rng = np.random.default_rng(3)
    n = 3_001
    codes = np.asfortranarray(np.column_stack([rng.integers(0, 90, n), rng.integers(0, 40, n)]).astype(np.uint32))
    s = wb.Solver(codes)
    Y = torch.tensor(rng.standard_normal((2, n)), device="cuda").t()
    _, D, _ = s.solve_device(Y)
    want = D.clone()
    _, D, _ = s.solve_device(Y, D=Y)
    assert torch.equal(D, want)
