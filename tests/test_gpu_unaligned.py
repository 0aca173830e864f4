"""Device vectors that start between 16-byte boundaries (slices), through every
device entry point that takes one: the results of the same values aligned."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def aligned_and_slice(values):
    import torch
    a = torch.tensor(values, dtype=torch.float64, device="cuda")
    b = torch.empty(a.numel() + 1, dtype=torch.float64, device="cuda")[1:]
    b.copy_(a)
    assert a.data_ptr() % 16 == 0 and b.data_ptr() % 16 == 8
    return a, b


@pytest.mark.parametrize("tuning", [{}, {"staged_sweep": 0}])
@pytest.mark.parametrize("n", [129, 40_003])
def test_slices(wb, n, tuning):
    import torch
    rng = np.random.default_rng(n)
    worker = np.sort(rng.integers(0, max(1, n // 10), n))
    spell = np.repeat(rng.integers(0, max(1, n // 40), n // 5 + 1), 5)[:n]
    codes = np.asfortranarray(np.column_stack([worker, spell, rng.integers(0, 20, n)]).astype(np.uint32))
    s = wb.Solver(codes, weights=rng.lognormal(0, 1, n), tuning=tuning)

    def out(m):
        return aligned_and_slice(np.zeros(m))

    u, x, y = (aligned_and_slice(rng.standard_normal(m)) for m in (n, s.n_dofs, n))
    for call, args, m in ((s.operator_apply_adjoint_device, u, s.n_dofs), (s.operator_apply_device, x, n),
                          (s.preconditioner.apply_device, x, s.n_dofs)):
        want, got = out(m)
        call(args[0], want)
        for a in args:
            for o in out(m):
                call(a, o)
                assert torch.equal(o, want), call
    Xa, Xs = out(s.n_dofs)
    Da, Ds = out(n)
    s.solve_device(y[0], X=Xa, D=Da)
    s.solve_device(y[1], X=Xs, D=Ds)
    assert torch.equal(Xs, Xa) and torch.equal(Ds, Da)
