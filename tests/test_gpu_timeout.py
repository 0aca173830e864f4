"""A timed-out device wait, from the state it leaves (the word is preset from
the host; nothing on the GPU waits): the call that meets it ends early, fails,
writes nothing and leaves the handle usable."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(wb):
    from within_b200 import workloads as WL
    s = wb.Solver(WL.fixest_like(n=600_000)[0], tuning={})   # narrow rounds: kernels that wait for bulk copies
    assert s.preconditioner.stats()["n_rounds"] > 8
    return s


@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("graph_loop", ["1", "0"])
def test_solve_after_a_timeout(wb, monkeypatch, k, graph_loop):
    import torch
    from within_b200 import _ffi
    monkeypatch.setenv("WITHIN_GRAPH_LOOP", graph_loop)
    s = _solver(wb)
    Y = torch.tensor(np.random.default_rng(k).standard_normal((k, s.n_obs)), device="cuda").t()
    L = _ffi.lib()
    L.within_launch_count_reset()
    good = [t.clone() for t in s.solve_device(Y)[:2]]
    full = L.within_launch_count()
    X = torch.full((k, s.n_dofs), 7.0, dtype=torch.float64, device="cuda").t()
    D = torch.full((k, s.n_obs), 7.0, dtype=torch.float64, device="cuda").t()
    _ffi.check(L.within_solver_inject_timeout(s._h))
    L.within_launch_count_reset()
    with pytest.raises(RuntimeError, match="did not complete"):
        s.solve_device(Y, X=X, D=D)
    # the loop ends after its first body (two iterations) or burst (two bodies) instead of running to convergence
    assert L.within_launch_count() < full
    assert bool((X == 7.0).all()) and bool((D == 7.0).all())
    again = s.solve_device(Y)[:2]
    assert torch.equal(again[0], good[0]) and torch.equal(again[1], good[1])


def test_apply_after_a_timeout(wb):
    import torch
    from within_b200 import _ffi
    s = _solver(wb)
    m = s.preconditioner
    r = torch.randn(s.n_dofs, dtype=torch.float64, device="cuda")
    good = torch.empty_like(r)
    m.apply_device(r, good)
    _ffi.check(_ffi.lib().within_preconditioner_inject_timeout(m._h))
    out = torch.full_like(r, 7.0)
    with pytest.raises(RuntimeError, match="did not complete"):
        m.apply_device(r, out)
    assert bool((out == 7.0).all())
    m.apply_device(r, out)
    assert torch.equal(out, good)


def test_operator_after_a_timeout(wb):
    import torch
    from within_b200 import _ffi
    s = _solver(wb)
    x = torch.randn(s.n_dofs, dtype=torch.float64, device="cuda")
    y = torch.empty(s.n_obs, dtype=torch.float64, device="cuda")
    _ffi.check(_ffi.lib().within_solver_inject_timeout(s._h))
    with pytest.raises(RuntimeError, match="did not complete"):
        _ffi.check(_ffi.lib().within_solver_operator_apply(s._h, x.data_ptr(), y.data_ptr(), None))
    _ffi.check(_ffi.lib().within_solver_operator_apply(s._h, x.data_ptr(), y.data_ptr(), None))
