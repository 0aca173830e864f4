"""One apply of the preconditioner on the list engine against the block-tile
engine: each on a handle of its own of the same image, the tile one with its
engine chosen by the environment when the handle builds its plans.  Covers
narrow rounds in one launch, rounds of their own, and a factor of many rounds
whose reduced vector is too long for the shared memory of the narrow rounds."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_seglist import design

pytestmark = pytest.mark.gpu


def ladder(firms=30_000):
    """Workers between neighbouring firms only: a path of 30,000 kept levels, eliminated in many short rounds."""
    w = np.arange(2 * (firms - 1))
    codes = np.empty((2 * w.size, 2), np.uint32, order="F")
    codes[:, 0] = np.repeat(w, 2)
    codes[0::2, 1] = w // 2
    codes[1::2, 1] = w // 2 + 1
    return codes


def codes_of(kind):
    return ladder() if kind == "ladder" else design(kind, np.random.default_rng(1))


def handles(wb, kind, monkeypatch):
    """(list handle, tile handle, solver) of one image; each has built its plans."""
    import torch
    s = wb.Solver(codes_of(kind), tuning={})
    m = s.preconditioner
    t = type(m).from_bytes(m.to_bytes())
    r = torch.zeros(s.n_dofs, dtype=torch.float64, device="cuda")
    z = torch.empty_like(r)
    monkeypatch.setenv("WITHIN_WARP_RANGES", "0")
    t.apply_device(r, z)
    monkeypatch.delenv("WITHIN_WARP_RANGES")
    m.apply_device(r, z)
    return m, t, s


@pytest.mark.parametrize("kind", ["panel", "islands", "gaps", "rounds", "rounds_wide", "ladder"])
def test_apply_matches_tiles(wb, monkeypatch, kind):
    import torch
    m, t, s = handles(wb, kind, monkeypatch)
    r = torch.randn(s.n_dofs, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    za, zb = torch.empty_like(r), torch.empty_like(r)
    t.apply_device(r, za)
    m.apply_device(r, zb)
    # sums of at most 2e5 terms in another order, through at most 64 rounds of a diagonally dominant factor:
    # 2e5 * 2.2e-16 per step, a factor of 2 for the operands' own errors
    assert float((za - zb).norm() / za.norm()) < 1e-10
    assert bool(torch.isfinite(zb).all())
    again = torch.empty_like(r)
    m.apply_device(r, again)
    assert torch.equal(again, zb)


def test_ladder_solves(wb):
    """Every column count against the tile engine's solves."""
    codes = ladder()
    n = codes.shape[0]
    a = wb.Solver(codes, tuning={"warp_ranges": 0})
    b = wb.Solver(codes, tuning={}, preconditioner=a.preconditioner)
    assert a.preconditioner.stats()["n_rounds"] > 3   # the tile engine runs their tail in one launch
    assert a.preconditioner.stats()["n_reduced"] > 9_300   # beyond the shared memory of k_rounds
    for k in (1, 2, 4, 8):
        Y = np.asfortranarray(np.random.default_rng(k).standard_normal((n, k)))
        opts = wb.LsmrOptions(tol=1e-12, maxiter=5000)
        ra, rb = a.solve_batch(Y, opts), b.solve_batch(Y, opts)
        assert all(ra.converged) and all(rb.converged)
        for c in range(k):
            d = np.abs(rb.demeaned[:, c] - ra.demeaned[:, c]).max() / np.abs(Y[:, c]).max()
            assert d < 1e-8   # the same preconditioner, both at tol 1e-12: the contract's 1e-7 at 1e-8, scaled with room
