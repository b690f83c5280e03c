"""The 2D solve by kernels per iteration on grids that would fit on chip: nothing on chip is allowed here, so the
edges of a strip (30 owned columns, batches of four rows) and of a chunk of 32 iterations are those kernels' own.

Grids of one interior node, one column fewer and one more than a strip, row counts around a multiple of four,
problems that end at different iterations of a chunk, a budget that ends inside one, a zero source, and a limit
that leaves the on-chip part a few blocks.  Solutions are checked by the CPU oracle's operator to the solve's own
tolerance; after a fixed number of iterations the iterate is the oracle's to 1e-9 of its largest value, the
rounding of up to 50 FP64 iterations on these well-scaled operators.
"""
import numpy as np
import pytest

import oracle as O
from test_gpu_mag2d_strips import SHAPES, _batch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _solve(shapes, mus, rhss, blocks=0, wait_polls=-1, **kw):
    from similie_b200 import magnetostatics as m2
    limits = m2.ChipLimits(blocks, wait_polls)
    sols = [torch.full((len(b),), float("nan"), device="cuda", dtype=torch.float64) for b in rhss]
    diag = m2.solve_batch_within(limits, [torch.from_numpy(m).cuda() for m in mus],
                                 [torch.from_numpy(b).cuda() for b in rhss], sols, shapes, **kw)
    return [s.cpu().numpy() for s in sols], diag, limits


def _check(shapes, mus, rhss, sols, diag, tol):
    for (nx, ny), mu, b, x, d in zip(shapes, mus, rhss, sols, diag):
        assert d.converged, (nx, ny)
        r = b - O.mag2d_apply(nx, ny, mu, x)
        assert np.linalg.norm(r) <= 1.01 * tol * np.linalg.norm(b), (nx, ny)


@pytest.mark.parametrize("solver", ["cg", "mixed"])
@pytest.mark.parametrize("shapes", [SHAPES, SHAPES[::-1], [(161, 130)], [(29, 33), (31, 34), (60, 35), (61, 36)]])
def test_solutions(shapes, solver):
    mus, rhss = _batch(shapes, 3)
    sols, diag, limits = _solve(shapes, mus, rhss, solver=solver, tol=1e-10, max_iterations=3000)
    assert limits.solved == 0
    _check(shapes, mus, rhss, sols, diag, 1e-10)


@pytest.mark.parametrize("budget", [1, 31, 32, 33, 50])
def test_budget_counts_every_iteration(budget):
    shapes = [(161, 130), (90, 95)]
    mus, rhss = _batch(shapes, 4)
    sols, diag, _ = _solve(shapes, mus, rhss, solver="cg", tol=1e-30, max_iterations=budget)
    for (nx, ny), mu, b, x, d in zip(shapes, mus, rhss, sols, diag):
        assert d.iterations == budget and not d.converged
        ref, _, _ = O.mag2d_cg(nx, ny, mu, b, tol=1e-300, max_iter=budget)
        assert np.max(np.abs(x - ref)) <= 1e-9 * np.max(np.abs(ref))


def test_zero_source():
    shapes = [(33, 20), (40, 41)]
    mus, rhss = _batch(shapes, 5)
    rhss[0][:] = 0.0
    sols, diag, _ = _solve(shapes, mus, rhss, solver="cg", tol=1e-10)
    assert np.all(sols[0] == 0.0) and diag[0].iterations == 0
    _check(shapes[1:], mus[1:], rhss[1:], sols[1:], diag[1:], 1e-10)


@pytest.mark.parametrize("blocks,solved", [(1, 2), (2, 3), (-1, 3)])
def test_a_few_blocks(blocks, solved):
    # FP64: 1, 1 and 2 blocks of 7,168 nodes at least
    shapes = [(33, 20), (40, 41), (100, 90)]
    mus, rhss = _batch(shapes, 6)
    sols, diag, limits = _solve(shapes, mus, rhss, blocks=blocks, solver="cg", tol=1e-10)
    assert limits.solved == solved
    _check(shapes, mus, rhss, sols, diag, 1e-10)


def test_limits_are_checked():
    import ctypes

    import similie_b200 as sil
    from similie_b200 import _native
    for bad in ((-2, -1), (-1, -2)):
        lim = _native.SilChipLimits(*bad)
        assert sil.lib().sil_mag2d_solve_batch_within(ctypes.byref(lim), None, 0, None, None, None) == 1
        assert b"limits" in sil.lib().sil_last_error()
    assert sil.lib().sil_mag2d_solve_batch_within(None, None, 0, None, None, None) == 1
