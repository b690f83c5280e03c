"""When the on-chip part of a 2D solve cannot run, the kernels per iteration solve its problems.

The launch is refused here by planning for more blocks than the device can hold at once: two grids of 800 x 800
nodes take 100 blocks of 7,168 FP64 nodes each, one to a multiprocessor, in one cooperative launch of 200, which
the runtime answers with an error before anything runs.
"""
import numpy as np
import pytest

from test_gpu_mag2d_steps import _batch, _check, _solve

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_refused_launch():
    shapes = [(800, 800), (800, 800), (64, 48)]
    mus, rhss = _batch(shapes, 13)
    sols, diag, limits = _solve(shapes, mus, rhss, blocks=256, solver="cg", tol=1e-8)
    assert limits.handed_over == len(shapes) and limits.solved == 0
    _check(shapes, mus, rhss, sols, diag, 1e-8)
    want, _, _ = _solve(shapes, mus, rhss, blocks=0, solver="cg", tol=1e-8)
    for a, b in zip(sols, want):
        np.testing.assert_array_equal(a, b)
    # and the device still takes what fits it
    sols, diag, limits = _solve(shapes, mus, rhss, blocks=-1, solver="cg", tol=1e-8)
    assert limits.handed_over == 0 and limits.solved == len(shapes)
    _check(shapes, mus, rhss, sols, diag, 1e-8)


@pytest.mark.parametrize("solver", ["cg", "mixed"])
def test_waits_that_run_out(solver):
    # groups of one block and of several: every wait is bounded by nothing at all, so each gives up at once
    shapes = [(20, 20), (161, 130), (600, 500)]
    mus, rhss = _batch(shapes, 14)
    sols, diag, limits = _solve(shapes, mus, rhss, blocks=-1, wait_polls=0, solver=solver, tol=1e-9)
    assert limits.handed_over == len(shapes) and limits.solved == 0
    _check(shapes, mus, rhss, sols, diag, 1e-9)
    # the device, and the memory of the mail, serve the next solve as ever
    sols, diag, limits = _solve(shapes, mus, rhss, blocks=-1, solver=solver, tol=1e-9)
    assert limits.handed_over == 0 and limits.solved == len(shapes)
    _check(shapes, mus, rhss, sols, diag, 1e-9)


def test_one_lost_group_leaves_the_others_alone():
    # a few polls: some groups lose a wait, others may not; each problem is solved by whoever ends with it
    shapes = [(20, 20), (200, 190), (161, 130), (700, 600)]
    mus, rhss = _batch(shapes, 15)
    for polls in (1, 2, 4):
        sols, diag, limits = _solve(shapes, mus, rhss, blocks=-1, wait_polls=polls, solver="cg", tol=1e-9)
        assert limits.handed_over + limits.solved == len(shapes)
        _check(shapes, mus, rhss, sols, diag, 1e-9)
