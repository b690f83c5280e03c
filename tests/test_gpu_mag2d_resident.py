"""The on-chip 2D solve at the limits of what it holds, and beside the
kernel-per-step path that takes what it does not.

A CTA holds 7,168 FP64 (14,336 FP32) nodes of whole rows, a group at most one
CTA per multiprocessor, and rows of at most 2,474 (4,949) nodes.  Cases: a group
of nearly the whole GPU, rows that fill a CTA, one row more than a CTA holds,
single rows per CTA, batches of several waves, batches of which only some
problems fit, and grids that just do not.  After a fixed number of iterations
the iterate is the CPU oracle's CG iterate: 1e-9 of its largest value, the
rounding of up to 45 FP64 iterations on these well-scaled operators.
"""
import numpy as np
import pytest

import oracle as O
from test_gpu_mag2d_strips import _batch, _solve

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")

FITS = [[(1024, 1000)], [(512, 14), (512, 15), (7168 // 28, 28 * 3 + 1)], [(2474, 9), (1300, 33), (50, 700)],
        [(130, 128)] * 60]
MIXED = [[(2475, 20), (64, 64)], [(1100, 1000), (96, 100)], [(96, 100), (2600, 5), (161, 33)]]


@pytest.mark.parametrize("budget", [5, 45])
@pytest.mark.parametrize("shapes", FITS + MIXED)
def test_iterates(shapes, budget):
    mus, rhss = _batch(shapes, 6)
    sols, diag = _solve(shapes, mus, rhss, solver="cg", tol=1e-30, max_iterations=budget)
    step = max(1, len(shapes) // 3)
    for (nx, ny), mu, b, x, d in list(zip(shapes, mus, rhss, sols, diag))[::step]:
        assert d.iterations == budget
        ref, _, _ = O.mag2d_cg(nx, ny, mu, b, tol=1e-300, max_iter=budget)
        assert np.max(np.abs(x - ref)) <= 1e-9 * np.max(np.abs(ref)), (nx, ny)


@pytest.mark.parametrize("shapes", [[(300, 200), (14336 // 64, 64), (14336 // 64, 65)], [(4949, 6), (4950, 6), (80, 70)]])
def test_mixed_precision_converges(shapes):
    mus, rhss = _batch(shapes, 7)
    sols, diag = _solve(shapes, mus, rhss, solver="mixed", tol=1e-9)
    for (nx, ny), mu, b, x, d in zip(shapes, mus, rhss, sols, diag):
        assert d.converged, (nx, ny)
        r = b - O.mag2d_apply(nx, ny, mu, x)
        assert np.linalg.norm(r) <= 1.01e-9 * np.linalg.norm(b), (nx, ny)


def test_nonfinite_problem_leaves_the_others_alone():
    from similie_b200 import SilError
    shapes = [(90, 80), (100, 64)]
    mus, rhss = _batch(shapes, 8)
    rhss[0][90 * 40 + 45] = np.nan
    with pytest.raises(SilError):
        _solve(shapes, mus, rhss, solver="cg", tol=1e-10)
    sols, diag = _solve(shapes[1:], mus[1:], rhss[1:], solver="cg", tol=1e-10)
    assert diag[0].converged
