"""The mixed-precision 2D solve where CG reaches FP32's precision within one pass of 32 iterations: grids of a
single line of unknowns, and of a few.  The next pass then starts from a residual that the recurrence has lost,
and must not go on with the direction it kept.

Grids up to 4,949 nodes wide are solved on chip, wider ones by the kernels per iteration; both are here.  The
residual is the CPU oracle's.  A pass on a few unknowns or one line gains up to FP32's 1e-7, a line takes about 32
iterations for it, and (4, 129) and (5000, 4) about 130 in all, so 600 iterations are several times what 1e-10 needs.
"""
import numpy as np
import pytest

import oracle as O
from test_gpu_mag2d_strips import _batch, _solve

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")

CHIP = [(3, 3), (3, 4), (3, 9), (9, 3), (3, 70), (70, 3), (3, 600), (3, 5000), (4, 129)]
STEPS = [(5000, 3), (6001, 3), (5000, 4)]


@pytest.mark.parametrize("seed", [3, 12])
@pytest.mark.parametrize("shapes", [CHIP, STEPS, [(70, 3)], [(5000, 3)]])
def test_thin_grids_converge(shapes, seed):
    mus, rhss = _batch(shapes, seed)
    sols, diag = _solve(shapes, mus, rhss, solver="mixed", tol=1e-10, max_iterations=600)
    for (nx, ny), mu, b, x, d in zip(shapes, mus, rhss, sols, diag):
        assert d.converged, (nx, ny, d)
        r = b - O.mag2d_apply(nx, ny, mu, x)
        assert np.linalg.norm(r) <= 1.01e-10 * np.linalg.norm(b), (nx, ny)
