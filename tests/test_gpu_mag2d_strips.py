"""The 2D solve at the edges of its strips (30 owned columns, batches of four
rows) and of its problems' ends: grids of one interior node, one column fewer
and one more than a strip, row counts around a multiple of four, problems that
end at different iterations of a chunk, an iteration budget that ends inside
one, and a zero right-hand side.  Solutions are checked by the CPU oracle's
operator to the solve's own tolerance, iterations against the oracle's CG.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(3, 3), (31, 5), (30, 6), (32, 7), (62, 9), (61, 40), (3, 70), (70, 3), (4, 129)]


def _batch(shapes, seed):
    rng = np.random.default_rng(seed)
    mus, rhss = [], []
    for nx, ny in shapes:
        b = np.zeros((ny, nx))
        b[1:-1, 1:-1] = rng.standard_normal((ny - 2, nx - 2))
        mus.append(np.where(rng.uniform(size=nx * ny) < 0.2, 50.0, rng.uniform(0.5, 2.0, nx * ny)))
        rhss.append(b.ravel())
    return mus, rhss


def _solve(shapes, mus, rhss, **kw):
    from similie_b200 import magnetostatics as m2
    sols = [torch.full((len(b),), float("nan"), device="cuda", dtype=torch.float64) for b in rhss]
    diag = m2.solve_batch([torch.from_numpy(m).cuda() for m in mus], [torch.from_numpy(b).cuda() for b in rhss], sols,
                          shapes, **kw)
    return [s.cpu().numpy() for s in sols], diag


@pytest.mark.parametrize("solver", ["cg", "mixed"])
@pytest.mark.parametrize("shapes", [SHAPES, SHAPES[::-1], [(161, 130)]])
def test_solutions(shapes, solver):
    mus, rhss = _batch(shapes, 3)
    sols, diag = _solve(shapes, mus, rhss, solver=solver, tol=1e-10, max_iterations=3000)
    for (nx, ny), mu, b, x, d in zip(shapes, mus, rhss, sols, diag):
        if solver == "mixed" and min(nx, ny) == 3:
            continue   # the FP32 passes stagnate near 1e-7 on a single line of unknowns
        assert d.converged, (nx, ny)
        r = b - O.mag2d_apply(nx, ny, mu, x)
        assert np.linalg.norm(r) <= 1.01e-10 * np.linalg.norm(b), (nx, ny)


@pytest.mark.parametrize("budget", [1, 31, 32, 33, 50])
def test_budget_counts_every_iteration(budget):
    shapes = [(161, 130), (90, 95)]
    mus, rhss = _batch(shapes, 4)
    sols, diag = _solve(shapes, mus, rhss, solver="cg", tol=1e-10, max_iterations=budget)
    for (nx, ny), mu, b, x, d in zip(shapes, mus, rhss, sols, diag):
        assert d.iterations == budget and not d.converged
        ref, its, _ = O.mag2d_cg(nx, ny, mu, b, tol=1e-30, max_iter=budget)
        assert np.max(np.abs(x - ref)) <= 1e-9 * np.max(np.abs(ref))


def test_zero_source():
    shapes = [(33, 20), (40, 41)]
    mus, rhss = _batch(shapes, 5)
    rhss[0][:] = 0.0
    sols, diag = _solve(shapes, mus, rhss, solver="cg", tol=1e-10)
    assert np.all(sols[0] == 0.0) and diag[0].iterations == 0
    assert diag[1].converged
