"""The marching-tile 3D operator and solve at the edges of its tiles.

The operator takes the tiles from 300,000 nodes on; its values are those of
the thread-per-node kernel, which the CPU oracle's tests cover, so a grid that
takes the tiles is compared with the oracle: sides that are an exact number of
tiles (31 x 7 owned columns), one more and one fewer, and long thin boxes.
The solve always takes them: sides from 3 nodes, a single plane of interior
nodes, and a batch whose problems end at different times.  The solution is
checked by the oracle's operator to the solve's own tolerance.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _coords(rng, n):
    return np.cumsum(rng.uniform(0.5, 1.5, n)) / n


@pytest.mark.parametrize("shape", [(63, 64, 75), (62, 70, 70), (94, 8, 401), (3, 317, 320), (320, 3, 317), (317, 320, 3)])
def test_operator_tiles(shape):
    from similie_b200 import magnetostatics3d as m3
    rng = np.random.default_rng(sum(shape))
    xyz = [_coords(rng, s) for s in shape]
    n = int(np.prod(shape))
    assert n >= 300000
    mu = np.where(rng.uniform(size=n) < 0.2, 1000.0, rng.uniform(0.5, 2.0, n))
    a = rng.standard_normal(3 * n)
    op = m3.Operator(*xyz, torch.from_numpy(mu).cuda())
    y = torch.full((3 * n,), float("nan"), device="cuda", dtype=torch.float64)
    op.apply(torch.from_numpy(a).cuda(), y)
    ref = O.mag3d_apply(*xyz, mu, m3.DEFAULT_GAUGE_PENALTY, a)
    assert np.max(np.abs(y.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("solver", ["cg", "mixed"])
@pytest.mark.parametrize("shapes", [[(3, 3, 3)], [(33, 9, 5), (3, 40, 8), (12, 3, 34)], [(32, 15, 7), (64, 22, 16)]])
def test_solve_tiles(shapes, solver):
    from similie_b200 import magnetostatics3d as m3
    rng = np.random.default_rng(5)
    xyz, mus, rhss = [], [], []
    for nx, ny, nz in shapes:
        c = [_coords(rng, s) for s in (nx, ny, nz)]
        b = np.zeros((nz, ny, nx, 3))
        b[1:-1, 1:-1, 1:-1] = rng.standard_normal((nz - 2, ny - 2, nx - 2, 3))
        xyz.append(c)
        mus.append(rng.uniform(0.5, 3.0, nx * ny * nz))
        rhss.append(b.ravel())
    sols = [torch.full((len(b),), float("nan"), device="cuda", dtype=torch.float64) for b in rhss]
    diag = m3.solve_batch(xyz, [torch.from_numpy(m).cuda() for m in mus], [torch.from_numpy(b).cuda() for b in rhss], sols,
                          solver=solver, tol=1e-10)
    for c, mu, b, x, d in zip(xyz, mus, rhss, sols, diag):
        assert d.converged
        r = b - O.mag3d_apply(*c, mu, m3.DEFAULT_GAUGE_PENALTY, x.cpu().numpy())
        assert np.linalg.norm(r) <= 1.01e-10 * np.linalg.norm(b)
