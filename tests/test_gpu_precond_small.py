"""The learned preconditioner on batches whose grids are all too small for a second network level (a half-resolution
side below 16 pixels): its apply against the CPU oracle, and a learned solve.

The tolerance of the apply is that of the larger grids' test, 2e-2 of the norm: features and weights of these one-level
networks are rounded to BF16 once on both sides, at most 2^-8 each in a handful of steps.
"""
import os

import numpy as np
import pytest

import oracle as O
from oracle import precond_oracle as P
from test_gpu_precond import flat, make_batch, pc, rel, torch  # noqa: F401

pytestmark = pytest.mark.gpu

WEIGHTS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "similie_b200", "data",
                       "precond_2d.npy")


@pytest.mark.parametrize("shapes", [[(3, 3)], [(16, 16)], [(5, 40), (30, 30), (3, 4)]])
def test_apply_matches_oracle(torch, pc, shapes):  # noqa: F811
    batch = make_batch(shapes, 3)
    params = P.init_params(5)
    net = pc.LearnedPreconditioner(seed=0)
    net.set_params(params)
    nu, r = (flat(torch, [s[i] for s in batch]) for i in (0, 1))
    out = torch.zeros_like(r)
    net.apply(shapes, nu, r, out)
    got = out.cpu().numpy()
    off = 0
    for (nx, ny), (nub, b, _) in zip(shapes, batch):
        ref = P.precond(params, nub.astype(np.float32), b.astype(np.float32), emulate=True)
        g = got[off:off + nx * ny].reshape(ny, nx)
        off += nx * ny
        assert rel(g, ref) < 2e-2, ((nx, ny), rel(g, ref))


def test_learned_solve(torch, pc):  # noqa: F811
    from similie_b200 import magnetostatics as m2
    shapes = [(20, 20), (3, 9), (24, 17)]
    batch = make_batch(shapes, 4)
    net = pc.LearnedPreconditioner(seed=0)
    net.load(WEIGHTS)
    mus = [torch.from_numpy((1.0 / s[0]).ravel().copy()).cuda() for s in batch]
    rhss = [torch.from_numpy(s[1].ravel().copy()).cuda() for s in batch]
    sols = [torch.zeros_like(b) for b in rhss]
    diag = m2.solve_batch(mus, rhss, sols, shapes, solver="learned", tol=1e-10, preconditioner=net)
    for (nx, ny), mu, b, x, d in zip(shapes, mus, rhss, sols, diag):
        assert d.converged, (nx, ny, d)
        res = b.cpu().numpy() - O.mag2d_apply(nx, ny, mu.cpu().numpy(), x.cpu().numpy())
        assert np.linalg.norm(res) <= 1.01e-10 * np.linalg.norm(b.cpu().numpy())
