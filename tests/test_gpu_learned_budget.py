"""A learned solve whose iteration budget ends in the preconditioned stage: the plain solver, which takes over
what has not converged, has nothing left to spend, so it adds no iteration and no refinement pass.

The stage counts its iterations in chunks of eight, which every budget here is a multiple of.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

WEIGHTS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "similie_b200", "data",
                       "precond_2d.npy")


@pytest.mark.parametrize("budget", [8, 64, 96])
def test_a_spent_budget_ends_the_solve(budget):
    from similie_b200 import magnetostatics as m2
    from similie_b200.precond import LearnedPreconditioner
    net = LearnedPreconditioner(seed=0)
    net.load(WEIGHTS)
    probs = [m2.synthetic_problem(np.random.default_rng(1), 256)]
    mus = [torch.from_numpy(p.node_mu()).cuda() for p in probs]
    rhss = [torch.from_numpy(p.rhs()).cuda() for p in probs]
    sols = [torch.zeros_like(b) for b in rhss]
    # far below what so few iterations reach: nothing converges
    diag = m2.solve_batch(mus, rhss, sols, [(p.nx, p.ny) for p in probs], solver="learned", tol=1e-14,
                          max_iterations=budget, preconditioner=net)
    for d in diag:
        assert not d.converged and d.iterations == d.learned_iterations <= budget
        # one pass of the preconditioned stage runs a chunk at least
        assert d.refinements <= budget // 8
