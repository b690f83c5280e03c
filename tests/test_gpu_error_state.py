"""A call that fails before it runs anything does not make the next, valid call fail."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _deriv_is_right():
    import oracle as O
    import similie_b200 as sb
    w = np.random.default_rng(1).standard_normal((20, 30, 1))
    d = torch.full((20, 30, 2), float("nan"), device="cuda", dtype=torch.float64)
    sb.deriv(d, torch.from_numpy(w).cuda(), 0)
    ref = np.zeros((20, 30, 2))
    O.coboundary(w, ref, 0)
    np.testing.assert_array_equal(d.cpu().numpy(), ref)


@pytest.mark.parametrize("solver", ["cg", "mixed"])
def test_after_a_solve_without_memory(solver):
    # the working memory of four such problems is over 380 GB: refused before any of the fields is read
    from similie_b200 import SilError
    from similie_b200 import magnetostatics as m2
    field = [torch.zeros(16, device="cuda", dtype=torch.float64)] * 4
    with pytest.raises(SilError) as e:
        m2.solve_batch(field, field, field, [(46000, 46000)] * 4, solver=solver)
    assert e.value.status == 4   # SIL_ERR_ALLOC
    _deriv_is_right()
