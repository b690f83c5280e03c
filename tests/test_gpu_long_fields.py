"""2D scalar Laplacians with more rows than a launch has blocks along y (65,535)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows", [65536, 65537, 70001])   # 65,535 output rows and more
@pytest.mark.parametrize("staged", [True, False])
def test_scalar_laplacian(rows, staged):
    import similie_b200 as sb
    rng = np.random.default_rng(rows)
    shape = (rows, 5)
    coords = [np.cumsum(rng.uniform(0.5, 1.5, s)) for s in shape]
    w = rng.standard_normal(shape + (1,))
    geo = sb.Geometry(coords)
    inp = torch.from_numpy(w).cuda()
    out = torch.full((rows - 1, 4, 1), float("nan"), device="cuda", dtype=torch.float64)
    if staged:
        sb.make_staged_laplacian(geo, out, inp, 0).run(out, inp)
    else:
        sb.laplacian(geo, out, inp, 0)
    ref = O.laplacian(2, 0, O.position_from_coords(coords), w)
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))
