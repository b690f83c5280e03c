"""Boxes that the marching kernels' tiles cover badly (a few columns, or a few rows of them): the 3D curl-curl operator and
the 1- and 2-form Laplacians take a thread per node there, and the tiles on grids of an exact number of them, one more and
one fewer.

Values against the CPU oracle and the table-driven kernels; that the dispatch does it shows in the time, against a cube
of as many nodes: a march over 3x3x40000 nodes took 6 times the cube's, over 100000x3x3 21 times, a thread per node
takes less and 4 times.
"""
import numpy as np
import pytest

import oracle as O
from test_gpu_dec_dense import _run
from test_gpu_mag3d_march import _coords

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIDES = [(62, 70, 130), (63, 71, 130), (61, 69, 130), (94, 64, 90), (31, 140, 100), (62, 14, 500)]   # marched
THIN = [(3, 3, 40000), (5, 20000, 5), (20000, 5, 5), (33, 8, 1300), (400, 3, 400)]


def _operator(shape, seed):
    from similie_b200 import magnetostatics3d as m3
    rng = np.random.default_rng(seed)
    xyz = [_coords(rng, s) for s in shape]
    n = int(np.prod(shape))
    mu = np.where(rng.uniform(size=n) < 0.2, 1000.0, rng.uniform(0.5, 2.0, n))
    a = rng.standard_normal(3 * n)
    return m3.Operator(*xyz, torch.from_numpy(mu).cuda()), xyz, mu, a


@pytest.mark.parametrize("shape", SIDES + THIN)
def test_operator(shape):
    from similie_b200 import magnetostatics3d as m3
    op, xyz, mu, a = _operator(shape, 1)
    y = torch.full((len(a),), float("nan"), device="cuda", dtype=torch.float64)
    op.apply(torch.from_numpy(a).cuda(), y)
    ref = O.mag3d_apply(*xyz, mu, m3.DEFAULT_GAUGE_PENALTY, a)
    assert np.max(np.abs(y.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("shape", [(2000, 6, 6), (3, 5000, 5), (4, 4, 6000), (300, 300, 2), (120, 31, 13)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_laplacian_bits(shape, dtype):
    import similie_b200 as sb
    rng = np.random.default_rng(2)
    geo = sb.Geometry([np.cumsum(rng.uniform(0.3, 1.7, s + 4)) for s in shape])
    for k in (1, 2):
        inp = torch.from_numpy(rng.standard_normal(shape + (3,))).cuda().to(dtype)
        oshape = tuple(s - 1 for s in shape)
        for layout in ("last", "first", "reversed"):
            got, ref = (_run(sb, "laplacian", geo, shape, k, k, inp, oshape, (0, 0, 0), layout, dtype, sp)
                        for sp in (False, True))
            assert torch.equal(got, ref), (k, layout)


def _time(call):
    call()
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        for _ in range(10):
            call()
    best = float("inf")
    for _ in range(5):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        graph.replay()
        t1.record()
        t1.synchronize()
        best = min(best, t0.elapsed_time(t1))
    return best


def test_thin_operators_are_not_marched():
    def time_of(shape):
        op, _, _, a = _operator(shape, 3)
        x = torch.from_numpy(a).cuda()
        y = torch.zeros_like(x)
        return _time(lambda: op.apply(x, y))

    assert time_of((3, 3, 40000)) <= 3 * time_of((72, 71, 70))


def test_thin_laplacians_are_not_marched():
    import similie_b200 as sb

    def time_of(shape):
        geo = sb.Geometry([np.linspace(0.0, 1.0, s) for s in shape])
        inp = torch.randn(*shape, 3, device="cuda", dtype=torch.float64)
        out = torch.zeros(*[s - 1 for s in shape], 3, device="cuda", dtype=torch.float64)
        plan = sb.make_staged_laplacian(geo, out, inp, 1)
        return _time(lambda: plan.run(out, inp))

    assert time_of((100000, 3, 3)) <= 10 * time_of((74, 74, 74))
