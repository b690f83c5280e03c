"""Working memory of the batched solves: small ones (up to 64 MiB) take it from a pool the library keeps,
larger ones from the device.

Calls of both kinds from several threads, each on its own stream, give the solutions of the same calls one
after another, the device keeps no more than the pool's 64 MiB afterwards, and what a call leaves in the
pool (here NaN) does not reach the next.
"""
import threading

import numpy as np
import pytest

from test_gpu_mag2d_strips import _batch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _batch_on_gpu(shapes, seed):
    mus, rhss = _batch(shapes, seed)
    return [torch.as_tensor(m).cuda().double() for m in mus], [torch.as_tensor(b).cuda().double() for b in rhss], shapes


def _solve_on_gpu(batch, **kw):
    from similie_b200 import magnetostatics as m2
    mus, rhss, shapes = batch
    sols = [torch.zeros_like(b) for b in rhss]
    m2.solve_batch(mus, rhss, sols, shapes, **kw)
    return sols


@pytest.mark.parametrize("solver", ["cg", "mixed"])
def test_threads_and_streams_share_the_pool(solver):
    # 900 x 900 nodes are beyond the pool
    made = [_batch_on_gpu(shapes, 5) for shapes in ([(33, 64), (64, 33)], [(48, 48)], [(900, 900)], [(65, 40), (40, 33)])]
    one_by_one = [_solve_on_gpu(b, solver=solver, tol=1e-8) for b in made]
    torch.cuda.synchronize()
    got = [[] for _ in made]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(3):
                got[i].append(_solve_on_gpu(made[i], solver=solver, tol=1e-8))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(made))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i, want in enumerate(one_by_one):
        assert len(got[i]) == 3
        for sols in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(sols, want))


def test_the_device_keeps_at_most_the_pool():
    made = [_batch_on_gpu([(n, n)], 6) for n in (64, 700, 900)]
    first = None
    for _ in range(3):
        for b in made:
            _solve_on_gpu(b, solver="cg", tol=1e-2)
            torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        # the first pass loads the kernels; from then on nothing may pile up
        first = free if first is None else first
        assert free >= first - (64 << 20)


def _with_nan(b):
    bad = b.clone()
    bad[b.numel() // 2] = float("nan")
    return bad


@pytest.mark.parametrize("solver", ["cg", "mixed"])
@pytest.mark.parametrize("shape", [(64, 64), (2600, 12)])   # on chip, and too wide for that
def test_a_nonfinite_solve_leaves_nothing_behind(shape, solver):
    from similie_b200 import SilError
    mus, rhss, shapes = _batch_on_gpu([shape], 9)
    want = _solve_on_gpu((mus, rhss, shapes), solver=solver, tol=1e-6)
    with pytest.raises(SilError):
        _solve_on_gpu((mus, [_with_nan(rhss[0])], shapes), solver=solver, tol=1e-6)
    assert torch.equal(_solve_on_gpu((mus, rhss, shapes), solver=solver, tol=1e-6)[0], want[0])


@pytest.mark.parametrize("gauge", ["penalty", "divergence"])
@pytest.mark.parametrize("solver", ["cg", "mixed"])
def test_a_nonfinite_3d_solve_leaves_nothing_behind(gauge, solver):
    from similie_b200 import SilError
    from similie_b200 import magnetostatics3d as m3
    p = m3.synthetic_problem(np.random.default_rng(4), 16)
    mu, b = torch.from_numpy(p.node_mu()).cuda(), torch.from_numpy(p.rhs()).cuda()

    def solve(rhs):
        x = torch.zeros_like(rhs)
        m3.solve_batch([(p.x, p.y, p.z)], [mu], [rhs], [x], solver=solver, tol=1e-6, gauge=gauge)
        return x

    want = solve(b)
    with pytest.raises(SilError):
        solve(_with_nan(b))
    assert torch.equal(solve(b), want)
