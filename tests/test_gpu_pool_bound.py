"""What the library's pool of solve memory keeps: at most 64 MiB, however much the solves of several threads held at
once.

Free memory is read before the pool has held anything large (a small solve of every kernel instance has loaded the
kernels), so a pool that kept all it was asked for shows: eight solves hold 45 MB each at the same time.
"""
import threading

import pytest

from test_gpu_solve_memory import _batch_on_gpu

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MIB = 1 << 20


def test_the_pool_keeps_at_most_its_bound():
    from similie_b200 import magnetostatics as m2
    small = _batch_on_gpu([(20, 20), (40, 40), (64, 64), (100, 100), (33, 2600)], 6)
    # 700 x 730 nodes: eight FP64 vectors and three more, 45 MB, from the pool; on chip they need 75 blocks each
    made = [_batch_on_gpu([(700, 730)], 7) for _ in range(8)]
    sols = [[torch.zeros_like(b) for b in rhss] for _, rhss, _ in made]
    small_sols = [torch.zeros_like(b) for b in small[1]]
    for solver in ("cg", "mixed"):
        m2.solve_batch(small[0], small[1], small_sols, small[2], solver=solver, tol=1e-2)
        m2.solve_batch(made[0][0], made[0][1], sols[0], made[0][2], solver=solver, tol=1e-1, max_iterations=2)
    streams = [torch.cuda.Stream() for _ in made]
    torch.cuda.synchronize()
    # what the warm-up left in the pool is at most its bound, so this is the device's free memory without the pool
    # less 64 MiB at most
    before = torch.cuda.mem_get_info()[0]
    together = threading.Barrier(len(made))
    failed = []

    def work(i):
        mus, rhss, shapes = made[i]
        try:
            with torch.cuda.stream(streams[i]):
                for _ in range(4):
                    together.wait(60)
                    m2.solve_batch(mus, rhss, sols[i], shapes, solver="cg", tol=1e-8)
        except Exception as e:  # noqa: BLE001 - a thread's failure is the test's
            failed.append(str(e))
            together.abort()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(made))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= before - 64 * MIB
