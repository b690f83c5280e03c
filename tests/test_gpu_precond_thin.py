"""Weight gradients of the two thin convolutions against FP64 sums over the
GPU's own operands: images of one pixel row, narrower than a tile, an exact
number of tiles, and several images behind one another.

Tolerance: a weight's sum goes through at most 16 products per tile and lane
(two tiles a block at these sizes), eight warps and up to 592 partials in
eighths: under 128 additions, so 2^-17 times the sum of the magnitudes.
"""
import numpy as np
import pytest

from oracle import precond_oracle as P
from test_gpu_precond import flat, make_batch, pc, torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [[(3, 3)], [(40, 7)], [(252, 255)], [(96, 130), (3, 5), (65, 34)]])
def test_thin_weight_gradients(torch, pc, shapes):  # noqa: F811
    batch = make_batch(shapes, 9)
    net = pc.LearnedPreconditioner(seed=0)
    net.set_params(P.init_params(12))
    nu, b, x = (flat(torch, [s[i] for s in batch]) for i in range(3))
    _, _, grad = net.loss_grad(shapes, nu, b, x)
    dims = [((ny + 1) // 2, (nx + 1) // 2) for nx, ny in shapes]
    total = sum((h + 2) * (w + 2) for h, w in dims)
    h0, g0, dh0 = (net.debug_fetch(which, 0, total * P.C).astype(np.float64).reshape(total, P.C) for which in (0, 2, 3))
    feat = net.debug_fetch(5, 0, total * 2).astype(np.float64).reshape(total, 2)
    gnet = net.debug_fetch(8, 0, total).astype(np.float64)
    want, size = np.zeros(P.NUM_PARAMS), np.zeros(P.NUM_PARAMS)
    at = 0
    for h, w in dims:
        sl = slice(at, at + (h + 2) * (w + 2))
        at = sl.stop
        pad = lambda a: a[sl].reshape(h + 2, w + 2, -1)  # noqa: E731
        dz = (pad(dh0) * (pad(h0) > 0))[1:-1, 1:-1]
        for to, mag in ((want, False), (size, True)):
            f = np.abs if mag else (lambda a: a)
            dw, db = P.conv_wgrad(f(pad(gnet[:, None]))[1:-1, 1:-1], f(pad(g0)))
            to[P.OFF_OUT:P.OFF_OUT + P.OUT_W] += dw[0].ravel()
            to[P.OFF_OUT + P.OUT_W] += db[0]
            dw, db = P.conv_wgrad(f(dz), f(pad(feat)))
            to[P.OFF_IN:P.OFF_IN + P.IN_W] += dw.ravel()
            to[P.OFF_IN + P.IN_W:P.OFF_IN + P.IN_W + P.C] += db
    for a, e in ((P.OFF_IN, P.OFF_IN + P.IN_W + P.C), (P.OFF_OUT, P.NUM_PARAMS)):
        assert np.all(np.abs(grad[a:e] - want[a:e]) <= 2.0 ** -17 * size[a:e])
