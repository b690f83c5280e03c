"""The compile-time-rank DEC kernels against the table-driven ones, bit for bit.

A spectator dim of extent one makes a field take the table-driven kernels, so
the same data runs both ways.  Boxes hold one node, an edge pair, and runs
past a block; strides are the two component orders and reversed lattice axes;
output boxes are the input's, one smaller, and shifted across its faces.  The
Laplacian's marching kernels (3D, and 2D 1-forms, for boxes inside the input)
meet an exact number of tiles (30 owned nodes along the lanes, 6 rows), one
more, several runs of planes, and clamped and unclamped upper faces.
"""
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = {1: [(1,), (2,), (300,)], 2: [(1, 2), (3, 5), (2, 131), (37, 6)],
          3: [(1, 1, 2), (3, 2, 4), (4, 5, 67), (9, 3, 3)]}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shape,ks", [((7, 31), (1,)), ((67, 62), (1,)), ((301, 241), (1,)), ((5, 13, 61), (1, 2)),
                                      ((40, 14, 35), (1, 2)), ((41, 12, 30), (1, 2)), ((131, 125, 124), (0, 3))])
def test_marching_laplacians_equal_the_table_driven_ones(shape, ks, dtype):
    import similie_b200 as sb
    n = len(shape)
    rng = np.random.default_rng(sum(shape))
    geo = sb.Geometry([np.cumsum(rng.uniform(0.3, 1.7, s + 4)) for s in shape])
    for k in ks:
        inp = torch.from_numpy(rng.standard_normal(shape + (comb(n, k),))).cuda().to(dtype)
        inp.view(-1)[11], inp.view(-1)[97] = float("inf"), float("nan")
        boxes = [(shape, (0,) * n), (tuple(s - 1 for s in shape), (0,) * n), (tuple(s - 2 for s in shape), (1,) * n)]
        for oshape, front in boxes if inp.numel() < 10 ** 6 else boxes[:2]:
            for layout in ("last", "first", "reversed"):
                got, ref = (_run(sb, "laplacian", geo, shape, k, k, inp, oshape, front, layout, dtype, sp)
                            for sp in (False, True))
                assert torch.equal(torch.isnan(got), torch.isnan(ref)), (k, oshape, front, layout)
                assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(ref)), (k, oshape, front, layout)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shape,ks", [((83, 77, 92), (1, 2, 3)), ((84, 78, 94), (2,)), ((78, 84, 93), (1, 3)),
                                      ((3, 447, 400), (2, 3))])
def test_marching_codifferentials_equal_the_table_driven_ones(shape, ks, dtype):
    """Tiles of 31 x 7 owned nodes: just under, exactly, and one over a whole number of them; few planes."""
    import similie_b200 as sb
    rng = np.random.default_rng(sum(shape))
    geo = sb.Geometry([np.cumsum(rng.uniform(0.3, 1.7, s + 4)) for s in shape])
    for k in ks:
        inp = torch.from_numpy(rng.standard_normal(shape + (comb(3, k),))).cuda().to(dtype)
        inp.view(-1)[11], inp.view(-1)[-97] = float("inf"), float("nan")
        for oshape, front in ((shape, (0, 0, 0)), ((shape[0],) + tuple(s - 1 for s in shape[1:]), (0, 1, 0)),
                              (tuple(s - 1 for s in shape), (1, 0, 1))):
            for layout in ("last", "first", "reversed"):
                got, ref = (_run(sb, "codifferential", geo, shape, k, k - 1, inp, oshape, front, layout, dtype, sp)
                            for sp in (False, True))
                assert torch.equal(torch.isnan(got), torch.isnan(ref)), (k, oshape, front, layout)
                assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(ref)), (k, oshape, front, layout)


def _laid_out(t, layout):
    """The same values under another layout: component last, component first, lattice axes reversed in memory."""
    n = t.dim() - 1
    if layout == "last":
        return t.contiguous(), -1
    if layout == "first":
        return t.movedim(-1, 0).contiguous(), 0
    order = list(range(n))[::-1] + [n]
    return t.permute(order).contiguous().permute(order), -1


def _run(sb, op, geo, shape, k, ko, inp, oshape, front, layout, dtype, spectator):
    n = len(shape)
    i, ax = _laid_out(inp, layout)
    o, _ = _laid_out(torch.full(oshape + (comb(n, ko),), float("nan"), device="cuda", dtype=dtype), layout)
    kw = {"comp_axis": ax, "in_front": (2,) * n, "out_front": tuple(2 + f for f in front)}
    ii, oo = i, o
    if spectator:
        # a leading lattice dim of extent one that carries no form
        at = 1 if ax == 0 else 0
        ii, oo = i.unsqueeze(at), o.unsqueeze(at)
        kw.update(form_dims=tuple(range(1, n + 1)), in_front=(0,) + kw["in_front"], out_front=(0,) + kw["out_front"])
    if op in ("deriv", "transposed_coboundary"):
        getattr(sb, op)(oo, ii, k, **kw)
    else:
        getattr(sb, op)(geo, oo, ii, k, **kw)
    return o if layout != "first" else o.movedim(0, -1)


@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("op", ["deriv", "transposed_coboundary", "codifferential", "laplacian"])
def test_dense_kernels_equal_the_table_driven_ones(n, dtype, op):
    import similie_b200 as sb
    rng = np.random.default_rng(11 * n)
    for shape in SHAPES[n]:
        # the geometry covers every output box below
        geo = sb.Geometry([np.cumsum(rng.uniform(0.3, 1.7, s + 4)) for s in shape])
        for k in range(n + 1):
            ko = {"deriv": k + 1, "transposed_coboundary": k + 1, "codifferential": k - 1, "laplacian": k}[op]
            if not 0 <= ko <= n:
                continue
            inp = torch.from_numpy(rng.standard_normal(shape + (comb(n, k),))).cuda().to(dtype)
            if inp.numel() > 40:
                inp.view(-1)[7], inp.view(-1)[23] = float("inf"), float("nan")
            for oshape, front in ((shape, (0,) * n), (tuple(max(1, s - 1) for s in shape), (0,) * n),
                                  (tuple(s + 1 for s in shape), (-1,) * n), (shape, (1,) * n)):
                for layout in ("last", "first", "reversed"):
                    got, ref = (_run(sb, op, geo, shape, k, ko, inp, oshape, front, layout, dtype, sp)
                                for sp in (False, True))
                    assert torch.equal(torch.isnan(got), torch.isnan(ref)), (shape, k, oshape, front, layout)
                    assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(ref)), (shape, k, oshape, front, layout)
