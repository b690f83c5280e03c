"""The work whose speed this repository watches: what a user of the library has
it do, through its public entry points.

Families (`"family"` of a case):

  laplacian  a staged Hodge Laplacian of a k-form on a rectilinear grid
             (make_staged_laplacian once, run per step), the output on the
             lattice without its last node per axis, as in the field solvers
             that step a form in time;
  exterior   the separate operators in the order a field evaluation chains
             them: F = d A, the star of F, and the codifferential of F;
  operator   one apply of the 3D curl-curl operator object, as an outer
             Krylov loop or a time stepper calls it;
  solve2d    a batch of 2D magnetostatics solves to a relative residual, by
             the FP64 ("cg"), mixed-precision ("mixed") or learned solver;
  solve3d    the same for 3D curl-curl problems on stretched grids;
  network    the learned preconditioner by itself: its apply, and the loss
             gradient of a training step.

Sizes are written in the case ("512x512", or a list of sides for a batch);
the inputs come from the seed alone.
"""
import math
import os

import numpy as np
import torch

import similie_b200 as sb
from similie_b200 import magnetostatics as m2
from similie_b200 import magnetostatics3d as m3

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(sb.__file__)), "data", "precond_2d.npy")


def listed():
    return [
        # The scalar Laplacian of a small 2D field: the call a diffusion or wave
        # step makes thousands of times, bound by its launch.
        {"name": "laplacian_scalar_512", "family": "laplacian", "shape": "512x512", "k": 0, "dtype": "f64"},
        # The vector Laplacian of a large 2D field, the benchmark's headline.
        {"name": "laplacian_vector_4096", "family": "laplacian", "shape": "4096x4096", "k": 1, "dtype": "f64"},
        # The same in single precision on the odd-sized grid a mesh file gives.
        {"name": "laplacian_vector_ragged_f32", "family": "laplacian", "shape": "1999x2741", "k": 1, "dtype": "f32"},
        # The vector Laplacian in 3D, on a box with three different sides.
        {"name": "laplacian_vector_3d", "family": "laplacian", "shape": "161x144x130", "k": 1, "dtype": "f64"},
        # B = dA, H = star B, J = delta B on a 3D potential: the post-processing
        # of a solved field.
        {"name": "exterior_3d", "family": "exterior", "shape": "150x171x128", "k": 1, "dtype": "f64"},
        # One apply of the 3D operator at the size of the 3D batch.
        {"name": "operator_256", "family": "operator", "shape": "256x256x256"},
        # A batch of uneven 2D problems in double precision, as a parameter
        # study submits it.
        {"name": "solve2d_batch", "family": "solve2d", "sizes": "128,256,384,512,768,1024", "solver": "cg",
         "tol": 1e-10},
        # A few small problems, as an optimiser's inner loop solves them.
        {"name": "solve2d_small", "family": "solve2d", "sizes": "96,128,128,161", "solver": "cg", "tol": 1e-10},
        # A batch under the learned preconditioner.
        {"name": "solve2d_learned", "family": "solve2d", "sizes": "256,384,512,512,768", "solver": "learned",
         "tol": 1e-10},
        # 3D coils in mixed precision.
        {"name": "solve3d_mixed", "family": "solve3d", "sizes": "64,80,96", "solver": "mixed", "tol": 1e-10},
        # The network alone on a batch of residuals.
        {"name": "network_apply", "family": "network", "sizes": "256,384,512,512,768,768,1024,1024", "grad": False},
        # The gradient of one training step, at the trainer's batch of eight.
        {"name": "network_gradient", "family": "network", "sizes": "256,256,256,256,256,256,256,256", "grad": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["laplacian", "laplacian", "exterior", "operator", "solve2d", "solve2d", "solve3d", "network"])
    if family in ("laplacian", "exterior"):
        n = rng.choice([2, 3])
        side = [_log(rng, 48, 3800) for _ in range(2)] if n == 2 else [_log(rng, 12, 170) for _ in range(3)]
        k = rng.randrange(0, n + 1) if family == "laplacian" else rng.randrange(0, n)
        return {"family": family, "shape": "x".join(map(str, side)), "k": k, "dtype": rng.choice(["f64", "f64", "f32"])}
    if family == "operator":
        return {"family": family, "shape": "x".join(str(_log(rng, 20, 250)) for _ in range(3))}
    if family == "solve2d":
        solver = rng.choice(["cg", "mixed", "learned"])
        sides = [_log(rng, 48, 700) for _ in range(rng.randrange(1, 6))]
        return {"family": family, "sizes": ",".join(map(str, sides)), "solver": solver, "tol": 1e-10}
    if family == "solve3d":
        sides = [_log(rng, 16, 80) for _ in range(rng.randrange(1, 4))]
        return {"family": family, "sizes": ",".join(map(str, sides)), "solver": rng.choice(["cg", "mixed"]),
                "tol": 1e-10}
    grad = rng.choice([False, True])
    sides = [_log(rng, 64, 256 if grad else 900) for _ in range(rng.randrange(1, 9))]
    return {"family": family, "sizes": ",".join(map(str, sides)), "grad": grad}


# ------------------------------------------------------------------ inputs

def _shape(case):
    return [int(v) for v in case["shape"].split("x")]


def _sizes(case):
    return [int(v) for v in case["sizes"].split(",")]


def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _coords(side, ratio_span=4.0):
    """Node coordinates on [0, 1] whose spacing grows geometrically, by `ratio_span` from end to end."""
    return m3.stretched_coords(side, ratio_span ** (1.0 / max(1, side - 2)))


def _random_field(shape, ncomp, generator):
    """Gaussian random components with power spectrum k^-2 and unit rms, (*shape, ncomp) in FP64."""
    noise = torch.randn([ncomp] + list(shape), generator=generator, device="cuda", dtype=torch.float64)
    dims = tuple(range(1, len(shape) + 1))
    spec = torch.fft.rfftn(noise, dim=dims)
    k2 = torch.zeros([1] * len(shape), device="cuda", dtype=torch.float64)
    for a, s in enumerate(shape):
        f = torch.fft.rfftfreq(s, 1.0 / s) if a == len(shape) - 1 else torch.fft.fftfreq(s, 1.0 / s)
        k2 = k2 + (f.cuda().double() ** 2).reshape([-1 if b == a else 1 for b in range(len(shape))])
    spec = spec / torch.sqrt(torch.clamp(k2, min=1.0))
    field = torch.fft.irfftn(spec, s=list(shape), dim=dims)
    field = field / field.square().mean(dim=dims, keepdim=True).sqrt()
    return field.movedim(0, -1).contiguous()


def _problems2d(case, seed):
    rng = np.random.default_rng(seed)
    return [m2.synthetic_problem(rng, n) for n in _sizes(case)]


def _problems3d(case, seed):
    rng = np.random.default_rng(seed)
    return [m3.synthetic_problem(rng, n) for n in _sizes(case)]


def _network_inputs(case, seed):
    """(nu, b, x) FP64 [n, n] per sample: the reluctivity of a synthetic problem and an exact (source, solution)
    pair, x a random field that vanishes on the boundary and b = K x."""
    g = _generator(seed)
    out = []
    for p in _problems2d(case, seed):
        n = p.nx
        nu = (1.0 / torch.from_numpy(p.node_mu()).cuda()).reshape(n, n).float().double()
        x = torch.zeros(n, n, device="cuda", dtype=torch.float64)
        x[1:-1, 1:-1] = _random_field([n, n], 1, g)[1:-1, 1:-1, 0]
        out.append((nu, _k2_apply(x, nu), x))
    return out


def _network(seed):
    from similie_b200.precond import LearnedPreconditioner
    net = LearnedPreconditioner(seed=seed)
    net.load(WEIGHTS)
    return net


def prepare(case, seed):
    fam = case["family"]
    if fam in ("laplacian", "exterior"):
        shape, k, n, dt = _shape(case), case["k"], len(_shape(case)), _dtype(case)
        field = _random_field(shape, math.comb(n, k), _generator(seed)).to(dt)
        geo = sb.Geometry([_coords(s) for s in shape])
        st = {"case": dict(case), "geo": geo, "in": field}
        if fam == "laplacian":
            out = torch.zeros([s - 1 for s in shape] + [math.comb(n, k)], device="cuda", dtype=dt)
            st["out"] = out
            st["plan"] = sb.make_staged_laplacian(geo, out, field, k)
        else:
            st["d"] = torch.zeros(shape + [math.comb(n, k + 1)], device="cuda", dtype=dt)
            st["star"] = torch.zeros(shape + [math.comb(n, n - k - 1)], device="cuda", dtype=dt)
            st["codiff"] = torch.zeros(shape + [math.comb(n, k)], device="cuda", dtype=dt)
        return st
    if fam == "operator":
        nx, ny, nz = _shape(case)
        g = _generator(seed)
        mu = torch.ones(nz, ny, nx, device="cuda", dtype=torch.float64)
        lo = [max(1, s // 4 + (seed % 3)) for s in (nz, ny, nx)]
        mu[lo[0]:lo[0] + nz // 3, lo[1]:lo[1] + ny // 3, lo[2]:lo[2] + nx // 3] = 1000.0
        a = torch.zeros(nz, ny, nx, 3, device="cuda", dtype=torch.float64)
        a[1:-1, 1:-1, 1:-1] = _random_field([nz, ny, nx], 3, g)[1:-1, 1:-1, 1:-1]
        xyz = [_coords(s) for s in (nx, ny, nz)]
        op = m3.Operator(*xyz, mu.reshape(-1))
        return {"case": dict(case), "op": op, "a": a.reshape(-1), "y": torch.zeros_like(a).reshape(-1)}
    if fam == "solve2d":
        probs = _problems2d(case, seed)
        rhs = [torch.from_numpy(p.rhs()).cuda() for p in probs]
        st = {"case": dict(case), "shapes": [(p.nx, p.ny) for p in probs],
              "mu": [torch.from_numpy(p.node_mu()).cuda() for p in probs], "rhs": rhs,
              "sol": [torch.zeros_like(b) for b in rhs]}
        st["net"] = _network(0) if case["solver"] == "learned" else None
        return st
    if fam == "solve3d":
        probs = _problems3d(case, seed)
        rhs = [torch.from_numpy(p.rhs()).cuda() for p in probs]
        return {"case": dict(case), "coords": [(p.x, p.y, p.z) for p in probs], "gammas": [p.gamma for p in probs],
                "mu": [torch.from_numpy(p.node_mu()).cuda() for p in probs], "rhs": rhs,
                "sol": [torch.zeros_like(b) for b in rhs]}
    samples = _network_inputs(case, seed)
    nu, b, x = (torch.cat([s[i].reshape(-1) for s in samples]).float() for i in range(3))
    return {"case": dict(case), "net": _network(0), "shapes": [(n, n) for n in _sizes(case)], "nu": nu, "b": b, "x": x,
            "out": torch.zeros_like(b)}


# ------------------------------------------------------------------ one pass

def run(st):
    case = st["case"]
    fam = case["family"]
    if fam == "laplacian":
        return st["plan"].run(st["out"], st["in"])
    if fam == "exterior":
        k = case["k"]
        sb.deriv(st["d"], st["in"], k)
        sb.hodge_star(st["geo"], st["star"], st["d"], k + 1)
        sb.codifferential(st["geo"], st["codiff"], st["d"], k + 1)
        return {"d": st["d"], "star": st["star"], "codiff": st["codiff"]}
    if fam == "operator":
        return st["op"].apply(st["a"], st["y"])
    if fam == "solve2d":
        m2.solve_batch(st["mu"], st["rhs"], st["sol"], st["shapes"], solver=case["solver"], tol=case["tol"],
                       preconditioner=st["net"])
        return st["sol"]
    if fam == "solve3d":
        m3.solve_batch(st["coords"], st["mu"], st["rhs"], st["sol"], gammas=st["gammas"], solver=case["solver"],
                       tol=case["tol"])
        return st["sol"]
    if case["grad"]:
        loss, per, grad = st["net"].loss_grad(st["shapes"], st["nu"], st["b"], st["x"])
        return {"loss": np.asarray([loss], dtype=np.float32), "per_sample": np.asarray(per, dtype=np.float32),
                "grad": grad}
    return st["net"].apply(st["shapes"], st["nu"], st["b"], st["out"])


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    fam = case["family"]
    if fam in ("laplacian", "exterior"):
        shape, k = _shape(case), case["k"]
        n, es, nodes = len(shape), 8 if case["dtype"] == "f64" else 4, math.prod(shape)
        if fam == "laplacian":
            outn = math.prod(s - 1 for s in shape)
            return {"bytes": es * math.comb(n, k) * (nodes + outn), "flops": 12 * n * math.comb(n, k) * nodes}
        comps = math.comb(n, k) + 3 * math.comb(n, k + 1) + math.comb(n, n - k - 1) + math.comb(n, k)
        return {"bytes": es * nodes * comps, "flops": nodes * n * 10}
    if fam == "operator":
        nodes = math.prod(_shape(case))
        return {"bytes": 8 * 7 * nodes, "flops": 90 * nodes}
    # A solve reads the material and the source and writes the solution; its
    # arithmetic is that of the plain method, about 6 iterations per node of a
    # side (2D) or 20 (3D), an apply and five vector operations each.
    if fam == "solve2d":
        return {"bytes": sum(24 * n * n for n in _sizes(case)), "flops": sum(6 * n * 24 * n * n for n in _sizes(case))}
    if fam == "solve3d":
        return {"bytes": sum(56 * n ** 3 for n in _sizes(case)),
                "flops": sum(20 * n * 120 * n ** 3 for n in _sizes(case))}
    # Network: per top-level pixel (a quarter of the nodes) the decoder, and the
    # two encoder convolutions and the decoder of each coarser level; the
    # gradient adds a data and a weight gradient of each.
    conv = 2 * 9 * 32 * 32
    flops = sum((n * n / 4) * (conv * (1 + 3 / 3) + 2 * 9 * 32 * 3) for n in _sizes(case))
    return {"bytes": sum((16 if case["grad"] else 12) * n * n for n in _sizes(case)),
            "flops": flops * (3 if case["grad"] else 1)}


# ------------------------------------------------------------------ the same in plain FP64

def _combos(n, k):
    import itertools
    return list(itertools.combinations(range(n), k))


def _shift(f, axis, up):
    """f at the next node along `axis`, the last one repeated (up), or at the previous one, zero before the first."""
    if up:
        return torch.cat([f.narrow(axis, 1, f.shape[axis] - 1), f.narrow(axis, f.shape[axis] - 1, 1)], axis)
    return torch.cat([torch.zeros_like(f.narrow(axis, 0, 1)), f.narrow(axis, 0, f.shape[axis] - 1)], axis)


def _d(comps, n, k, transposed):
    """Coboundary of the components of a k-form, or the transposed one (backward differences, zero outside)."""
    low = _combos(n, k)
    out = []
    for c in _combos(n, k + 1):
        acc = None
        for i, a in enumerate(c):
            f = comps[low.index(c[:i] + c[i + 1:])]
            t = f - _shift(f, a, False) if transposed else _shift(f, a, True) - f
            t = -t if i % 2 else t
            acc = t if acc is None else acc + t
        out.append(acc)
    return out


def _star(comps, n, k, h):
    low = _combos(n, k)
    out = []
    for t in _combos(n, n - k):
        c = tuple(a for a in range(n) if a not in t)
        sign = (-1) ** sum(1 for a in c for b in t if a > b)
        f = comps[low.index(c)] * sign
        for a in t:
            f = f * h[a]
        for a in c:
            f = f / h[a]
        out.append(f)
    return out


def _codiff(comps, n, k, h):
    f = _star(_d(_star(comps, n, k, h), n, n - k, True), n, n - k + 1, h)
    return [-v for v in f] if (n * (k + 1) + 1) % 2 else f


def _lengths(shape):
    h = []
    for a, s in enumerate(shape):
        c = torch.from_numpy(_coords(s)).cuda()
        e = torch.cat([c[1:] - c[:-1], c[-1:] - c[-2:-1]])
        h.append(e.reshape([-1 if b == a else 1 for b in range(len(shape))]))
    return h


def _k2_apply(a, nu):
    """The 2D residual operator on [ny, nx] arrays (identity rows on the boundary)."""
    y = a.clone()
    c = a[1:-1, 1:-1]
    r = (c - a[2:, 1:-1]) * nu[1:-1, 1:-1] + (c - a[1:-1, 2:]) * nu[1:-1, 1:-1]
    r[1:, :] += (c[1:, :] - a[1:-2, 1:-1]) * nu[1:-2, 1:-1]
    r[:, 1:] += (c[:, 1:] - a[1:-1, 1:-2]) * nu[1:-1, 1:-2]
    y[1:-1, 1:-1] = r
    return y


def _k2_diagonal(nu):
    d = torch.ones_like(nu)
    t = 2.0 * nu[1:-1, 1:-1]
    t[1:, :] += nu[1:-2, 1:-1]
    t[:, 1:] += nu[1:-1, 1:-2]
    d[1:-1, 1:-1] = t
    return d


def _spacing(c):
    c = np.asarray(c, dtype=np.float64)
    h = np.empty(len(c))
    h[0], h[-1] = c[1] - c[0], c[-1] - c[-2]
    h[1:-1] = 0.5 * (c[2:] - c[:-2])
    return torch.from_numpy(h).cuda()


class _CurlCurl:
    """The 3D residual operator with the penalty gauge on [nz, ny, nx, 3] arrays."""

    def __init__(self, xyz, mu, gamma):
        lx, ly, lz = (_spacing(c).reshape(s) for c, s in zip(xyz, ((1, 1, -1), (1, -1, 1), (-1, 1, 1))))
        nu = (1.0 / mu).clone()
        mask = torch.zeros_like(nu)
        mask[1:-1, 1:-1, 1:-1] = 1.0
        self.mask = mask
        # moments are taken at interior nodes only
        self.w = (lx / (ly * lz) * nu * mask, ly / (lx * lz) * nu * mask, lz / (lx * ly) * nu * mask)
        self.g = (gamma * ly * lz / lx * mask, gamma * lx * lz / ly * mask, gamma * lx * ly / lz * mask)

    @staticmethod
    def _up(f, axis):
        return torch.cat([f.narrow(axis, 1, f.shape[axis] - 1), torch.zeros_like(f.narrow(axis, 0, 1))], axis)

    def apply(self, a):
        ax, ay, az = (a[..., c] * self.mask for c in range(3))
        up, dn = self._up, lambda f, axis: _shift(f, axis, False)
        bx = self.w[0] * ((ay - up(ay, 0)) + (up(az, 1) - az))
        by = self.w[1] * ((up(ax, 0) - ax) + (az - up(az, 2)))
        bz = self.w[2] * ((ax - up(ax, 1)) + (up(ay, 2) - ay))
        rx = (dn(by, 0) - by) + (bz - dn(bz, 1)) + self.g[0] * ax
        ry = (bx - dn(bx, 0)) + (dn(bz, 2) - bz) + self.g[1] * ay
        rz = (dn(bx, 1) - bx) + (by - dn(by, 2)) + self.g[2] * az
        inner = torch.stack([rx, ry, rz], -1)
        m = self.mask[..., None]
        return inner * m + a * (1.0 - m)

    def diagonal(self):
        wx, wy, wz = self.w
        dn = lambda f, axis: _shift(f, axis, False)  # noqa: E731
        d = torch.stack([wy + dn(wy, 0) + wz + dn(wz, 1) + self.g[0], wx + dn(wx, 0) + wz + dn(wz, 2) + self.g[1],
                         wx + dn(wx, 1) + wy + dn(wy, 2) + self.g[2]], -1)
        m = self.mask[..., None]
        return d * m + (1.0 - m)


def _cg(apply, diag, b, limit):
    """x with A x = b as far as FP64 goes: Jacobi-CG on the residual of the sum so far, until it no longer falls."""
    x, best, norm, spent = torch.zeros_like(b), None, float(b.norm()), 0
    while norm > 0 and spent < limit:
        r = b - apply(x)
        rel = float(r.norm()) / norm
        if best is not None and rel > 0.25 * best[0]:
            break
        best = (rel, x.clone())
        e, z = torch.zeros_like(b), r / diag
        p, rz, goal = z.clone(), (r * z).sum(), 1e-5 * float(r.norm()) if best[0] < 1 else 1e-9 * norm
        for i in range(limit - spent):
            q = apply(p)
            alpha = rz / (p * q).sum()
            e += alpha * p
            r -= alpha * q
            z = r / diag
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
            if i % 64 == 63 and float(r.norm()) <= goal:
                break
        spent += i + 1
        x = x + e
    return best[1] if best is not None else x


def _net_parts(p):
    C, T = 32, 9
    big = C * T * C
    cut = [0]

    def take(count):
        cut[0] += count
        return p[cut[0] - count:cut[0]]

    w_in, b_in = take(C * T * 2).reshape(C, 3, 3, 2).permute(0, 3, 1, 2), take(C)
    layers = []
    for _ in range(9):
        layers.append((take(big).reshape(C, 3, 3, C).permute(0, 3, 1, 2), take(C)))
    w_out, b_out = take(T * C).reshape(1, 3, 3, C).permute(0, 3, 1, 2), take(1)
    return w_in, b_in, layers, w_out, b_out


def _net_precondition(p, nu, r):
    """M(r) of the learned preconditioner for one [n, n] sample, in FP64."""
    F = torch.nn.functional
    w_in, b_in, layers, w_out, b_out = _net_parts(p)
    conv = lambda x, w, b: F.conv2d(x, w, b, padding=1)  # noqa: E731

    def pool(x):
        return F.avg_pool2d(F.pad(x, (0, x.shape[-1] % 2, 0, x.shape[-2] % 2)), 2)

    def up(x, h, w):
        return x.repeat_interleave(2, -2).repeat_interleave(2, -1)[..., :h, :w]

    n0, n1 = r.shape
    dinv = 1.0 / _k2_diagonal(nu)
    e1 = 0.8 * dinv * r
    r1 = r - _k2_apply(e1, nu)
    sq = dinv.sqrt()
    s = (dinv * r1 * r1).mean().sqrt()
    x = pool(torch.stack([sq * r1 / s, nu.log() / math.log(1000.0)])[None])
    hs = [torch.relu(conv(x, w_in, b_in))]
    while min(hs[-1].shape[-2:]) >= 16:
        j = 3 * min(len(hs) - 1, 2)
        hs.append(torch.relu(conv(torch.relu(conv(pool(hs[-1]), *layers[j])), *layers[j + 1])))
    g = hs[-1]
    for level in range(len(hs) - 2, -1, -1):
        h, w = hs[level].shape[-2:]
        g = torch.relu(conv(hs[level] + up(g, h, w), *layers[3 * min(level, 2) + 2]))
    inner = torch.zeros_like(r)
    inner[1:-1, 1:-1] = 1.0
    e2 = e1 + s * sq * up(conv(g, w_out, b_out), n0, n1)[0, 0] * inner
    return e2 + 0.8 * dinv * (r - _k2_apply(e2, nu))


def exact(case, seed):
    fam = case["family"]
    if fam in ("laplacian", "exterior"):
        shape, k = _shape(case), case["k"]
        n = len(shape)
        f = _random_field(shape, math.comb(n, k), _generator(seed)).to(_dtype(case)).double()
        comps, h = [f[..., c].contiguous() for c in range(f.shape[-1])], _lengths(shape)
        if fam == "exterior":
            d = _d(comps, n, k, False)
            return {"d": torch.stack(d, -1), "star": torch.stack(_star(d, n, k + 1, h), -1),
                    "codiff": torch.stack(_codiff(d, n, k + 1, h), -1)}
        total = [torch.zeros_like(c) for c in comps]
        if k < n:
            total = [t + v for t, v in zip(total, _codiff(_d(comps, n, k, False), n, k + 1, h))]
        if k > 0:
            total = [t + v for t, v in zip(total, _d(_codiff(comps, n, k, h), n, k - 1, False))]
        return torch.stack(total, -1)[tuple(slice(0, s - 1) for s in shape)].contiguous()
    if fam == "operator":
        st = prepare(case, seed)
        nx, ny, nz = _shape(case)
        mu = torch.ones(nz, ny, nx, device="cuda", dtype=torch.float64)
        lo = [max(1, s // 4 + (seed % 3)) for s in (nz, ny, nx)]
        mu[lo[0]:lo[0] + nz // 3, lo[1]:lo[1] + ny // 3, lo[2]:lo[2] + nx // 3] = 1000.0
        op = _CurlCurl([_coords(s) for s in (nx, ny, nz)], mu, m3.DEFAULT_GAUGE_PENALTY)
        return op.apply(st["a"].reshape(nz, ny, nx, 3)).reshape(-1)
    if fam == "solve2d":
        out = []
        for p in _problems2d(case, seed):
            nu = 1.0 / torch.from_numpy(p.node_mu()).cuda().reshape(p.ny, p.nx)
            b = torch.from_numpy(p.rhs()).cuda().reshape(p.ny, p.nx)
            out.append(_cg(lambda a: _k2_apply(a, nu), _k2_diagonal(nu), b, 16 * p.nx + 2000).reshape(-1))
        return out
    if fam == "solve3d":
        out = []
        for p in _problems3d(case, seed):
            nx, ny, nz = p.shape
            mu = torch.from_numpy(p.node_mu()).cuda().reshape(nz, ny, nx)
            op = _CurlCurl((p.x, p.y, p.z), mu, p.gamma)
            b = torch.from_numpy(p.rhs()).cuda().reshape(nz, ny, nx, 3)
            out.append(_cg(op.apply, op.diagonal(), b, 100 * nx + 2000).reshape(-1))
        return out
    p = torch.from_numpy(np.load(WEIGHTS).astype(np.float64)).cuda().requires_grad_(case["grad"])
    samples = [tuple(t.float().double() for t in s) for s in _network_inputs(case, seed)]
    if not case["grad"]:
        return torch.cat([_net_precondition(p, nu, b).reshape(-1) for nu, b, _ in samples])
    per = []
    for nu, b, x in samples:
        u = _net_precondition(p, nu, b)
        loss = 1.0 - (u * b).sum() ** 2 / ((u * _k2_apply(u, nu)).sum() * (x * b).sum())
        (loss / len(samples)).backward()
        per.append(loss.detach())
    per = torch.stack(per)
    return {"loss": per.mean().reshape(1), "per_sample": per, "grad": p.grad}
