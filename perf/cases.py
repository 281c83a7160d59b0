"""Performance cases of the batched spline builder / evaluator: what user programs call, over the
sizes, meshes, closures and layouts they call it with. Each case is one pass through the Python API;
inputs are synthetic (cosine families on [0, 1] with a seeded wave number and phase per line, plus a
little noise where real data would have it).

Kinds:
  two_calls   SplineBuilder.__call__, then SplineEvaluator (a value, or a first derivative)
  step        SplineBuilder.build_and_evaluate: the same in one call
  build       SplineBuilder.__call__ alone
  evaluate    SplineEvaluator alone, on given coefficients
  advect      SplineBuilder.advect: one semi-Lagrangian step
  train       autograd.build_evaluate forward, then the gradients of samples and coordinates
  tensor2d    SplineBuilder2D (periodic x Hermite), then SplineEvaluator2D at the feet
  tensor3d    SplineBuilder3D (periodic x Hermite x Greville), then SplineEvaluator3D
  uneven      UnevenBatch: problems of different size, degree, closure and mesh in one launch
"""
import math

import numpy as np
import torch

import ddc_b200 as D
from ddc_b200.autograd import build_evaluate

CLOSURE = {"periodic": D.SplineBuilderClosure.PERIODIC, "hermite": D.SplineBuilderClosure.HERMITE,
           "greville": D.SplineBuilderClosure.GREVILLE}
MOST_ROWS = 1 << 26  # rows x lines of the largest 1D case


def listed():
    return [
        # the smallest call: a plasma code's test grid, or one rank's last few lines; latency and launches count
        {"name": "small_two_calls", "kind": "two_calls", "degree": 3, "ncells": 64, "mesh": "uniform", "closure": "periodic",
         "lines": 16, "layout": "x_first", "points": 64, "where": "feet", "order": 0, "precision": "fp64"},
        # the 1000 x 1000 periodic cubic step of the benchmark: an ordinary 1D semi-Lagrangian problem
        {"name": "step_1000x1000", "kind": "step", "degree": 3, "ncells": 1000, "mesh": "uniform", "closure": "periodic",
         "lines": 1000, "layout": "x_first", "points": 1000, "where": "feet", "order": 0, "precision": "fp64"},
        # odd sizes throughout (no line pairs, ragged tiles): an irregular mesh, interpolated and differentiated
        {"name": "ragged_deriv", "kind": "two_calls", "degree": 3, "ncells": 333, "mesh": "perturbed", "closure": "greville",
         "lines": 1999, "layout": "x_first", "points": 517, "where": "random", "order": 1, "precision": "fp64"},
        # the benchmark's headline, its two calls apart: quintic, irregular mesh, Hermite ends, 2^16 lines
        {"name": "build_quintic", "kind": "build", "degree": 5, "ncells": 1024, "mesh": "perturbed", "closure": "hermite",
         "lines": 65536, "layout": "x_first", "points": 0, "where": "none", "order": 0, "precision": "fp64"},
        {"name": "deriv_quintic", "kind": "evaluate", "degree": 5, "ncells": 1024, "mesh": "perturbed", "closure": "hermite",
         "lines": 65536, "layout": "x_first", "points": 1024, "where": "random", "order": 1, "precision": "fp64"},
        # the interpolation dimension contiguous (the reference's (batch, x) order), clamped ends
        {"name": "x_last_16384", "kind": "two_calls", "degree": 3, "ncells": 1024, "mesh": "uniform", "closure": "hermite",
         "lines": 16384, "layout": "x_last", "points": 1025, "where": "feet", "order": 0, "precision": "fp64"},
        # advection along the first dimension of 512 x 512 x 64 fields, a velocity per row of the second
        {"name": "advect_512x512x64", "kind": "advect", "degree": 3, "ncells": 512, "mesh": "uniform", "closure": "periodic",
         "lines": 32768, "layout": "x_first", "points": 512, "where": "feet", "order": 0, "precision": "fp64"},
        # differentiating through the interpolation: forward and backward of a periodic cubic batch
        {"name": "train_cubic", "kind": "train", "degree": 3, "ncells": 1024, "mesh": "uniform", "closure": "periodic",
         "lines": 65536, "layout": "x_first", "points": 1024, "where": "random", "order": 0, "precision": "fp64"},
        # single-precision solves refined to double results, the library's other arithmetic
        {"name": "refine_cubic", "kind": "build", "degree": 3, "ncells": 512, "mesh": "perturbed", "closure": "hermite",
         "lines": 8192, "layout": "x_first", "points": 0, "where": "none", "order": 0, "precision": "fp32_refine"},
        # two-dimensional advection of 64 fields: build, then values at the feet
        {"name": "tensor2d_512x64", "kind": "tensor2d", "degree": 3, "ncells1": 512, "ncells2": 512, "fields": 64},
        # three-dimensional fields: build, then values at scattered points
        {"name": "tensor3d_96x16", "kind": "tensor3d", "degree": 3, "ncells1": 96, "ncells2": 96, "ncells3": 96, "fields": 16},
        # many small independent problems of every degree, closure and mesh
        {"name": "uneven_256", "kind": "uneven", "count": 256, "nmin": 32, "nmax": 4096, "pattern": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["two_calls", "step", "build", "evaluate", "advect", "train", "tensor2d", "tensor3d", "uneven"])
    degree = rng.choice([2, 3, 3, 4, 5])
    if kind == "uneven":
        nmin = _log(rng, 16, 128)
        return {"kind": kind, "count": _log(rng, 16, 256), "nmin": nmin, "nmax": _log(rng, 2 * nmin, 4096),
                "pattern": rng.randrange(1 << 20)}
    if kind == "tensor2d":
        n1, n2 = _log(rng, 24, 512), _log(rng, 24, 512)
        return {"kind": kind, "degree": degree, "ncells1": n1, "ncells2": n2, "fields": _log(rng, 1, 64)}
    if kind == "tensor3d":
        n = [_log(rng, 12, 96) for _ in range(3)]
        return {"kind": kind, "degree": degree, "ncells1": n[0], "ncells2": n[1], "ncells3": n[2], "fields": _log(rng, 1, 16)}
    ncells = _log(rng, 24, 4096)
    lines = _log(rng, 1, min(65536, MOST_ROWS // (2 * ncells)))
    points = max(1, int(ncells * rng.uniform(0.5, 1.5)))
    mesh = rng.choice(["uniform", "perturbed"])
    closure = rng.choice(["periodic", "hermite", "greville"])
    layout = rng.choice(["x_first", "x_first", "x_last", "x_mid"])
    order = rng.choice([0, 1])
    where = "random" if order or rng.random() < 0.5 else "feet"
    precision = "fp64"
    if kind == "build":
        points, where, order = 0, "none", 0
        precision = rng.choice(["fp64", "fp64", "fp32_refine"])
    elif kind == "advect":
        where, order = "feet", 0
    elif kind == "train":
        layout, order = "x_first", 0
    return {"kind": kind, "degree": degree, "ncells": ncells, "mesh": mesh, "closure": closure, "lines": lines,
            "layout": layout, "points": points, "where": where, "order": order, "precision": precision}


# ---- the bases: knots and interpolation points, written out here so that exact() needs no library code ----

class Axis:
    """One dimension: break points, knots and Greville points of a basis on [0, 1]."""

    def __init__(self, degree, ncells, closure, breaks=None):
        self.d, self.nc, self.closure = degree, ncells, closure
        self.periodic = closure == "periodic"
        self.uniform = breaks is None
        self.nb = degree // 2 if closure == "hermite" else 0  # derivative rows per side
        self.odd = degree % 2
        h = 1.0 / ncells
        self.breaks = np.arange(ncells + 1) * h if breaks is None else breaks
        self.breaks[-1] = 1.0
        self.size = ncells + degree
        self.n = ncells if self.periodic else self.size
        self.npoints = self.n - 2 * self.nb
        d, b = degree, self.breaks
        if self.uniform:
            self.knots = np.arange(-d, ncells + d + 1) * h
            self.knots[d:d + ncells + 1] = b
        elif self.periodic:
            self.knots = np.concatenate([b[ncells - d:ncells] - 1.0, b, b[1:d + 1] + 1.0])
        else:
            self.knots = np.concatenate([np.zeros(d), b, np.ones(d)])
        self.points = self._points(h)

    def _points(self, h):
        d, nc, b = self.d, self.nc, self.breaks
        if not self.uniform:
            g = np.array([self.knots[i + 1:i + 1 + d].sum() / d for i in range(self.size)])
            if self.periodic:
                g = g[:nc]
                return np.concatenate([g[g >= 0.0], g[g < 0.0] + 1.0])
            return g[self.nb:self.nb + self.npoints]
        shift = 0.0 if d % 2 else 0.5 * h
        if self.periodic or self.nb:
            return shift + np.arange(self.npoints) * h
        p = np.zeros(self.npoints)
        half = d // 2 + 1
        for i in range(1, nc):
            p[half + i - 1] = shift + i * h
        for i in range(half):
            p[i] = b[1:i + 1].sum() / d
            p[self.npoints - 1 - i] = ((d - i) + b[nc - i:nc].sum()) / d
        return p

    def bsplines(self):
        if self.uniform:
            return D.UniformBSplines(self.d, self.periodic, 0.0, 1.0, self.nc)
        return D.NonUniformBSplines(self.d, self.periodic, self.breaks)

    def builder(self, bsplines, precision="fp64", **kw):
        c = CLOSURE[self.closure]
        return D.SplineBuilder(bsplines, None, c, c, precision=precision, **kw)

    def derivs(self, k, ph, x):
        """The derivative rows of a cosine family at an end: orders odd .. odd + nb - 1."""
        if not self.nb:
            return None
        return torch.stack([_cosines(torch.full((1,), x, dtype=torch.float64, device=k.device), k, ph, o + self.odd)[0]
                            for o in range(self.nb)])

    # -- exact() only: everything below is plain 64-bit torch --

    def basis(self, x, order=0):
        """First B-spline and the d+1 values of the order-th derivative of the B-splines at x."""
        d = self.d
        t = torch.from_numpy(self.knots).to(x.device)
        c = torch.searchsorted(t[d:d + self.nc + 1].contiguous(), x.contiguous(), right=True) - 1
        c = c.clamp(0, self.nc - 1)
        K = c + d
        v = [torch.ones_like(x)]
        p = d - order
        for j in range(p):
            nv, saved = [], torch.zeros_like(x)
            for r in range(j + 1):
                hi, lo = t[K + r + 1], t[K + r - j]
                w = v[r] / (hi - lo)
                nv.append(saved + (hi - x) * w)
                saved = (x - lo) * w
            v = nv + [saved]
        for q in range(p + 1, d + 1):
            nv = []
            for i in range(q + 1):  # B-spline with first knot K - q + i
                f = K - q + i
                a = v[i - 1] / (t[f + q] - t[f]) if i >= 1 else torch.zeros_like(x)
                b = v[i] / (t[f + q + 1] - t[f + 1]) if i < q else torch.zeros_like(x)
                nv.append(q * (a - b))
            v = nv
        return c, v

    def matrix(self, dev):
        """The interpolation matrix, derivative rows scaled by the cell width to their order."""
        rows = [(torch.zeros(1, dtype=torch.float64, device=dev), o + self.odd) for o in range(self.nb)]
        rows += [(torch.from_numpy(self.points).to(dev), 0)]
        rows += [(torch.ones(1, dtype=torch.float64, device=dev), o + self.odd) for o in range(self.nb)]
        A = torch.zeros(self.n, self.n, dtype=torch.float64, device=dev)
        at = 0
        for x, o in rows:
            j, v = self.basis(x, o)
            for i, w in enumerate(v):
                A[torch.arange(at, at + len(x), device=dev), (j + i) % self.n] += w / self.nc ** o
            at += len(x)
        return A

    def solve(self, vals, lo=None, hi=None):
        """Spline coefficients (size, ...) of samples (npoints, ...) along the first dimension."""
        tail = vals.shape[1:]
        rhs = [vals.reshape(self.npoints, -1)]
        if self.nb:
            s = torch.tensor([float(self.nc) ** -(o + self.odd) for o in range(self.nb)], dtype=torch.float64, device=vals.device)
            rhs = [lo.reshape(self.nb, -1) * s[:, None]] + rhs + [hi.reshape(self.nb, -1) * s[:, None]]
        c = torch.linalg.solve(self.matrix(vals.device), torch.cat(rhs))
        if self.periodic:
            c = torch.cat([c, c[:self.d]])
        return c.reshape(self.size, *tail)

    def place(self, x):
        return x - torch.floor(x) if self.periodic else x.clamp(0.0, 1.0)


def _mesh(ncells, seed):
    """Break points of an irregular mesh: a uniform one with its inner points moved by up to 0.3 cells."""
    h = 1.0 / ncells
    b = np.arange(ncells + 1) * h
    b[1:-1] += (np.random.RandomState(seed % (1 << 31)).rand(ncells - 1) - 0.5) * 0.6 * h
    return b


def _axis(case, seed):
    return Axis(case["degree"], case["ncells"], case["closure"],
                _mesh(case["ncells"], seed) if case["mesh"] == "perturbed" else None)


def _cosines(x, k, ph, order=0):
    w = 2 * math.pi * k
    return w ** order * torch.cos(0.5 * math.pi * order + w * x.reshape(-1, *([1] * k.dim())) + ph)


def _rand(g, *shape):
    return torch.rand(*shape, dtype=torch.float64, device=g.device, generator=g)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


class Layout:
    """(rows, lines) arrays in the case's order: x_first (x, batch), x_last (batch, x), x_mid (b1, x, b2)."""

    def __init__(self, case):
        self.kind = case["layout"]
        self.lines = case["lines"]
        self.b2 = next(q for q in (16, 8, 4, 2, 1) if self.lines % q == 0)
        self.dim = 0 if self.kind == "x_first" else 1

    def put(self, a):
        if a is None or self.kind == "x_first":
            return a
        if self.kind == "x_last":
            return a.t().contiguous()
        return a.reshape(a.shape[0], -1, self.b2).transpose(0, 1).contiguous()

    def empty(self, n):
        shape = {"x_first": (n, self.lines), "x_last": (self.lines, n), "x_mid": (self.lines // self.b2, n, self.b2)}[self.kind]
        return torch.empty(shape, dtype=torch.float64, device="cuda")


def _inputs_1d(case, seed):
    """The canonical (rows, lines) inputs of a 1D case, the same for prepare() and exact()."""
    g = _generator(seed)
    ax = _axis(case, seed)
    B, m = case["lines"], case["points"]
    k = torch.floor(_rand(g, B) * 8) + 1
    ph = _rand(g, B) * 2 * math.pi
    i = {"ax": ax}
    pts = torch.from_numpy(ax.points).cuda()
    if case["kind"] == "evaluate":
        i["coefs"] = _cosines(torch.linspace(0, 1, ax.size, dtype=torch.float64, device="cuda"), k, ph)
        if ax.periodic:
            i["coefs"][ax.nc:] = i["coefs"][:ax.d]
    else:
        i["vals"] = _cosines(pts, k, ph)
        i["lo"], i["hi"] = ax.derivs(k, ph, 0.0), ax.derivs(k, ph, 1.0)
    if case["kind"] == "advect":
        i["v"] = 2 * _rand(g, (B + 63) // 64) - 1  # a velocity for every 64 lines
        i["dt"] = 0.5 / ax.nc
    elif case["where"] == "random":
        i["x"] = _rand(g, m, B)
    elif case["where"] == "feet":
        base = torch.linspace(0, 1, m + 1, dtype=torch.float64, device="cuda")[:m] if ax.periodic else \
            torch.linspace(0, 1, m, dtype=torch.float64, device="cuda")
        i["x"] = ax.place(base[:, None] + (_rand(g, 1, B) - 0.5) / ax.nc + 0.1 * (_rand(g, m, B) - 0.5) / ax.nc)
    if case["kind"] == "train":
        i["g"] = 2 * _rand(g, m, B) - 1
    return i


def _inputs_tensor(case, seed):
    """Samples (np1, np2[, np3], fields), the Hermite slabs of dimension 2, and the evaluation points."""
    g = _generator(seed)
    two = case["kind"] == "tensor2d"
    d, F = case["degree"], case["fields"]
    axes = [Axis(d, case["ncells1"], "periodic"), Axis(d, case["ncells2"], "hermite")]
    if not two:
        axes.append(Axis(d, case["ncells3"], "greville"))
    p = [torch.from_numpy(a.points).cuda() for a in axes]
    amp = 0.5 + 1.5 * _rand(g, F)
    f1, f2 = torch.sin(2 * math.pi * p[0]), torch.cos(math.pi * p[1])
    base = f1[:, None] * f2[None, :]
    if not two:
        base = base[:, :, None] * torch.exp(-p[2])[None, None, :]
    shape = base.shape + (F,)
    vals = base[..., None] * amp + 0.01 * torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
    lo = 0.1 * _rand(g, shape[0], axes[1].nb, *shape[2:])
    hi = 0.1 * _rand(g, shape[0], axes[1].nb, *shape[2:])
    if two:  # the feet of a shear flow along dimension 1
        v = 2 * _rand(g, len(p[1])) - 1
        x = torch.stack([(p[0][:, None] - v[None, :] * 0.5 / axes[0].nc), p[1][None, :].expand(len(p[0]), -1)], dim=-1)
    else:
        x = _rand(g, max(1, vals[..., 0].numel() // 4), 3)
    return {"axes": axes, "vals": vals, "lo": lo, "hi": hi, "x": x.reshape(-1, len(axes))}


def _inputs_uneven(case, seed):
    """The problems: their bases from the case's pattern, their data from the seed."""
    shape, r = np.random.RandomState(case["pattern"]), np.random.RandomState(seed % (1 << 31))
    probs = []
    for q in range(case["count"]):
        n = int(np.exp(shape.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))
        closure = ("periodic", "hermite", "greville")[shape.randint(3)]
        ax = Axis(int(shape.randint(1, 6)), n, closure, _mesh(n, case["pattern"] + q) if shape.rand() < 0.5 else None)
        k, ph = float(r.randint(1, 9)), float(r.rand() * 2 * np.pi)
        w = 2 * np.pi * k
        f = lambda x, o=0: w ** o * np.cos(0.5 * np.pi * o + w * x + ph)  # noqa: E731
        ends = [np.array([f(x, o + ax.odd) for o in range(ax.nb)]) for x in (0.0, 1.0)]
        probs.append((ax, f(ax.points), ends[0], ends[1], r.rand(n)))
    return probs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "uneven":
        probs = _inputs_uneven(case, seed)
        builders, evaluators = [], []
        for ax, *_ in probs:
            bs = ax.bsplines()
            # one line each: whole warps of chunks, at most 16 rows per chunk
            chunks = min(512, 32 * max(1, -(-ax.size // 512)))
            builders.append(ax.builder(bs, tile_lines=2, chunks=chunks))
            evaluators.append(D.SplineEvaluator(bs))
        cat = lambda q: torch.from_numpy(np.concatenate([p[q] for p in probs])).cuda()  # noqa: E731
        batch = D.UnevenBatch(builders, evaluators, [len(p[4]) for p in probs])
        new = lambda n: torch.empty(n, dtype=torch.float64, device="cuda")  # noqa: E731
        return {"kind": kind, "batch": batch, "vals": cat(1), "lo": cat(2), "hi": cat(3), "x": cat(4),
                "coefs": new(sum(p[0].size for p in probs)), "out": new(sum(len(p[4]) for p in probs))}
    if kind in ("tensor2d", "tensor3d"):
        i = _inputs_tensor(case, seed)
        axes, F = i["axes"], case["fields"]
        bs = [a.bsplines() for a in axes]
        one = [a.builder(b) for a, b in zip(axes, bs)]
        ev = [D.SplineEvaluator(b, D.Extrapolation.CONSTANT, D.Extrapolation.CONSTANT) for b in bs]
        build = (D.SplineBuilder2D if kind == "tensor2d" else D.SplineBuilder3D)(*one)
        new = lambda *n: torch.empty(n, dtype=torch.float64, device="cuda")  # noqa: E731
        m = len(i["x"])
        return {"kind": kind, "builder": build, "vals": i["vals"].contiguous(), "lo": i["lo"], "hi": i["hi"],
                "evaluator": (D.SplineEvaluator2D if kind == "tensor2d" else D.SplineEvaluator3D)(*ev),
                "x": i["x"][:, None, :].expand(m, F, len(axes)).contiguous(), "coefs": new(*[a.size for a in axes], F),
                "out": new(m, F), "workspace": new(build.workspace_bytes(F) // 8 + 1)}
    i = _inputs_1d(case, seed)
    ax, lay = i["ax"], Layout(case)
    bs = ax.bsplines()
    s = {"kind": kind, "dim": lay.dim, "order": case["order"], "bsplines": bs}
    if kind != "evaluate":
        s["builder"] = ax.builder(bs, case["precision"])
        s["vals"], s["lo"], s["hi"] = lay.put(i["vals"]), lay.put(i["lo"]), lay.put(i["hi"])
    if kind != "build":
        s["evaluator"] = D.SplineEvaluator(bs, D.Extrapolation.CONSTANT, D.Extrapolation.CONSTANT)
    if kind == "advect":
        s["v"], s["dt"], s["out"] = i["v"], i["dt"], torch.empty_like(s["vals"])
        return s
    if kind == "train":
        s["vals"].requires_grad_(True)
        s["x"], s["g"] = i["x"].requires_grad_(True), i["g"]
        return s
    s["coefs"] = lay.put(i["coefs"]) if kind == "evaluate" else lay.empty(ax.size)
    if kind != "build":
        s["x"], s["out"] = lay.put(i["x"]), lay.empty(case["points"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "uneven":
        s["batch"](s["vals"], s["lo"], s["hi"], s["coefs"], s["x"], s["out"])
        return {"coefs": s["coefs"], "values": s["out"]}
    if kind in ("tensor2d", "tensor3d"):
        names = ("derivs_min2", "derivs_max2")
        s["builder"](s["coefs"], s["vals"], workspace=s["workspace"], **dict(zip(names, (s["lo"], s["hi"]))))
        s["evaluator"](s["out"], s["x"], s["coefs"])
        return {"coefs": s["coefs"], "values": s["out"]}
    dim = s["dim"]
    if kind == "advect":
        s["builder"].advect(s["evaluator"], s["out"], s["vals"], s["dt"], s["v"], s["lo"], s["hi"], velocity_div=64, dim=dim)
        return {"values": s["out"]}
    if kind == "train":
        y = build_evaluate(s["vals"], s["x"], s["builder"], s["evaluator"], 0, s["lo"], s["hi"])
        gv, gx = torch.autograd.grad(y, (s["vals"], s["x"]), s["g"])
        return {"values": y.detach(), "g_vals": gv, "g_coords": gx}
    if kind == "step":
        s["builder"].build_and_evaluate(s["evaluator"], s["coefs"], s["vals"], s["x"], s["out"], s["lo"], s["hi"],
                                        order=s["order"], dim=dim)
        return {"coefs": s["coefs"], "values": s["out"]}
    if kind in ("build", "two_calls"):
        s["builder"](s["coefs"], s["vals"], s["lo"], s["hi"], dim=dim)
    if kind in ("evaluate", "two_calls"):
        if s["order"]:
            s["evaluator"].deriv(s["order"], s["out"], s["x"], s["coefs"], dim=dim)
        else:
            s["evaluator"](s["out"], s["x"], s["coefs"], dim=dim)
    if kind == "build":
        return {"coefs": s["coefs"]}
    return {"values": s["out"]} if kind == "evaluate" else {"coefs": s["coefs"], "values": s["out"]}


def work(case):
    kind = case["kind"]
    if kind == "uneven":
        rows = case["count"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        return {"bytes": 8 * 4 * rows, "flops": 60 * rows}
    d = case["degree"]
    band = 8 * (d // 2) + 2           # one banded forward and backward substitution, per row
    point = 3 * d * (d + 1) // 2 + 2 * (d + 1)
    if kind in ("tensor2d", "tensor3d"):
        ax = [Axis(d, case["ncells1"], "periodic"), Axis(d, case["ncells2"], "hermite")]
        ax += [Axis(d, case["ncells3"], "greville")] if kind == "tensor3d" else []
        N, F = len(ax), case["fields"]
        samples = math.prod(a.npoints for a in ax) * F
        slabs = samples // ax[1].npoints * 2 * ax[1].nb
        coefs = math.prod(a.size for a in ax) * F
        m = samples if N == 2 else max(1, samples // F // 4) * F
        return {"bytes": 8 * (samples + slabs + 2 * coefs + (N + 1) * m),
                "flops": N * band * coefs + m * (2 * (d + 1) ** N + N * point)}
    ax = Axis(d, case["ncells"], case["closure"])
    B, m = case["lines"], case["points"]
    build = (ax.n + ax.size) * B
    if kind == "build":
        return {"bytes": 8 * build, "flops": band * ax.n * B}
    if kind == "evaluate":
        return {"bytes": 8 * (ax.size + 2 * m) * B, "flops": point * m * B}
    if kind == "advect":
        m = ax.npoints
        return {"bytes": 8 * (ax.n + m) * B, "flops": (band * ax.n + point * m) * B}
    if kind == "train":  # forward, then backward: x, g_y and the coefficients in, g_x and g_vals out
        return {"bytes": 8 * (build + 2 * m * B + (3 * m + ax.size + ax.n) * B), "flops": 2 * (band * ax.n + 2 * point * m) * B}
    return {"bytes": 8 * (build + 2 * m * B), "flops": (band * ax.n + point * m) * B}


# ---- what run() returns, in plain 64-bit torch ----

def _values(ax, coefs, x, order=0):
    """The order-th derivative of the splines with coefficients (size, lines) at x (m, lines)."""
    y = torch.empty_like(x)
    step = max(1, (1 << 24) // max(1, x.shape[1]))
    for q in range(0, x.shape[0], step):
        j, v = ax.basis(x[q:q + step], order)
        y[q:q + step] = sum(torch.gather(coefs, 0, j + i) * w for i, w in enumerate(v))
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "uneven":
        coefs, values = [], []
        for ax, f, lo, hi, x in _inputs_uneven(case, seed):
            up = lambda a: torch.from_numpy(a).cuda()[:, None]  # noqa: E731
            c = ax.solve(up(f), up(lo), up(hi))
            coefs.append(c[:, 0])
            values.append(_values(ax, c, up(x))[:, 0])
        return {"coefs": torch.cat(coefs), "values": torch.cat(values)}
    if kind in ("tensor2d", "tensor3d"):
        i = _inputs_tensor(case, seed)
        axes = i["axes"]
        c, lo, hi = (axes[0].solve(i[n]) if i[n].numel() else i[n] for n in ("vals", "lo", "hi"))
        if not axes[1].nb:
            lo = hi = None
        flip = lambda a, q: None if a is None else a.transpose(0, q).contiguous()  # noqa: E731
        c = flip(axes[1].solve(flip(c, 1), flip(lo, 1), flip(hi, 1)), 1)
        if len(axes) == 3:
            c = flip(axes[2].solve(flip(c, 2)), 2)
        b = [a.basis(a.place(i["x"][:, q])) for q, a in enumerate(axes)]
        flat = c.reshape(-1, case["fields"])
        y = torch.zeros(len(i["x"]), case["fields"], dtype=torch.float64, device="cuda")
        stencil = [()]
        for a in axes:
            stencil = [s + (q,) for s in stencil for q in range(a.d + 1)]
        for s in stencil:
            row, w = 0, 1.0
            for q, a in enumerate(axes):
                row = row * a.size + b[q][0] + s[q]
                w = w * b[q][1][s[q]]
            y += flat[row] * w[:, None]
        return {"coefs": c, "values": y}
    i = _inputs_1d(case, seed)
    ax, lay, o = i["ax"], Layout(case), case["order"]
    c = i["coefs"] if kind == "evaluate" else ax.solve(i["vals"], i["lo"], i["hi"])
    if kind == "build":
        return {"coefs": lay.put(c)}
    if kind == "advect":
        v = i["v"].repeat_interleave(64)[:case["lines"]]
        x = ax.place(torch.from_numpy(ax.points).cuda()[:, None] - v[None, :] * i["dt"])
        return {"values": lay.put(_values(ax, c, x))}
    y = _values(ax, c, i["x"], o)
    if kind == "evaluate":
        return {"values": lay.put(y)}
    if kind == "train":
        gc = torch.zeros_like(c)
        j, v = ax.basis(i["x"])
        for q, w in enumerate(v):
            gc.scatter_add_(0, j + q, i["g"] * w)
        if ax.periodic:
            gc[:ax.d] += gc[ax.nc:]
        r = torch.linalg.solve(ax.matrix("cuda").t(), gc[:ax.n])
        return {"values": y, "g_vals": r[ax.nb:ax.nb + ax.npoints], "g_coords": i["g"] * _values(ax, c, i["x"], 1)}
    return {"coefs": lay.put(c), "values": lay.put(y)}
