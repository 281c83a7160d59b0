"""The fused kernels over the register solve where their tiles change: the advection step with Hermite and
Greville ends (feet that leave the domain, both extrapolation rules), every degree, both layouts, and
batches of one tile, of many and of more than the blocks that run at once (the tile loop comes round);
and the backward without a period, orders 0 and 1, with and without coordinate cotangents, at the same
batches. Against the oracle on 29 lines that the batch repeats, <= 1e-12 of the largest value (10
cond(A) eps for an ill-conditioned system)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P, H, G = 0, 1, 3
LINES = 29


def plan(D, O, degree, closure, nc, ex):
    bs = D.UniformBSplines(degree, closure == P, 0.0, 1.0, nc)
    obs = O.BSplines(degree, closure == P, rmin=0.0, rmax=1.0, ncells=nc)
    b = D.SplineBuilder(bs, None, closure, closure)
    ob = O.Builder(obs, b.interpolation_points, closure, closure)
    tol = max(1e-12, 10 * np.linalg.cond(ob.matrix()) * np.finfo(float).eps)
    return bs, obs, b, ob, D.SplineEvaluator(bs, *ex), tol


def spread(a, B, layout):
    """Line j of the batch: column 7 j mod 29 of a."""
    if a is None or a.size == 0:
        return None
    t = torch.from_numpy(np.ascontiguousarray(a[..., np.arange(B) * 7 % LINES])).cuda()
    return t.t().contiguous() if layout and t.ndim == 2 else t


def close(got, want, layout, tol):
    got = got.cpu().numpy()
    got = got.T if layout else got
    want = want[:, np.arange(got.shape[1]) * 7 % LINES]
    return np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("layout,B", [(0, 5), (0, 2401), (1, 2401), (0, 10001), (1, 10000)])
@pytest.mark.parametrize("degree,closure,nc,ex", [(3, H, 100, (1, 1)), (5, H, 300, (2, 2)), (2, G, 40, (1, 2)), (4, G, 64, (2, 1)), (4, P, 31, (0, 0)),
                                                  (1, G, 17, (2, 2))])
def test_advection(oracle_mod, degree, closure, nc, ex, layout, B):
    import ddc_b200 as D

    O = oracle_mod
    bs, obs, b, ob, e, tol = plan(D, O, degree, closure, nc, ex)
    rng = np.random.default_rng(nc)
    pts = b.interpolation_points
    nd = b.s_nbv_xmin if closure == H else 0
    f, lo, hi = rng.standard_normal((pts.size, LINES)), rng.standard_normal((nd, LINES)), rng.standard_normal((nd, LINES))
    v, dt = rng.uniform(-2.0, 2.0, LINES), 0.03
    c = ob(f, lo if nd else None, hi if nd else None)
    want = O.evaluate(obs, pts[:, None] - dt * v[None, :], c, ex_lo=ex[0], ex_hi=ex[1])
    vals = spread(f, B, layout)
    out = torch.full_like(vals, float("nan"))
    coefs = torch.full((B, bs.size) if layout else (bs.size, B), float("nan"), dtype=torch.float64, device="cuda")
    assert b.advect(e, out, vals, dt, spread(v, B, 0), spread(lo, B, layout), spread(hi, B, layout), spline=coefs, dim=layout)
    assert close(out, want, layout, tol) and close(coefs, c, layout, tol)


@pytest.mark.parametrize("B", [5, 2401, 10001])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("degree,closure,nc", [(3, H, 100), (5, H, 250), (2, G, 40), (4, G, 64), (3, P, 31)])
def test_backward(oracle_mod, degree, closure, nc, order, B):
    import ddc_b200 as D

    O = oracle_mod
    bs, obs, b, ob, e, tol = plan(D, O, degree, closure, nc, (1, 2) if closure != P else (0, 0))
    rng = np.random.default_rng(nc + order)
    m = 33
    x = rng.uniform(-0.1, 1.1, (m, LINES)) if order == 0 else rng.uniform(0.0, 1.0, (m, LINES))
    gy, c = rng.standard_normal((m, LINES)), rng.standard_normal((bs.size, LINES))
    # coefficients from samples: one oracle build per unit sample; values: one evaluation per unit coefficient
    nd = b.s_nbv_xmin if closure == H else 0
    zero = np.zeros((nd, b.npoints)) if nd else None
    M = ob(np.eye(b.npoints), zero, zero)
    dy, gc = np.zeros((m, LINES)), np.zeros((bs.size, LINES))
    kw = dict(ex_lo=1, ex_hi=2) if closure != P else dict(ex_lo=0, ex_hi=0)
    for j in range(LINES):
        E = O.evaluate(obs, np.repeat(x[:, j:j + 1], bs.size, axis=1), np.eye(bs.size), order=order or None, **kw)
        gc[:, j] = E.T @ gy[:, j]
        xi = x[:, j] - np.floor(x[:, j]) if closure == P else x[:, j]
        inside = (xi >= 0.0) & (xi <= 1.0)
        if degree > order:
            dy[:, j] = np.where(inside, O.evaluate(obs, np.clip(xi, 0.0, 1.0)[:, None], c[:, j:j + 1], order=order + 1)[:, 0], 0.0)
    want_v, want_x = M.T @ gc, gy * dy
    for coords in (True, False):
        gv = torch.full((b.npoints, B), float("nan"), dtype=torch.float64, device="cuda")
        gx = torch.full((m, B), float("nan"), dtype=torch.float64, device="cuda") if coords else None
        fused = b.build_and_evaluate_adjoint(e, spread(x, B, 0), spread(c, B, 0) if coords else None, spread(gy, B, 0), gv, gx, order=order)
        assert fused
        assert close(gv, want_v, 0, tol)
        assert not coords or close(gx, want_x, 0, 1e-12)
