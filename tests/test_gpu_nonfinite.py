"""Coordinates that are not finite: the value there is NaN (a NaN anywhere, an infinity on a periodic
basis, which has no point for it), every other point of the call is what it is without them, and no index
leaves its array. Through every kernel that locates points: the evaluators of one and more dimensions,
the fused step, the advection step (a NaN velocity) and the backward."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P, H, G = 0, 1, 3
NAN, INF = math.nan, math.inf


def basis(D, degree, periodic, uniform, nc):
    br = np.linspace(0.0, 1.0, nc + 1)
    br[1:-1] += np.random.default_rng(nc).uniform(-0.3, 0.3, nc - 1) / nc
    return D.UniformBSplines(degree, periodic, 0.0, 1.0, nc) if uniform else D.NonUniformBSplines(degree, periodic, br)


def spoil(x, bad, g):
    """x with about one in twenty coordinates replaced by `bad`, and where."""
    where = torch.rand(x.shape, dtype=torch.float64, device="cuda", generator=g) < 0.05
    where.view(-1)[0] = where.view(-1)[-1] = True
    return torch.where(where, torch.full_like(x, bad), x), where


def check(got, ref, where):
    assert torch.isnan(got[where]).all()
    assert torch.equal(got[~where], ref[~where])


def rand(g, *shape):
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=g)


@pytest.mark.parametrize("layout,B", [(0, 13), (1, 13), (1, 1300)])
@pytest.mark.parametrize("degree,periodic,uniform,nc", [(3, True, True, 40), (3, False, True, 40), (5, False, False, 40), (3, False, True, 10000)])
def test_evaluation(layout, B, degree, periodic, uniform, nc):
    import ddc_b200 as D

    g = torch.Generator(device="cuda").manual_seed(nc + B)
    B = min(B, 13) if nc > 1000 else B
    bs = basis(D, degree, periodic, uniform, nc)
    e = D.SplineEvaluator(bs, D.Extrapolation.CONSTANT, D.Extrapolation.NULL)
    put = (lambda a: a.t().contiguous()) if layout else (lambda a: a)
    c, x = put(rand(g, bs.size, B)), put(rand(g, 70, B))
    for bad in (NAN, INF) if periodic else (NAN,):
        xb, where = spoil(x, bad, g)
        for order in (0, 1, 2):
            if order and math.isinf(bad):
                continue
            run = (lambda o, q: e.deriv(order, o, q, c, dim=layout)) if order else (lambda o, q: e(o, q, c, dim=layout))
            got, ref = torch.zeros_like(x), torch.zeros_like(x)
            run(got, xb)
            run(ref, x)
            check(got, ref, where)


@pytest.mark.parametrize("closure,uniform,degree", [(P, True, 3), (H, True, 5), (G, True, 2), (P, False, 3)])
def test_fused_step_advection_and_backward(closure, uniform, degree):
    import ddc_b200 as D

    g = torch.Generator(device="cuda").manual_seed(degree)
    nc, B = 100, 37
    bs = basis(D, degree, closure == P, uniform, nc)
    b = D.SplineBuilder(bs, None, closure, closure)
    e = D.SplineEvaluator(bs, D.Extrapolation.CONSTANT, D.Extrapolation.NULL)
    nd = b.s_nbv_xmin if closure == H else 0
    lo, hi = (rand(g, nd, B), rand(g, nd, B)) if nd else (None, None)
    vals, x, c = rand(g, b.npoints, B), rand(g, 90, B), rand(g, bs.size, B)
    xb, where = spoil(x, NAN, g)
    got, ref = torch.zeros_like(x), torch.zeros_like(x)
    b.build_and_evaluate(e, c, vals, xb, got, lo, hi)
    b.build_and_evaluate(e, c, vals, x, ref, lo, hi)
    check(got, ref, where)
    v = rand(g, B) - 0.5
    vb = v.clone()
    vb[::9] = NAN
    fa, fb = torch.zeros_like(vals), torch.zeros_like(vals)
    b.advect(e, fa, vals, 0.01, vb, lo, hi)
    b.advect(e, fb, vals, 0.01, v, lo, hi)
    check(fa, fb, torch.isnan(vb)[None, :].expand_as(fa))
    # backward: NaN coordinate cotangents there; sample cotangents of the other lines as without
    xb = x.clone()
    xb[5, ::9] = NAN
    gy, out = rand(g, 90, B), []
    for q in (xb, x):
        gv, gx = torch.zeros_like(vals), torch.zeros_like(x)
        b.build_and_evaluate_adjoint(e, q, c, gy, gv, gx)
        out.append((gv, gx))
    check(out[0][1], out[1][1], torch.isnan(xb))
    spoiled = torch.isnan(xb).any(dim=0)
    assert torch.isnan(out[0][0][:, spoiled]).any(dim=0).all()
    torch.testing.assert_close(out[0][0][:, ~spoiled], out[1][0][:, ~spoiled], rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("ndims,uniform,degrees", [(2, True, (3, 3)), (2, False, (3, 3)), (3, True, (3, 3, 3)), (3, True, (3, 2, 3)), (3, False, (2, 2, 2))])
@pytest.mark.parametrize("fields", [1, 2, 7])
def test_tensor_evaluation(ndims, uniform, degrees, fields):
    import ddc_b200 as D

    g = torch.Generator(device="cuda").manual_seed(fields)
    bases = [basis(D, d, q == 0, uniform, n) for q, (d, n) in enumerate(zip(degrees, (12, 9, 8)))]
    evs = [D.SplineEvaluator(s, D.Extrapolation.CONSTANT, D.Extrapolation.NULL) for s in bases]
    e = (D.SplineEvaluator2D if ndims == 2 else D.SplineEvaluator3D)(*evs)
    c, x = rand(g, *[s.size for s in bases], fields), rand(g, 300, fields, ndims)
    for shared in (False, True):
        if shared:
            x = x[:, :1].expand_as(x).contiguous()
        for q in range(ndims):
            xb, where = spoil(x[..., q], NAN, g)
            xb = torch.cat([x[..., :q], xb[..., None], x[..., q + 1:]], dim=-1).contiguous()
            got, ref = torch.zeros_like(x[..., 0].contiguous()), torch.zeros_like(x[..., 0].contiguous())
            e(got, xb, c)
            e(ref, x, c)
            check(got, ref, where)
