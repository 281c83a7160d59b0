"""The builder's tile_lines option: whatever width a caller asks for, on plans of the register solve and
of the shared-memory tile, the plan reports it and the coefficients are those of the automatic
width, bit for bit (the same operations on every line). The fused step and the backward, which other
widths run as separate kernels, agree to rounding: 1e-13 of the largest value, 1e-12 for sums that the
transposed solve spreads."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P, H = 0, 1


@pytest.mark.parametrize("lines", [2, 4, 8, 16])
@pytest.mark.parametrize("degree,closure,nc,B,layout", [(3, P, 31, 2401, 0), (3, P, 200, 1203, 1), (5, H, 100, 700, 0), (5, H, 60, 31, 1), (3, P, 2500, 18, 0)])
def test_width_changes_no_result(lines, degree, closure, nc, B, layout):
    import ddc_b200 as D

    bs = D.UniformBSplines(degree, closure == P, 0.0, 1.0, nc)
    e = D.SplineEvaluator(bs)
    g = torch.Generator(device="cuda").manual_seed(nc)
    put = (lambda a: a.t().contiguous()) if layout else (lambda a: a)
    rand = lambda *s: put(torch.rand(s, dtype=torch.float64, device="cuda", generator=g))  # noqa: E731
    out = []
    for width in (0, lines):
        chunks = 32 if width == 16 and nc > 2000 else 0  # sixteen-line tiles take that many
        b = D.SplineBuilder(bs, None, closure, closure, tile_lines=width, chunks=chunks)
        if width:
            assert b.info.tile_lines == width
        g.manual_seed(nc)
        nd = b.s_nbv_xmin if closure == H else 0
        lo, hi = (rand(nd, B), rand(nd, B)) if nd else (None, None)
        v, x, gy, c = rand(b.npoints, B), rand(50, B), rand(50, B), rand(bs.size, B)
        b(c, v, lo, hi, dim=layout)
        y, c2 = torch.zeros_like(x), torch.zeros_like(c)
        b.build_and_evaluate(e, c2, v, x, y, lo, hi, dim=layout)
        gv, gx = torch.zeros_like(v), torch.zeros_like(x)
        b.build_and_evaluate_adjoint(e, x, c, gy, gv, gx, dim=layout)
        out.append((c, c2, y, gx, gv))
    exact = nc <= 2000  # the long line's chunk count follows its width, and with it the rounding
    for q, (a, w) in enumerate(zip(*out)):
        if exact and q < 2:
            assert torch.equal(a, w)
        else:
            assert (a - w).abs().max() <= (1e-13 if exact and q < 4 else 1e-12) * a.abs().max()
