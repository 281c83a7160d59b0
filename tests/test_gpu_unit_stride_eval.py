"""Evaluation with the evaluated dimension contiguous: enough lines take one warp per line, few lines the
line tiles. Both compute a point from the same coefficients with the same operations, so the values of
a large batch have to equal, bit for bit, those of its lines evaluated a few at a time and those of the
batch-contiguous layout (which the oracle tests cover)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("degree,uniform,periodic", [(3, True, True), (3, True, False), (5, False, False), (2, False, True)])
@pytest.mark.parametrize("nc,m,B", [(6, 1, 1184), (31, 32, 1185), (97, 131, 1201), (700, 33, 1190), (1500, 200, 1184)])
def test_lines_alone_and_together(order, degree, uniform, periodic, nc, m, B):
    import ddc_b200 as D

    br = np.linspace(0.0, 1.0, nc + 1)
    br[1:-1] += np.random.default_rng(nc).uniform(-0.3, 0.3, nc - 1) / nc
    bs = D.UniformBSplines(degree, periodic, 0.0, 1.0, nc) if uniform else D.NonUniformBSplines(degree, periodic, br)
    e = D.SplineEvaluator(bs, D.Extrapolation.CONSTANT, D.Extrapolation.NULL)
    g = torch.Generator(device="cuda").manual_seed(m)
    c = torch.randn((B, bs.size), dtype=torch.float64, device="cuda", generator=g)
    x = torch.rand((B, m), dtype=torch.float64, device="cuda", generator=g)
    if order == 0:
        x = x * 1.2 - 0.1
    run = (lambda o, p, q, **kw: e.deriv(order, o, p, q, **kw)) if order else e
    y = torch.full((B, m), float("nan"), dtype=torch.float64, device="cuda")
    run(y, x, c, dim=1)
    few = torch.full((40, m), float("nan"), dtype=torch.float64, device="cuda")
    run(few, x[-40:], c[-40:], dim=1)
    assert torch.equal(y[-40:], few)
    first = torch.full((m, B), float("nan"), dtype=torch.float64, device="cuda")
    run(first, x.t().contiguous(), c.t().contiguous(), dim=0)
    assert torch.equal(y, first.t())
