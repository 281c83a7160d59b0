"""2D and 3D evaluation over batches that fill a warp in different ways: single fields, odd counts, pairs
of fields that share their points (one basis, 16-byte loads), that do not, or do only in part, and
point sets around the block size. Every field has to come out bit for bit as when it is evaluated
alone (which the oracle tests cover), since no operation on a field depends on its neighbours."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def spline_parts(D, ndims, degree, uniform):
    sizes = (17, 12, 9)[:ndims]
    bases = []
    for q, n in enumerate(sizes):
        br = np.linspace(0.0, 1.0, n + 1)
        br[1:-1] += np.random.default_rng(q).uniform(-0.2, 0.2, n - 1) / n
        bases.append(D.UniformBSplines(degree, q == 0, 0.0, 1.0, n) if uniform else D.NonUniformBSplines(degree, q == 0, br))
    ev = [D.SplineEvaluator(b, D.Extrapolation.CONSTANT, D.Extrapolation.NULL) for b in bases]
    return [b.size for b in bases], (D.SplineEvaluator2D if ndims == 2 else D.SplineEvaluator3D)(*ev)


@pytest.mark.parametrize("ndims,degree,uniform", [(2, 3, True), (2, 4, False), (3, 3, True), (3, 2, False)])
@pytest.mark.parametrize("B,m", [(1, 2049), (2, 63), (3, 700), (16, 257), (63, 33), (64, 65), (66, 31), (130, 17)])
@pytest.mark.parametrize("points", ["shared", "own", "mixed"])
def test_fields_alone_and_together(ndims, degree, uniform, B, m, points):
    import ddc_b200 as D

    sizes, ev = spline_parts(D, ndims, degree, uniform)
    g = torch.Generator(device="cuda").manual_seed(B + m)
    coefs = torch.randn((*sizes, B), dtype=torch.float64, device="cuda", generator=g)
    x = torch.rand((m, B, ndims), dtype=torch.float64, device="cuda", generator=g) * 1.2 - 0.1
    if points == "shared":
        x = x[:, :1].expand(m, B, ndims).contiguous()
    elif points == "mixed":
        x[::2] = x[::2, :1].clone()
    together = torch.full((m, B), float("nan"), dtype=torch.float64, device="cuda")
    ev(together, x, coefs)
    for b in sorted({0, B // 2, B - 1}):
        alone = torch.empty((m, 1), dtype=torch.float64, device="cuda")
        ev(alone, x[:, b:b + 1].contiguous(), coefs[..., b:b + 1].contiguous())
        assert torch.equal(together[:, b], alone[:, 0])
