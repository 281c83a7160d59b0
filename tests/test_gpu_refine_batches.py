"""Refined builds of batches large enough for the kernel with four blocks an SM, and just below, at tiles
of few and of many chunks, and of lines too long for it. Against the oracle; tolerance: max-norm
relative error <= 1e-12, or 10 cond(A) eps for an ill-conditioned system."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P, H, G = 0, 1, 3


@pytest.mark.parametrize("B", [2368, 2369, 2406])
@pytest.mark.parametrize("degree,closure,uniform,nc", [(3, P, True, 13), (3, H, False, 64), (5, H, False, 130), (4, G, True, 300),
                                                       (2, P, False, 520), (5, P, False, 700)])
def test_large_batches(oracle_mod, degree, closure, uniform, nc, B):
    import ddc_b200 as D

    O = oracle_mod
    rng = np.random.default_rng(nc + B)
    br = np.linspace(0.0, 1.0, nc + 1)
    if uniform:
        bs, obs = D.UniformBSplines(degree, closure == P, 0.0, 1.0, nc), O.BSplines(degree, closure == P, rmin=0.0, rmax=1.0, ncells=nc)
    else:
        br[1:-1] += rng.uniform(-0.3, 0.3, nc - 1) / nc
        bs, obs = D.NonUniformBSplines(degree, closure == P, br), O.BSplines(degree, closure == P, breaks=br)
    b = D.SplineBuilder(bs, None, closure, closure, precision="fp32_refine")
    ob = O.Builder(obs, b.interpolation_points, closure, closure)
    nd = b.s_nbv_xmin if closure == H else 0
    few = rng.standard_normal((b.npoints, 31)), rng.standard_normal((nd, 31)), rng.standard_normal((nd, 31))
    ref = ob(few[0], few[1] if nd else None, few[2] if nd else None)
    lines = np.arange(B) * 7 % 31
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a[:, lines])).cuda() if a.size else None  # noqa: E731
    coefs = torch.full((bs.size, B), float("nan"), dtype=torch.float64, device="cuda")
    b(coefs, *map(put, few))
    tol = max(1e-12, 10 * np.linalg.cond(ob.matrix()) * np.finfo(float).eps)
    assert np.abs(coefs.cpu().numpy() - ref[:, lines]).max() <= tol * np.abs(ref).max()
