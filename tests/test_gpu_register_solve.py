"""The builder's register solve (chunks of at most 17 rows in registers, tiles of lines passed
through shared memory) at the sizes where its bookkeeping changes: row counts around the multiples
of the chunk length, the longest lines it takes and the first ones beyond, batches of one line, of
odd and even counts, of more tiles than blocks, and each place of the interpolation dimension. Against
the oracle; tolerance: max-norm relative error <= 1e-12, or 10 cond(A) eps for an ill-conditioned
system (two backward-stable FP64 solves agree to about that)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P, H, G = 0, 1, 3


def cuda(a):
    return None if a is None or a.size == 0 else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def build_and_compare(D, O, degree, closure, uniform, nc, B, layout, seed):
    rng = np.random.default_rng(seed)
    br = np.linspace(0.0, 1.0, nc + 1)
    if uniform:
        bs, obs = D.UniformBSplines(degree, closure == P, 0.0, 1.0, nc), O.BSplines(degree, closure == P, rmin=0.0, rmax=1.0, ncells=nc)
    else:
        br[1:-1] += rng.uniform(-0.3, 0.3, nc - 1) / nc
        bs, obs = D.NonUniformBSplines(degree, closure == P, br), O.BSplines(degree, closure == P, breaks=br)
    b = D.SplineBuilder(bs, None, closure, closure)
    ob = O.Builder(obs, b.interpolation_points, closure, closure)
    vals = rng.standard_normal((b.npoints, B))
    nd = b.s_nbv_xmin if closure == H else 0
    dlo, dhi = rng.standard_normal((nd, B)), rng.standard_normal((nd, B))
    ref = ob(vals, dlo if nd else None, dhi if nd else None)

    def put(a):
        if layout == "first" or a.size == 0:
            return cuda(a)
        if layout == "last":
            return cuda(a.T)
        return cuda(a.reshape(a.shape[0], -1, 3).transpose(1, 0, 2))

    dim = 0 if layout == "first" else 1
    shape = {"first": (bs.size, B), "last": (B, bs.size), "mid": (B // 3, bs.size, 3)}[layout]
    coefs = torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")
    b(coefs, put(vals), put(dlo), put(dhi), dim=dim)
    got = coefs.cpu().numpy()
    got = got if layout == "first" else got.T if layout == "last" else got.transpose(1, 0, 2).reshape(bs.size, B)
    tol = max(1e-12, 10 * np.linalg.cond(ob.matrix()) * np.finfo(float).eps)
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    return b, ob


@pytest.mark.parametrize("nc", [13, 17, 18, 19, 34, 35, 52, 97, 255, 513, 1024])
@pytest.mark.parametrize("degree,closure,uniform", [(1, G, False), (2, P, True), (3, H, True), (3, P, True), (4, G, True), (5, H, False),
                                                    (5, P, False)])
def test_rows(oracle_mod, nc, degree, closure, uniform):
    import ddc_b200 as D

    build_and_compare(D, oracle_mod, degree, closure, uniform, nc, 21, "first", nc + degree)


@pytest.mark.parametrize("nc", [1088, 1390, 1720, 2200])
@pytest.mark.parametrize("degree,closure", [(3, H), (5, P)])
def test_longest_lines(oracle_mod, nc, degree, closure):
    import ddc_b200 as D

    build_and_compare(D, oracle_mod, degree, closure, False, nc, 6, "first", nc)


@pytest.mark.parametrize("layout,B", [("first", 1), ("first", 2), ("first", 599), ("first", 600), ("last", 1), ("last", 601), ("mid", 603)])
@pytest.mark.parametrize("degree,closure,uniform,nc", [(3, P, True, 100), (5, H, False, 70), (3, G, False, 600)])
def test_batches_and_layouts(oracle_mod, layout, B, degree, closure, uniform, nc):
    import ddc_b200 as D

    build_and_compare(D, oracle_mod, degree, closure, uniform, nc, B, layout, B)


@pytest.mark.parametrize("B", [20001, 20002])
def test_many_tiles_and_in_place_solve(oracle_mod, B):
    import ddc_b200 as D

    b, ob = build_and_compare(D, oracle_mod, 3, P, True, 40, B, "first", B)
    A = ob.matrix()
    rhs = np.random.default_rng(1).standard_normal((b.info.nbasis, B))
    for transpose in (False, True):
        x = b.solve(cuda(rhs), transpose).cpu().numpy()
        assert np.abs((A.T if transpose else A) @ x - rhs).max() <= 1e-12 * np.abs(rhs).max()
