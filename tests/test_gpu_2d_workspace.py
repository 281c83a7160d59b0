"""The 2D build in workspaces between the least and the one it asks for, and without one when the device
has no room for the widest groups: the groups of fields change, the coefficients do not, bit for bit."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

P, H = 0, 1


@pytest.fixture(scope="module")
def case():
    import ddc_b200 as D

    bx, by = D.UniformBSplines(3, True, 0.0, 1.0, 512), D.UniformBSplines(3, False, 0.0, 1.0, 512)
    b1, b2 = D.SplineBuilder(bx), D.SplineBuilder(by, None, H, H)
    b = D.SplineBuilder2D(b1, b2)
    F = 70  # a whole group of 64 and a part of one
    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.rand(s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    v, kw = rand(512, b2.npoints, F), dict(derivs_min2=rand(512, 1, F), derivs_max2=rand(512, 1, F))
    want = torch.full((bx.size, by.size, F), float("nan"), dtype=torch.float64, device="cuda")
    need = b.workspace_bytes(F)
    b(want, v, workspace=torch.empty(need, dtype=torch.uint8, device="cuda"), **kw)
    return b, v, kw, want, need


@pytest.mark.parametrize("mib", [44, 64, 100, 128])
def test_smaller_workspaces(case, mib):
    b, v, kw, want, need = case
    assert mib << 20 < need
    got = torch.full_like(want, float("nan"))
    b(got, v, workspace=torch.empty(mib << 20, dtype=torch.uint8, device="cuda"), **kw)
    assert torch.equal(got, want)


def test_too_small_a_workspace_is_refused(case):
    import ddc_b200 as D

    b, v, kw, want, need = case
    with pytest.raises(D.DdcbError):
        b(torch.empty_like(want), v, workspace=torch.empty(4 << 20, dtype=torch.uint8, device="cuda"), **kw)


def test_little_free_memory(case):
    b, v, kw, want, need = case
    got = torch.full_like(want, float("nan"))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    rest = 100 << 20
    assert rest < need
    full = torch.empty(torch.cuda.mem_get_info()[0] - rest, dtype=torch.uint8, device="cuda")
    try:
        b(got, v, **kw)
        torch.cuda.synchronize()
    finally:
        del full
        torch.cuda.empty_cache()
    assert torch.equal(got, want)
