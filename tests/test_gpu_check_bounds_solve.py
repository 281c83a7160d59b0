"""The bounds-checked build over the register solve's row indices: builds, fused steps, backwards and
in-place solves of several layouts, closures and line counts, in two fresh processes, one per library.
On these valid inputs nothing may be recorded, and the results must be the default build's bit for bit
(but for the backward's atomic sums)."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_workloads(out_path):
    import torch

    import ddc_b200 as D

    res = {"checked": np.array([int(D.bounds_checked())])}
    g = torch.Generator(device="cuda").manual_seed(3)
    for degree, closure, uniform, nc, B, layout in ((3, 0, True, 100, 37, 0), (3, 0, True, 52, 37, 1), (5, 1, False, 70, 24, 0),
                                                    (4, 3, True, 300, 25, 1), (2, 1, True, 33, 1, 0), (5, 0, False, 200, 600, 0)):
        br = np.linspace(0.0, 1.0, nc + 1)
        br[1:-1] += np.random.default_rng(nc).uniform(-0.3, 0.3, nc - 1) / nc
        bs = D.UniformBSplines(degree, closure == 0, 0.0, 1.0, nc) if uniform else D.NonUniformBSplines(degree, closure == 0, br)
        b, e = D.SplineBuilder(bs, None, closure, closure), D.SplineEvaluator(bs)
        put = (lambda a: a.t().contiguous()) if layout else (lambda a: a)
        rand = lambda *s: put(torch.rand(s, dtype=torch.float64, device="cuda", generator=g))  # noqa: E731
        nd = b.s_nbv_xmin if closure == 1 else 0
        lo, hi = (rand(nd, B), rand(nd, B)) if nd else (None, None)
        v, x, gy, c, c2 = rand(b.npoints, B), rand(60, B), rand(60, B), rand(bs.size, B), rand(bs.size, B)
        y, gv, gx = torch.zeros_like(x), torch.zeros_like(v), torch.zeros_like(x)
        b(c, v, lo, hi, dim=layout)
        b.build_and_evaluate(e, c2, v, x, y, lo, hi, dim=layout)
        b.build_and_evaluate_adjoint(e, x, c, gy, gv, gx, dim=layout)
        rhs = torch.rand((b.info.nbasis, B), dtype=torch.float64, device="cuda", generator=g)
        s1, s2 = b.solve(rhs.clone()), b.solve(rhs.clone(), True)
        k = f"d{degree}_{nc}_"
        for name, t in (("c", c), ("c2", c2), ("y", y), ("gx", gx), ("s1", s1), ("s2", s2), ("atomic", gv)):
            res[k + name] = t.cpu().numpy()
    torch.cuda.synchronize()
    D.last_device_error()  # raises if a kernel recorded an out-of-range index
    np.savez(out_path, **res)


def test_register_solve_indices(tmp_path):
    got = []
    for checked in ("0", "1"):
        path = str(tmp_path / f"out{checked}.npz")
        code = f"import sys; sys.path[:0] = [{ROOT!r}, {os.path.join(ROOT, 'tests')!r}]; import test_gpu_check_bounds_solve as t; t.run_workloads({path!r})"
        env = {k: v for k, v in os.environ.items() if k != "DDCB_CHECK_BOUNDS"}
        if checked == "1":
            env["DDCB_CHECK_BOUNDS"] = "1"
        r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        got.append(np.load(path))
    assert got[0]["checked"][0] == 0 and got[1]["checked"][0] == 1
    for k in got[0].files:
        if "atomic" in k:
            np.testing.assert_allclose(got[1][k], got[0][k], rtol=1e-12, atol=1e-12)
        elif k != "checked":
            assert np.array_equal(got[0][k], got[1][k]), k
