"""The residual that a query returns is the distance from its point to the surface at the returned
parameters, on every knot range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def T(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("what", ["invert", "quadtree", "project", "pcurve"])
@pytest.mark.parametrize("lo,hi", [(0.0, 1.0), (-1.0, 1.0), (0.2, 1.1)], ids=["unit", "symmetric", "shorter"])
@pytest.mark.parametrize("pq", [(3, 3), (2, 4)], ids=lambda d: f"p{d[0]}q{d[1]}")
def test_residual_is_the_distance(nurbs, pq, lo, hi, what, precision):
    """Points on the surface, where the derivatives' scale by the knot range shows in a residual formed
    from the last step.  Bound: the rounding of S, of unit size, is a few eps in either evaluation."""
    from gpu_nurbs_gb300 import synth
    r = synth.Rng(77)
    p, q, nu, nv, n = *pq, 20, 18, 2000
    x, y = np.repeat(np.arange(nu) / (nu - 1), nv), np.tile(np.arange(nv) / (nv - 1), nu)
    z = 0.15 * np.sin(5 * x + 3 * y) + r.normal(nu * nv, 0.005)
    s = nurbs.Surface(dict(p=p, q=q, nu=nu, nv=nv, knots_u=lo + (hi - lo) * synth.gapped_knots(p, nu, r),
                           knots_v=lo + (hi - lo) * synth.gapped_knots(q, nv, r), cps=np.stack([x, y, z], 1),
                           weights=r.uniform(nu * nv, 0.5, 2.0)))
    P = s.eval(T(lo + (hi - lo) * np.random.default_rng(5).random((n, 2))), 1).T.contiguous()
    if what == "quadtree":
        uv, st, res = s.invert_quadtree(P, 1e-2, precision)
    else:
        uv, st, res = getattr(s, what)(P, precision)[:3]
    found = st <= 1
    assert int(found.sum()) > n // 2
    dist = (s.eval(uv[found].contiguous(), 1).T - P[found]).norm(dim=1)
    assert float((res[found] - dist).abs().max()) <= 64 * np.finfo(float).eps
