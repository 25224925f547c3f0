"""The quadtree inversion's search beyond the root: layers wider than a lane keeps, nodes of many control
points, layer overflow; and the device memory its local arrays reserve."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
from conftest import ROOT

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def T(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")


def surface(p, q, nu, nv, relief):
    from gpu_nurbs_gb300 import synth
    r = synth.Rng(91)
    x, y = np.repeat(np.arange(nu) / (nu - 1), nv), np.tile(np.arange(nv) / (nv - 1), nu)
    return dict(p=p, q=q, nu=nu, nv=nv, knots_u=synth.gapped_knots(p, nu, r), knots_v=synth.gapped_knots(q, nv, r),
                cps=np.stack([x, y, r.normal(nu * nv, relief)], 1), weights=r.uniform(nu * nv, 0.5, 2.0))


# relief, max_edge and offset from the surface: rough nets widen the layers past the 8 nodes that a lane
# keeps and past the 64 of a layer; the large net's undivided halves and deep nodes have hundreds of control
# points; 1-degree nets have kinks where trajectories end without a result
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("pq,net,relief,max_edge,off", [
    ((3, 3), (8, 8), 0.2, 1e-1, 0.3), ((3, 3), (8, 8), 0.2, 1e-2, 0.2), ((2, 4), (12, 30), 0.1, 3e-2, 0.1),
    ((3, 3), (260, 40), 1e-2, 1e-2, 0.05), ((3, 3), (300, 300), 1e-3, 1e-3, 0.01), ((1, 1), (20, 20), 0.05, 1e-2, 0.05)],
    ids=["wide", "rough", "uneven", "spans260", "large", "kinked"])
def test_search_matches_the_oracle(nurbs, pq, net, relief, max_edge, off, precision):
    """Points off the surface, most without an answer at the root: FP64 the oracle's status, answer to the
    1e-9 of a converged Newton iteration, residual to rounding; mixed a status that differs for at most 1 %
    (its FP32 trajectories may end in another basin), and answers within max_edge."""
    sf = surface(*pq, *net, relief)
    s, o = nurbs.Surface(sf), O.OracleSurface(sf)
    rng = np.random.default_rng(8)
    E = o.eval(rng.random((600, 2)), 1).T
    P = E + off * (rng.random((600, 3)) - 0.5)
    uv, st, res = (x.cpu().numpy() for x in s.invert_quadtree(T(P), max_edge, precision))
    ouv, ost, ores, layers = o.invert_quadtree(P, max_edge)
    assert np.count_nonzero(layers > 1) >= 50
    if precision == 0:
        f = ost <= 1
        assert np.array_equal(st, ost)
        assert np.all(np.abs(uv - ouv)[f] <= 1e-9)
        assert np.all(np.abs(res - ores)[f] <= 1e-12 * ores[f] + 1e-14)
    else:
        assert np.count_nonzero((st <= 1) != (ost <= 1)) <= 6
        assert np.all(res[st <= 1] < max_edge)
    for n in (1, 2, 33):  # the same bits in another launch
        a, b, c = (x.cpu().numpy() for x in s.invert_quadtree(T(P[:n]), max_edge, precision))
        assert np.array_equal(b, st[:n]) and np.array_equal(a, uv[:n], equal_nan=True)
        assert np.array_equal(c, res[:n], equal_nan=True)


MEMORY = """
import importlib.util, os, sys, torch
pkg = os.path.join({root!r}, "gpu-nurbs_gb300")
spec = importlib.util.spec_from_file_location("gpu_nurbs_gb300", os.path.join(pkg, "__init__.py"),
                                              submodule_search_locations=[pkg])
gn = importlib.util.module_from_spec(spec)
sys.modules["gpu_nurbs_gb300"] = gn
spec.loader.exec_module(gn)
from gpu_nurbs_gb300 import synth
P = torch.zeros((64, 3), dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
for surf in (synth.surface_small(), synth.surface_quintic(n=32)):
    s = gn.Surface(surf)
    for precision in (0, 1):
        s.invert(P, precision), s.project(P, precision), s.invert_quadtree(P, 1e-3, precision), s.pcurve(P, precision)
torch.cuda.synchronize()
print((before - torch.cuda.mem_get_info()[0]) >> 20)
"""


def test_local_memory_reserved():
    """A kernel's stack is reserved for every resident thread and kept by the context: 152 SMs of 2,048
    threads at 1 KB each are 304 MiB, the bound for all queries together."""
    r = subprocess.run([sys.executable, "-c", MEMORY.format(root=ROOT)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ))
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) <= 304
