"""A query's result is bit-identical whatever else is in its launch: projection and quadtree inversion, which
search by a lane or by the whole warp according to what the launch holds (the inversion's counterpart is in
test_gpu_launch_forms.py)."""
import numpy as np
import pytest

from test_gpu_launch_forms import T, WARPS, host, queries, surface

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("which", ["quadtree", "wide", "project"])
@pytest.mark.parametrize("pq", [(3, 3), (5, 5), (2, 4), (1, 1)], ids=lambda d: f"p{d[0]}q{d[1]}")
def test_same_bits_in_every_launch(nurbs, pq, which, precision):
    s = nurbs.Surface(surface(*pq, 20, 17))
    run = {"quadtree": lambda P: s.invert_quadtree(P, 1e-2, precision), "project": lambda P: s.project(P, precision),
           "wide": lambda P: s.invert_quadtree(P, 1e-1, precision)}[which]
    total = 4099
    P = queries(s, nurbs, total, 6, 4e-3)
    P[::7] += 0.2  # far points: line searches, and searches without an answer
    P[3::11] *= 3.0
    whole = host(*run(T(P)))
    for n in (1, 2, 3, 31, 33, 128, 129, WARPS + 1, total):
        for step in (1, -1):
            at = np.arange(total)[::step][:n]
            for a, b in zip(host(*run(T(P[at]))), whole):
                assert np.array_equal(a, b[at], equal_nan=True), (n, step)
