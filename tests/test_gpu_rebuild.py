"""Rebuilding a surface's tree while other streams query the surface: the rebuild writes the values that
are there, so the queries' results are those of a quiet surface."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_queries_during_a_rebuild(nurbs, precision):
    from gpu_nurbs_gb300 import synth
    s = nurbs.Surface(synth.surface_large())
    rng = np.random.default_rng(4)
    uv = torch.as_tensor(rng.random((3000, 2)), dtype=torch.float64, device="cuda")
    P = s.eval(uv, 1).T.contiguous()
    P[::5] += 0.3 * torch.as_tensor(rng.random((600, 3)) - 0.5, device="cuda")
    calls = [lambda: s.invert(P, precision), lambda: s.project(P, precision), lambda: s.invert_quadtree(P, 1e-3, precision),
             lambda: s.candidates(P)]
    quiet = [[x.cpu().numpy() for x in c()] for c in calls]
    records = [np.concatenate([np.ravel(x) for x in (*s.tree(), *s.normal_cones())])]
    torch.cuda.synchronize()
    rebuild, stop, codes = torch.cuda.Stream(), threading.Event(), []

    def loop():
        while not stop.is_set() and len(codes) < 2000:
            codes.append(nurbs.lib().nurbs_build_tree(s.h, 2, rebuild.cuda_stream))

    t = threading.Thread(target=loop)
    t.start()
    try:
        mine = torch.cuda.Stream()
        with torch.cuda.stream(mine):
            got = [[c() for c in calls] for _ in range(60)]
            mine.synchronize()
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    assert len(codes) >= 3 and not any(codes)
    counts = quiet[3][1]
    for one in got:
        for k, (a, b) in enumerate(zip(one, quiet)):
            a = [x.cpu().numpy() for x in a]
            if k == 3:  # a candidate list is filled up to its count
                assert np.array_equal(a[1], counts)
                used = np.arange(a[0].shape[1]) < counts[:, None]
                assert np.array_equal(a[0][used], b[0][used])
                continue
            assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b)), k
    records.append(np.concatenate([np.ravel(x) for x in (*s.tree(), *s.normal_cones())]))
    assert np.array_equal(*records)
