"""The pool's launch configuration: CTAs per SM beyond what fits, and the autotuner's cache file."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def work(nurbs):
    from gpu_nurbs_gb300 import synth
    r = synth.Rng(61)
    surfs = [synth.surface_random(r) for _ in range(6)]
    pool = nurbs.Pool(1 << 27, max_surfaces=8)
    ids = pool.add(surfs)
    per = 900
    uv = torch.as_tensor(np.random.default_rng(2).random((per * len(surfs), 2)), device="cuda")
    batch = nurbs.Batch(ids, np.arange(len(surfs) + 1) * per)
    P = pool.eval(batch, uv, 1).T.contiguous()
    out = (torch.empty((len(P), 2), dtype=torch.float64, device="cuda"),
           torch.empty(len(P), dtype=torch.int32, device="cuda"), torch.empty(len(P), dtype=torch.float64, device="cuda"))
    return pool, batch, P, out


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_ctas_per_sm(nurbs, work, precision):
    """1..16 are accepted and give the same bits, launched directly or from a graph; 4 fit an SM."""
    pool, batch, P, out = work
    pool.set_config(128, 4)
    ref = [x.cpu().numpy() for x in pool.invert(batch, P, precision)]
    for tile in (16, 128):
        for ctas in (1, 3, 5, 6, 16):
            pool.set_config(tile, ctas)
            assert pool.info().ctas_per_sm == ctas
            g = pool.graph(batch, P, out, precision)
            g.launch()
            for got in (pool.invert(batch, P, precision), out):
                assert all(np.array_equal(a.cpu().numpy(), b, equal_nan=True) for a, b in zip(got, ref)), (tile, ctas)
            g.close()
    for bad in (0, 17):
        with pytest.raises(nurbs.NurbsError):
            pool.set_config(128, bad)
    assert 1 <= pool.autotune(batch, P, out, precision)[1] <= 4


def test_autotune_cache(nurbs, work, tmp_path):
    """A line of this schedule is taken as it is; one written for another schedule, whose (tile, CTAs) pairs
    mean other launches, is not."""
    pool, batch, P, out = work
    cache = tmp_path / "tune.txt"
    best = pool.autotune(batch, P, out, 1, cache_path=str(cache))
    key = cache.read_text().split()[0]
    cache.write_text(f"{key} 64 2 0.5\n")
    assert pool.autotune(batch, P, out, 1, cache_path=str(cache)) == (64, 2, 0.5)
    assert (pool.info().tile_queries, pool.info().ctas_per_sm) == (64, 2)
    old = "/".join(part for part in key.split("/") if not (part[0] == "s" and part[1:].isdigit()))
    assert old != key
    cache.write_text(f"{old} 7 6 0.0001\n")
    tile, ctas, ms = pool.autotune(batch, P, out, 1, cache_path=str(cache))
    assert tile != 7 and ctas <= 4 and ms > 0.0001
    assert len(cache.read_text().splitlines()) == 2
    assert best[2] > 0
