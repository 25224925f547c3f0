"""A result does not depend on the launch it is computed in.  Evaluation and inversion pick kernels, CTA
sizes and the distribution of work by the number of points: the forms are compared with one another at
the sizes where the choice changes, and the span lookup of the evaluation with numpy's search."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

WARPS = 4 * 152              # one warp per scheduler
FEW = 8 * WARPS              # FP64 evaluation: four lanes per point up to here
SMALL_CTAS = 32 * 4 * WARPS  # FP64 evaluation: CTAs of one warp; inversion: 4 CTAs per SM up to here


def T(x, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device="cuda")


def host(*x):
    return [a.cpu().numpy() for a in x]


def surface(p, q, nu, nv, seed=5):
    from gpu_nurbs_gb300 import synth
    r = synth.Rng(seed)
    x = np.repeat(np.arange(nu) / (nu - 1), nv)
    y = np.tile(np.arange(nv) / (nv - 1), nu)
    z = 0.15 * np.sin(3 * x + 2 * y) + r.normal(nu * nv, 0.02)
    return dict(p=p, q=q, nu=nu, nv=nv, knots_u=synth.gapped_knots(p, nu, r), knots_v=synth.uniform_knots(q, nv),
                cps=np.stack([x, y, z], 1), weights=r.uniform(nu * nv, 0.5, 2.0))


def queries(s, nurbs, n, seed, off):
    from gpu_nurbs_gb300 import synth
    rng = np.random.default_rng(seed)
    E = s.eval(T(rng.random((n, 2))), 7).cpu().numpy()
    return synth.form_queries(E[0:3].T, E[3:6].T, E[6:9].T, rng.normal(0, off, n))


@pytest.mark.parametrize("mask", [1, 7, 6, 63, 40, 1023], ids=lambda m: f"mask{m}")
@pytest.mark.parametrize("pq", [(1, 1), (2, 2), (3, 3), (5, 5), (2, 5), (7, 3)], ids=lambda d: f"p{d[0]}q{d[1]}")
def test_few_points_equal_many(nurbs, pq, mask):
    """The same operations per point in every form: the same bits, in and outside the domain."""
    s = nurbs.Surface(surface(*pq, 11, 9))
    rng = np.random.default_rng(3)
    uv = rng.random((SMALL_CTAS + 1, 2))
    b = np.asarray(surface(*pq, 11, 9)["knots_u"])
    uv[:len(b), 0] = b
    uv[len(b):len(b) + 5] = [[-0.5, 0.5], [1.5, -1.5], [-0.0, 1.0], [np.nan, 0.5], [np.inf, -np.inf]]
    uv[FEW - 1], uv[FEW], uv[SMALL_CTAS - 1], uv[SMALL_CTAS] = [1, 0], [0, 1], [0.25, 1], [1, 1]
    duv = T(uv)
    many = s.eval(duv, mask).cpu().numpy()
    for n in (1, 7, 8, 9, len(b) + 5, FEW - 1, FEW, FEW + 1, SMALL_CTAS):
        assert np.array_equal(s.eval(duv[:n], mask).cpu().numpy(), many[:, :n], equal_nan=True), n


def knots_of(kind):
    if kind == "clustered":  # 200 spans within 3e-4 of the domain, three spans besides
        inner = np.concatenate([[0.3], 0.6 + 1.5e-6 * np.arange(1, 201), [0.9]])
    elif kind == "one_in_fp32":  # all breakpoints the same FP32 number
        return 1e9 + np.array([0., 0., 1., 2., 4., 5., 7., 8., 8.])
    elif kind == "around_zero":
        inner = np.linspace(-1, 1, 9)[1:-1]
    else:
        inner = np.arange(1, kind) / kind
    lo, hi = (-1.0, 1.0) if kind == "around_zero" else (0.0, 1.0)
    return np.concatenate([[lo, lo], inner, [hi, hi]])


@pytest.mark.parametrize("kind", [1, 2, 3, 255, 256, 257, 700, "clustered", "around_zero", "one_in_fp32"])
def test_span_lookup(nurbs, kind):
    """Degree 1, weights 1: Su is constant in u within a span and jumps at every knot, so it shows the span
    that was looked up: the last whose start is not above u, in the precision of the evaluation."""
    ku = knots_of(kind)
    nu = len(ku) - 2
    rng = np.random.default_rng(9)
    b, z = ku[1:-1], rng.permutation(nu) + 1.0
    cps = np.zeros((nu, 2, 3))
    cps[:, :, 0], cps[:, :, 2] = b[:, None], np.cumsum(z)[:, None]
    cps[:, 1, 1] = 1.0
    s = nurbs.Surface(dict(p=1, q=1, nu=nu, nv=2, knots_u=ku, knots_v=np.array([0., 0., 1., 1.]),
                           cps=cps.reshape(-1, 3), weights=np.ones(nu * 2)))
    for dt, call in ((np.float32, s.eval_f32), (np.float64, s.eval)):
        bt = b.astype(dt)
        u = np.concatenate([bt, np.nextafter(bt, dt(-9)), np.nextafter(bt, dt(9)), (rng.random(6000) * 2.4 - 1.2).astype(dt),
                            (0.6 + rng.random(2000) * 4e-4).astype(dt), [dt(-0.0), dt(-2), dt(3)]]).astype(dt)
        span = np.clip(np.searchsorted(bt, u, "right") - 1, 0, nu - 2)
        # the derivative scaled by the knot range, as the evaluation returns it
        su = np.diff(np.cumsum(z))[span] * (b[-1] - b[0]) / np.diff(b)[span]
        uv = T(np.stack([u, np.full_like(u, 0.5)], 1), torch.float32 if dt is np.float32 else torch.float64)
        for n in (len(u), 100):
            got = call(uv[:n].contiguous(), 2).cpu().numpy()[2]
            # the slope is a difference of two sums of up to nu (nu + 1) / 2; a wrong span is another integer's slope
            tol = 16 * np.finfo(dt).eps * nu * (nu + 1) / np.diff(b)[span[:n]]
            assert np.all(np.abs(got - su[:n]) <= tol), (dt, n)


@pytest.mark.parametrize("pq,precision", [((3, 3), 1), ((2, 2), 1), ((5, 5), 1), ((4, 3), 1), ((3, 3), 0), ((5, 5), 0),
                                          ((3, 4), 0)])
def test_inversion_of_part_of_a_launch(nurbs, pq, precision):
    """A query's trajectories are its own: the same bits whatever the launch holds besides."""
    total = SMALL_CTAS + 1 if precision == 1 else 6000
    s = nurbs.Surface(surface(*pq, 12, 10))
    P = T(queries(s, nurbs, total, 4, 1e-2))
    all_ = host(*s.invert(P, precision))
    for n in (1, 31, 33, WARPS, WARPS + 1, total - 1):
        for lo in (0, total - n):
            for a, b in zip(host(*s.invert(P[lo:lo + n].contiguous(), precision)), all_):
                assert np.array_equal(a, b[lo:lo + n], equal_nan=True), (n, lo)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("which", ["quadtree", "project"])
@pytest.mark.parametrize("pq", [(3, 3), (2, 4)], ids=lambda d: f"p{d[0]}q{d[1]}")
def test_search_of_part_of_a_launch(nurbs, pq, which, precision):
    """Lane-wise and warp-wise searches, full and partial portions, reversed order: the same status, the
    answer to the 1e-9 of every converged Newton iteration, the residual to rounding."""
    s = nurbs.Surface(surface(*pq, 20, 17))
    run = (lambda P: s.invert_quadtree(P, 1e-2, precision)) if which == "quadtree" else (lambda P: s.project(P, precision))
    total = 4099
    P = queries(s, nurbs, total, 6, 4e-3)
    P[::7] += 0.2
    uv, st, res = host(*run(T(P)))
    for n in (1, 2, 31, 33, 128, 129, WARPS + 1, total):
        for step in (1, -1):
            at = np.arange(total)[::step][:n]
            u, t, r = host(*run(T(P[at])))
            assert np.array_equal(t, st[at]), (n, step)
            found = t <= 1
            assert np.all(np.abs(u - uv[at])[found] <= 1e-9), (n, step)
            assert np.all(np.abs(r - res[at])[found] <= 1e-12 * res[at][found] + 1e-14), (n, step)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_pool_tiles_taken_together(nurbs, precision):
    """Small tiles are taken several at a time, across surfaces too: the single surfaces' bits for every tile
    size, with more tiles than resident CTAs, empty and ragged ranges and a repeated surface."""
    surfs = [surface(p, q, 9, 8, 20 + p + q) for p, q in ((3, 3), (2, 5), (4, 3), (5, 5))]
    counts = [0, 1, 700, 17, 0, 33, 1300, 128]
    which = [0, 1, 2, 3, 1, 0, 0, 2]
    pool = nurbs.Pool(1 << 26, max_surfaces=8)
    ids = pool.add(surfs)
    singles = [nurbs.Surface(x) for x in surfs]
    P = np.concatenate([queries(singles[w], nurbs, max(c, 1), 30 + k, 1e-2)[:c]
                        for k, (w, c) in enumerate(zip(which, counts))])
    off = np.concatenate([[0], np.cumsum(counts)])
    batch = nurbs.Batch(np.asarray(ids)[which], off)
    ref = [np.concatenate(x) for x in zip(*(host(*singles[w].invert(T(P[a:b]), precision))
                                            for w, a, b in zip(which, off[:-1], off[1:]) if b > a))]
    for tile in (1, 2, 16, 31, 32, 64, 256):
        pool.set_config(tile, 6)
        for a, b in zip(host(*pool.invert(batch, T(P), precision)), ref):
            assert np.array_equal(a, b, equal_nan=True), tile
