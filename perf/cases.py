"""The work a user of this library has it do, as cases that can be timed and compared.

Every case goes through the public Python binding of the C-ABI: evaluation of points and
derivatives (FP64 and FP32), point inversion (mixed and FP64, device and host buffers, one surface
and a pool of many), projection, the tree-free quadtree inversion, p-curves, and the conversion of
a new surface.  Surfaces and queries are seeded synthetic ones with the shapes of the library's own
workloads (gpu-nurbs_gb300/synth.py): bicubic 8x8 and 64x64 nets, a quintic 256x256 net and many
small nets of uneven degree.

Queries are formed by a plain torch evaluation of the surface in 64 bits (below), not by the
library, which is also what exact() returns for the evaluation cases.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.getcwd()


def _package():
    """The library's binding: its folder is not an identifier, so it is loaded by path."""
    if "gpu_nurbs_gb300" in sys.modules:
        return sys.modules["gpu_nurbs_gb300"]
    folder = os.path.join(ROOT, "gpu-nurbs_gb300")
    spec = importlib.util.spec_from_file_location("gpu_nurbs_gb300", os.path.join(folder, "__init__.py"),
                                                  submodule_search_locations=[folder])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["gpu_nurbs_gb300"] = mod
    spec.loader.exec_module(mod)
    return mod


gn = _package()
from gpu_nurbs_gb300 import synth  # noqa: E402

DEV = "cuda"
F64 = torch.float64
PREC = {"mixed": gn.PREC_MIXED, "fp64": gn.PREC_FP64}


# ------------------------------------------------------------------------------ the cases
def listed():
    bicubic8 = dict(p=3, q=3, nu=8, nv=8, relief="rough")       # the small workload's surface
    bicubic64 = dict(p=3, q=3, nu=64, nv=64, relief="smooth")   # the large workload's surface
    return [
        # An interactive caller: a point and its tangents at a handful of parameters.
        dict(name="eval_few_points", kind="eval", dtype="fp64", mask=7, n=1003, grid=False, **bicubic8),
        # Analysis at scattered parameters: S and all derivatives to second order in FP64.
        dict(name="eval_fp64_second_order", kind="eval", dtype="fp64", mask=63, n=(1 << 22) - 5, grid=False,
             **bicubic64),
        # Tessellation for display: FP32 on a row-major parameter grid with odd sides.
        dict(name="eval_fp32_tessellation", kind="eval", dtype="fp32", mask=63, n=3001 * 2001, grid=True,
             **bicubic64),
        # One small batch of picks or probe points on a small surface: latency and launches count.
        dict(name="invert_small_batch", kind="invert", precision="mixed", host=False, n=1500, offset="near",
             **bicubic8),
        # A scanned point cloud against a part's surface, from pinned host buffers and back.
        dict(name="invert_cloud_host", kind="invert", precision="mixed", host=True, n=1 << 20, offset="cloud",
             **bicubic64),
        # The same in the plain FP64 schedule, for callers that ask for it.
        dict(name="invert_fp64", kind="invert", precision="fp64", host=False, n=50021, offset="cloud", **bicubic64),
        # A degree-5 surface with a big net: span tables beyond L1.
        dict(name="invert_quintic", kind="invert", precision="mixed", host=False, n=300007, offset="near", p=5, q=5,
             nu=256, nv=256, relief="waves"),
        # Closest points of a cloud partly far from the surface.
        dict(name="project_cloud", kind="project", precision="mixed", n=(1 << 18) + 3, **bicubic64),
        # Points on a freshly uploaded surface, without the tree.
        dict(name="quadtree_on_surface", kind="quadtree", precision="mixed", n=(1 << 18) - 9, **bicubic64),
        # Curves drawn on a surface: parameters of their ordered samples.
        dict(name="pcurve_loops", kind="pcurve", precision="mixed", n=200003, loops=64, **bicubic64),
        # A model of many faces of uneven degree, net and query count, in one call.
        dict(name="pool_many_faces", kind="pool", precision="mixed", faces=160, most=16384),
        # A new surface: conversion, tree and culling data, read back whole.
        dict(name="create_surface", kind="create", **bicubic64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "normal", "invert", "invert", "invert", "project", "quadtree", "pcurve", "pool",
                       "create"])
    if kind == "pool":
        return dict(kind="pool", precision=rng.choice(["mixed", "mixed", "fp64"]) if rng.random() < 0.5 else "mixed",
                    faces=_log_int(rng, 2, 128), most=rng.choice([64, 512, 4096]))
    # degrees: the bicubic and the other equal ones mostly, sometimes uneven or high
    p = q = rng.choice([2, 3, 3, 3, 3, 5, 5])
    if rng.random() < 0.25:
        p, q = rng.choice([1, 2, 3, 4, 5, 7]), rng.choice([1, 2, 3, 4, 5])
    case = dict(kind=kind, p=p, q=q, nu=max(p + 1, _log_int(rng, 4, 160)), nv=max(q + 1, _log_int(rng, 4, 160)),
                relief=rng.choice(["rough", "smooth", "waves"]))
    # points a pass at most: fewer for high degrees, and for degrees without a compiled variant
    weight = (p + 1) * (q + 1) / 16.0 * (1.0 if (p, q) in ((2, 2), (3, 3), (5, 5)) else 6.0)

    def points(most):
        return _log_int(rng, min(64, most), max(65, int(most / max(weight, 1.0))))

    if kind == "eval":
        dtype = rng.choice(["fp64", "fp32"])
        case.update(dtype=dtype, mask=rng.choice([1, 7, 7, 63, 63, 0b101001, 1023, 960]),
                    n=points(1 << 21), grid=rng.random() < 0.4)
    elif kind == "normal":
        case.update(mask=rng.choice([1, 7, 63]), n=points(1 << 20))
    elif kind == "invert":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        case.update(precision=precision, host=rng.random() < 0.3, offset=rng.choice(["near", "cloud"]),
                    n=points(1 << 18 if precision == "mixed" else 1 << 14))
    elif kind == "project":
        precision = rng.choice(["mixed", "fp64"])
        case.update(precision=precision, n=points(1 << 17 if precision == "mixed" else 1 << 14))
    elif kind == "quadtree":
        precision = rng.choice(["mixed", "fp64"])
        case.update(precision=precision, n=points(1 << 16 if precision == "mixed" else 1 << 14))
    elif kind == "pcurve":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        case.update(precision=precision, n=points(1 << 17 if precision == "mixed" else 1 << 13),
                    loops=rng.choice([1, 3, 17, 64]))
    return case


# --------------------------------------------------------------- surfaces and plain evaluation
def _surface(case, seed):
    p, q, nu, nv = (case[k] for k in ("p", "q", "nu", "nv"))
    r = synth.Rng(synth.SEED_BASE + 7919 * (seed % (1 << 31)))
    if case["relief"] == "rough":
        ku, kv = synth.uniform_knots(p, nu), synth.uniform_knots(q, nv)
    else:
        ku, kv = synth.gapped_knots(p, nu, r), synth.gapped_knots(q, nv, r)
    x = np.repeat(np.arange(nu) / (nu - 1), nv)
    y = np.tile(np.arange(nv) / (nv - 1), nu)
    if case["relief"] == "rough":
        z = r.normal(nu * nv, 0.2)
    elif case["relief"] == "smooth":
        z = synth.smooth5(r.normal(nu * nv, 0.1).reshape(nu, nv)).reshape(-1)
    else:
        a, b, phi = r.integers(1, 4, 8), r.integers(1, 4, 8), r.uniform(8, 0.0, 2 * math.pi)
        z = sum(0.05 * np.sin(2 * math.pi * (a[k] * x + b[k] * y) + phi[k]) for k in range(8))
    return dict(p=p, q=q, nu=nu, nv=nv, knots_u=ku, knots_v=kv, cps=np.stack([x, y, z], 1),
                weights=r.uniform(nu * nv, 0.5, 2.0))


def _basis(knots, deg, cp, t, order):
    """(span, ders): the B-spline basis functions that act at t and their derivatives to `order`;
    ders[k][j] is the k-th derivative of N_(span-deg+j)."""
    k = torch.as_tensor(knots, dtype=F64, device=t.device)
    span = torch.searchsorted(k, t.contiguous(), right=True) - 1
    span = span.clamp(deg, cp - 1)
    for _ in range(deg + 1):  # a parameter at the end belongs to the last non-empty span
        span = torch.where((k[span] >= k[span + 1]) & (span > deg), span - 1, span)

    def K(i):
        return k[(span + i).clamp(0, len(knots) - 1)]

    zero = torch.zeros_like(t)

    def ratio(a, b):
        return torch.where(b > 0, a / torch.where(b > 0, b, torch.ones_like(b)), zero)

    level = [[None] * (deg + 1) for _ in range(order + 1)]  # level[m][d][j]: m-th derivative, degree d
    for d in range(deg + 1):
        for m in range(order + 1):
            row = []
            for j in range(d + 1):
                if d == 0:
                    row.append(torch.ones_like(t) if m == 0 else zero)
                    continue
                i = j - d  # N_i of degree d over knots span+i .. span+i+d+1
                left = level[m][d - 1][j - 1] if m == 0 and j > 0 else (level[m - 1][d - 1][j - 1] if j > 0 else None)
                right = level[m][d - 1][j] if m == 0 and j < d else (level[m - 1][d - 1][j] if m and j < d else None)
                v = zero
                if left is not None:
                    v = v + ratio((t - K(i)) * left if m == 0 else d * left, K(i + d) - K(i))
                if right is not None:
                    w = ratio((K(i + d + 1) - t) * right if m == 0 else d * right, K(i + d + 1) - K(i + 1))
                    v = v + w if m == 0 else v - w
                row.append(v)
            level[m][d] = row
    return span, [level[m][deg] for m in range(order + 1)]


def _ders(surf, uv, order):
    """{(a, b): (n, 3)} the derivatives d^(a+b) S / du^a dv^b with a + b <= order, in 64 bits."""
    p, q, nu, nv = surf["p"], surf["q"], surf["nu"], surf["nv"]
    w = torch.as_tensor(surf["weights"], dtype=F64, device=uv.device)
    pw = torch.cat([torch.as_tensor(surf["cps"], dtype=F64, device=uv.device) * w[:, None], w[:, None]], 1)
    su, bu = _basis(surf["knots_u"], p, nu, uv[:, 0].double(), order)
    sv, bv = _basis(surf["knots_v"], q, nv, uv[:, 1].double(), order)
    R = {(a, b): torch.zeros((len(uv), 4), dtype=F64, device=uv.device)
         for a in range(order + 1) for b in range(order + 1 - a)}
    for i in range(p + 1):
        row = [torch.zeros((len(uv), 4), dtype=F64, device=uv.device) for _ in range(order + 1)]
        for j in range(q + 1):
            c = pw[(su - p + i) * nv + (sv - q + j)]
            for b in range(order + 1):
                row[b] += bv[b][j][:, None] * c
        for a, b in R:
            R[a, b] += bu[a][i][:, None] * row[b]
    S = {}
    for a, b in sorted(R, key=lambda k: (k[0] + k[1], k)):
        v = R[a, b][:, :3].clone()
        for i in range(a + 1):
            for j in range(b + 1):
                if i or j:
                    v -= math.comb(a, i) * math.comb(b, j) * R[i, j][:, 3:] * S[a - i, b - j]
        S[a, b] = v / R[0, 0][:, 3:]
    return S


def _on_normal(surf, uv, off):
    """P = S(u,v) + off * unit normal."""
    out = torch.empty((len(uv), 3), dtype=F64, device=uv.device)
    for k in range(0, len(uv), 1 << 19):
        sl = slice(k, k + (1 << 19))
        D = _ders(surf, uv[sl], 1)
        nrm = torch.linalg.cross(D[1, 0], D[0, 1], dim=1)
        out[sl] = D[0, 0] + off[sl, None] * nrm / nrm.norm(dim=1, keepdim=True)
    return out


BLOCKS = [(0, 0), (1, 0), (0, 1), (2, 0), (1, 1), (0, 2), (3, 0), (2, 1), (1, 2), (0, 3)]


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _params(case, seed):
    """The parameters a pass evaluates or its queries are formed at."""
    n, g = case["n"], _gen(seed)
    if case["kind"] == "pcurve":  # closed loops inside the domain, their samples in order
        per = -(-n // case["loops"])
        c = torch.rand((case["loops"], 4), generator=g, dtype=F64, device=DEV)
        k = torch.arange(n, device=DEV)
        t, c = 2 * math.pi * (k % per).double() / per, c[k // per]
        r = 0.05 + 0.15 * c[:, 2]
        return torch.stack([0.25 + 0.5 * c[:, 0] + r * torch.cos(t), 0.25 + 0.5 * c[:, 1] + r * torch.sin(t + c[:, 3])], 1)
    if case.get("grid"):
        rows = next(r for r in range(int(math.isqrt(n)), 0, -1) if n % r == 0)
        k = torch.arange(n, device=DEV)
        jitter = torch.rand(2, generator=g, dtype=F64, device=DEV)
        u = ((k // (n // rows)).double() + jitter[0]) / rows
        v = ((k % (n // rows)).double() + jitter[1]) / (n // rows)
        return torch.stack([u, v], 1)
    return torch.rand((n, 2), generator=g, dtype=F64, device=DEV)


def _offsets(case, seed):
    n, g = case["n"], _gen(seed + 1)
    if case["kind"] == "quadtree":  # within the tolerance that the call asks for
        return (torch.rand(n, generator=g, dtype=F64, device=DEV) - 0.5) * MAX_EDGE
    if case["kind"] == "pcurve":
        return torch.full((n,), 1e-3, dtype=F64, device=DEV)
    z = torch.randn(n, generator=g, dtype=F64, device=DEV)
    return 1e-2 * z.abs() if case["offset"] == "cloud" else 1e-3 * z


MAX_EDGE = 1e-4


def _queries(case, surf, seed):
    uv = _params(case, seed)
    if case["kind"] != "project":
        return _on_normal(surf, uv, _offsets(case, seed))
    # 80 % within a tenth of the extent of the surface, 20 % anywhere in a box six extents wide
    n, g = case["n"], _gen(seed + 1)
    P = _on_normal(surf, uv, 0.1 * (2 * torch.rand(n, generator=g, dtype=F64, device=DEV) - 1))
    far = torch.rand(n, generator=g, dtype=F64, device=DEV) < 0.2
    box = 6 * torch.rand((n, 3), generator=g, dtype=F64, device=DEV) - 2.5
    return torch.where(far[:, None], box, P)


# ------------------------------------------------------------------------------- one pass
def _faces(case, seed):
    r = synth.Rng(synth.SEED_BASE + 104729 * (seed % (1 << 31)))
    surfs = [synth.surface_random(r) for _ in range(case["faces"])]
    # the query counts are the case's own: every seed has the same number of results
    return surfs, _counts(case)


def _counts(case):
    c = synth.Rng(synth.SEED_BASE + 31 * case["faces"] + case["most"])
    return np.exp(c.uniform(case["faces"], math.log(16), math.log(case["most"]))).astype(np.int64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pool":
        surfs, counts = _faces(case, seed)
        budget = int(1.05 * sum(gn.surface_bytes(s) for s in surfs)) + (64 << 20)
        pool = gn.Pool(budget, max_surfaces=len(surfs))
        ids = pool.add(surfs)
        g = _gen(seed)
        P = torch.cat([_on_normal(s, torch.rand((int(c), 2), generator=g, dtype=F64, device=DEV),
                                  1e-3 * torch.randn(int(c), generator=g, dtype=F64, device=DEV))
                       for s, c in zip(surfs, counts)])
        return dict(kind=kind, pool=pool, P=P, batch=gn.Batch(ids, np.concatenate([[0], np.cumsum(counts)])),
                    precision=PREC[case["precision"]])
    surf = _surface(case, seed)
    if kind == "create":
        return dict(kind=kind, surf=surf)
    state = dict(kind=kind, s=gn.Surface(surf))
    if kind in ("eval", "normal"):
        f32 = case.get("dtype") == "fp32"
        uv = _params(case, seed)
        state.update(uv=uv.float() if f32 else uv, mask=case["mask"], f32=f32)
        return state
    state.update(P=_queries(case, surf, seed), precision=PREC[case["precision"]])
    if case.get("host"):
        n = case["n"]
        state["P"] = state["P"].cpu().pin_memory().numpy()
        state["out"] = (torch.empty((n, 2), dtype=F64).pin_memory().numpy(),
                        torch.empty(n, dtype=torch.int32).pin_memory().numpy(),
                        torch.empty(n, dtype=F64).pin_memory().numpy())
    return state


def run(state):
    kind, s = state["kind"], state.get("s")
    if kind == "eval":
        if state["f32"]:
            return s.eval_f32(state["uv"], state["mask"])
        return s.eval(state["uv"], state["mask"])
    if kind == "normal":
        return s.eval_normal(state["uv"], state["mask"])
    if kind == "invert":
        if "out" in state:
            return s.invert_host(state["P"], state["precision"], out=state["out"])
        return s.invert(state["P"], state["precision"])
    if kind == "project":
        return s.project(state["P"], state["precision"])
    if kind == "quadtree":
        return s.invert_quadtree(state["P"], MAX_EDGE, state["precision"])
    if kind == "pcurve":
        return s.pcurve(state["P"], state["precision"])
    if kind == "pool":
        return state["pool"].invert(state["batch"], state["P"], state["precision"])
    new = gn.Surface(state["surf"])
    return new.matrix_n(), new.tree(), new.normal_cones()


# ------------------------------------------------------------------------- work and truth
def work(case):
    kind = case["kind"]
    if kind == "pool":  # the mean of a degree from {2, 3, 5}
        n = int(_counts(case).sum())
        return {"bytes": 52.0 * n, "flops": n * _query_flops(3.33, 3.33)}
    k1, k2 = case["p"] + 1, case["q"] + 1
    net = case["nu"] * case["nv"] * 32.0
    if kind == "create":  # the net in; the span matrices out
        cells = (case["nu"] + case["p"]) * (case["nv"] + case["q"])
        return {"bytes": net + cells * k1 * k2 * 32.0,
                "flops": (case["nu"] - case["p"]) * (case["nv"] - case["q"]) * 8.0 * k1 * k2 * (k1 + k2)}
    n = case["n"]
    if kind == "eval":
        size, blocks = (4 if case["dtype"] == "fp32" else 8), bin(case["mask"]).count("1")
        return {"bytes": n * size * (2.0 + 3 * blocks) + net, "flops": n * 2.0 * 4 * (k1 * k2 + k1 * blocks)}
    if kind == "normal":
        blocks = bin(case["mask"]).count("1")
        return {"bytes": n * 8 * (2.0 + 3 * blocks) + net, "flops": n * 2.0 * 4 * (k1 * k2 + 2 * k1 * blocks)}
    return {"bytes": n * (56.0 if kind == "pcurve" else 52.0) + net, "flops": n * _query_flops(case["p"], case["q"])}


def _query_flops(p, q):
    """Seven evaluations of S, Su, Sv and six 2x2 solves: one accepted seed of six iterations."""
    return 7 * 2 * (4 * (p + 1) * (q + 1) * 2 + 4 * (p + 1) * 3) + 6 * 30


def exact(case, seed):
    kind = case["kind"]
    if kind == "pool":
        return None
    surf = _surface(case, seed)
    if kind == "create":
        # the span polynomials by Taylor's formula at each span's start; the tree's boxes and the
        # normal cones are defined by the library's own sampling
        return _matrix_n(surf), (None, None, None), (None, None, None)
    if kind == "eval":
        uv = _params(case, seed)
        uv = uv.float().double() if case["dtype"] == "fp32" else uv
        picked = [b for k, b in enumerate(BLOCKS) if case["mask"] >> k & 1]
        out = torch.empty((3 * len(picked), len(uv)), dtype=F64, device=DEV)
        for k in range(0, len(uv), 1 << 19):
            D = _ders(surf, uv[k:k + (1 << 19)], max(a + b for a, b in picked))
            for i, b in enumerate(picked):
                out[3 * i:3 * i + 3, k:k + (1 << 19)] = D[b].T
        return out
    if kind == "normal":
        D = _ders(surf, _params(case, seed), 3)
        d = {"".join("u" * a + "v" * b): D[a, b] for a, b in BLOCKS}

        def x(a, b):
            return torch.linalg.cross(d[a], d[b], dim=1)

        blocks = [x("u", "v"), x("uu", "v") + x("u", "uv"), x("uv", "v") + x("u", "vv"),
                  x("uuu", "v") + 2 * x("uu", "uv") + x("u", "uuv"),
                  x("uuv", "v") + x("uu", "vv") + x("u", "uvv"),
                  x("uvv", "v") + 2 * x("uv", "vv") + x("u", "vvv")]
        return torch.cat([b.T for k, b in enumerate(blocks) if case["mask"] >> k & 1])
    if kind == "quadtree":  # no other part of the surface lies within the tolerance of these points
        return _params(case, seed), None, _offsets(case, seed).abs()
    # which of a point's minima the tree's seeds reach, and so which is the answer, is the
    # algorithm's own definition: these outputs are held to the bound of their type
    return None


def _matrix_n(surf):
    p, q, nu, nv = surf["p"], surf["q"], surf["nu"], surf["nv"]

    def taylor(knots, deg, cp):
        """(spans, deg+1, deg+1): power coefficient a of basis function i on each non-empty span."""
        m = [k for k in range(deg, cp) if knots[k] < knots[k + 1]]
        t = torch.as_tensor([knots[k] for k in m], dtype=F64)
        h = torch.as_tensor([knots[k + 1] - knots[k] for k in m], dtype=F64)
        _, d = _basis(knots, deg, cp, t, deg)
        return m, torch.stack([torch.stack([d[a][i] * h ** a / math.factorial(a) for i in range(deg + 1)], 1)
                               for a in range(deg + 1)], 1)

    mu, Tu = taylor(surf["knots_u"], p, nu)
    mv, Tv = taylor(surf["knots_v"], q, nv)
    w = torch.as_tensor(surf["weights"], dtype=F64)
    pw = torch.cat([torch.as_tensor(surf["cps"], dtype=F64) * w[:, None], w[:, None]], 1).reshape(nu, nv, 4)
    out = torch.zeros((p + nu, q + nv, 4, p + 1, q + 1), dtype=F64)
    for i, k in enumerate(mu):
        for j, m in enumerate(mv):
            out[k, m] = torch.einsum("as,stc,bt->cab", Tu[i], pw[k - p:k + 1, m - q:m + 1], Tv[j])
    return out.reshape(-1)
