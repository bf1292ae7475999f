"""Workloads of the query path, through the public binding (``tetwild_gb300.Context``).

Each case is one call (or the short sequence of calls) that a TetWild operator
or driver makes: the smallest host call of one vertex, whole batches on device
buffers, host-buffer batches, in the default binary64 mode and in the
certified binary32 mode.  Sizes are those of the repository's configurations,
benchmark and tests, with odd counts so that no batch divides evenly.

``run`` ends with ``Context.synchronize`` after a device-pointer call: the
operators read the answers next, and the device error word is reported there.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

FP64, CERT = "fp64", "certified"


def listed():
    return [
        # isPointOutEnvelop for the vertices that one operator touches: the icosphere
        # configuration's 1,280 facets, stage-1 eps; launches and waits are all there is
        dict(name="points_call_fp64", kind="points", n=37, host=True, precision=FP64,
             surface="icosphere", detail=3, eps=1.46e-3),
        # a batch of point queries from an application's own (pageable) arrays, default mode
        dict(name="points_host_fp64", kind="points", n=300_007, host=True, precision=FP64,
             surface="torus", detail=64, eps=2.2e-3),
        # the benchmark's point batch: 10M resident points, 100,000-facet displaced sphere
        dict(name="points_10m_cert", kind="points", n=10_000_000, host=False, precision=CERT,
             surface="sphere", detail=500, eps=1e-3),
        # E / J / H / flip of a tet batch with the reference's own operations
        dict(name="amips_1m_fp64", kind="amips", n=1_000_003, precision=FP64),
        # the benchmark's energy batch
        dict(name="amips_4m_cert", kind="amips", n=4_000_000, precision=CERT),
        # isFaceOutEnvelop over the tracked surface at stage 1: sampling distance above eps
        # (State.cpp:38-39), edges from a tenth of to the ideal length, default mode
        dict(name="faces_20k_fp64", kind="faces", n=20_011, precision=FP64, surface="icosphere",
             detail=4, eps=1.46e-3, sd=3.46e-3, edge_lo=0.02, edge_hi=0.17),
        # the same after refinement: many small faces, sampling distance eps / 2
        dict(name="faces_300k_cert", kind="faces", n=300_007, precision=CERT, surface="sphere",
             detail=500, eps=1e-3, sd=5e-4, edge_lo=0.004, edge_hi=0.03),
        # NewtonsMethod to convergence, the reference's caps (15 steps, 20 halvings)
        dict(name="newton_20k_fp64", kind="newton", n=20_000, precision=FP64, max_step=15,
             max_it=20),
        # the benchmark's smoothing pass: half interior, half surface stars
        dict(name="smooth_200k_cert", kind="smooth", n=200_000, host=False, precision=CERT,
             surface="sphere", detail=500, eps=1e-3, sd=5e-4, max_step=1, max_it=8),
        # one colour class of VertexSmoother::smooth from host arrays, default mode and caps
        dict(name="smooth_host_fp64", kind="smooth", n=1_501, host=True, precision=FP64,
             surface="icosphere", detail=4, eps=1.46e-3, sd=3.46e-3, max_step=15, max_it=20),
        # EdgeCollapser's checks of a pass's candidates from host arrays
        dict(name="collapse_30k_cert", kind="collapse", n=30_011, precision=CERT,
             surface="sphere", detail=250, eps=1.5e-3, sd=1.5e-3),
        # opening a surface: tree, grid and index of 100,000 facets, then the first query
        dict(name="surface_open_cert", kind="open", n=4_099, precision=CERT, surface="sphere",
             detail=500, eps=1e-3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "points", "amips", "faces", "newton", "smooth", "collapse", "open"])
    c = dict(kind=kind, precision=rng.choice([FP64, CERT]))
    surface = rng.choice(["sphere", "icosphere", "torus"])
    detail = {"sphere": lambda: _log(rng, 60, 500), "icosphere": lambda: rng.randint(2, 5),
              "torus": lambda: _log(rng, 24, 200)}[surface]()
    if kind not in ("amips", "newton"):
        c.update(surface=surface, detail=detail, eps=math.exp(rng.uniform(math.log(7e-4), math.log(4e-3))))
    cert = c["precision"] == CERT
    if kind == "points":
        c["host"] = rng.random() < 0.5
        c["n"] = _log(rng, 9, 1_000_000 if c["host"] or not cert else 10_000_000)
    elif kind == "amips":
        c["n"] = _log(rng, 300, 4_000_000 if cert else 1_000_000)
    elif kind == "faces":
        c["n"] = _log(rng, 50, 300_000 if cert else 20_000)
        c["sd"] = c["eps"] * rng.uniform(0.5, 2.4)
        c["edge_lo"] = 2 * c["eps"] * rng.uniform(1, 4)
        c["edge_hi"] = c["edge_lo"] * rng.uniform(1.5, 6)
    elif kind == "newton":
        c["n"] = _log(rng, 50, 20_000)
        c["max_step"], c["max_it"] = rng.choice([(15, 20), (1, 8), (4, 20)])
    elif kind == "smooth":
        c["host"] = rng.random() < 0.5
        c["n"] = _log(rng, 50, 200_000 if cert and not c["host"] else 20_000)
        c["sd"] = c["eps"] * rng.uniform(0.5, 2.4)
        c["max_step"], c["max_it"] = (1, 8) if c["n"] > 20_000 else rng.choice([(15, 20), (1, 8)])
    elif kind == "collapse":
        c["n"] = _log(rng, 100, 30_000)
        c["sd"] = c["eps"] * rng.uniform(0.5, 2.4)
    else:
        c["n"] = _log(rng, 9, 20_000)
    return c


# ---- inputs ------------------------------------------------------------------------------
def _surface(case, seed):
    if case["surface"] == "sphere":
        return syn.displaced_sphere(seed, n_lon=case["detail"], n_rings=max(4, case["detail"] // 5))
    if case["surface"] == "icosphere":
        return syn.icosphere(case["detail"], seed=seed)
    V, F = syn.torus(n_major=case["detail"], n_minor=max(8, case["detail"] // 2))
    return V * (1.0 + np.random.default_rng(seed).normal(0.0, 5e-4, (len(V), 1))), F


def _on_surface(V, F, n, g):
    """n points uniform by area on (V, F) and their facets' unit normals, on the GPU."""
    V, F = torch.from_numpy(V).cuda(), torch.from_numpy(F.astype(np.int64)).cuda()
    A, B, C = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    nrm = torch.linalg.cross(B - A, C - A)
    area = nrm.norm(dim=1)
    cdf = torch.cumsum(area, 0)
    u = torch.rand(3, n, generator=g, device="cuda", dtype=torch.float64)
    f = torch.searchsorted(cdf, u[0] * cdf[-1]).clamp_(max=len(F) - 1)
    a, b = u[1], u[2]
    fold = a + b > 1
    a, b = torch.where(fold, 1 - a, a)[:, None], torch.where(fold, 1 - b, b)[:, None]
    return A[f] + a * (B[f] - A[f]) + b * (C[f] - A[f]), nrm[f] / area[f, None]


def _points(V, F, n, eps, g):
    """Points on the surface offset along the facet normal by U(-2 eps, 2 eps)."""
    P, N = _on_surface(V, F, n, g)
    off = torch.rand(n, 1, generator=g, device="cuda", dtype=torch.float64)
    return (P + (4 * off - 2) * eps * N).contiguous()


def _faces(V, F, case, g):
    """Triangles in the tangent plane of random surface points, circumradius log-uniform for
    edges in [edge_lo, edge_hi], each vertex offset along the normal by U(-0.4, 0.4) eps."""
    n = case["n"]
    P, N = _on_surface(V, F, n, g)
    u = torch.rand(n, 8, generator=g, device="cuda", dtype=torch.float64)
    ax = torch.zeros_like(N)
    ax[torch.arange(n, device="cuda"), N.abs().argmin(1)] = 1.0
    t1 = torch.linalg.cross(N, ax)
    t1 = t1 / t1.norm(dim=1, keepdim=True)
    t2 = torch.linalg.cross(N, t1)
    lo, hi = math.log(case["edge_lo"]), math.log(case["edge_hi"])
    r = torch.exp(lo + (hi - lo) * u[:, 0]) / math.sqrt(3.0)
    out = []
    for k in range(3):
        ang = 2 * math.pi * (u[:, 1] + (k + 0.5 * (u[:, 2 + k] - 0.5)) / 3)
        h = (0.8 * u[:, 5 + k] - 0.4) * case["eps"]
        out.append(P + (r * torch.cos(ang))[:, None] * t1 + (r * torch.sin(ang))[:, None] * t2
                   + h[:, None] * N)
    return torch.cat(out, 1).contiguous()


def _tets(n, g, edge=0.01, sigma_rel=0.1):
    """SoA [12, n]: regular tets of the given edge, random rotations, centres uniform in the
    unit cube, every coordinate perturbed by N(0, sigma_rel edge)."""
    q = torch.randn(4, n, generator=g, device="cuda", dtype=torch.float64)
    w, x, y, z = q / q.norm(dim=0)
    R = [[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
         [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
         [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]]
    c = torch.rand(3, n, generator=g, device="cuda", dtype=torch.float64)
    T = sigma_rel * edge * torch.randn(12, n, generator=g, device="cuda", dtype=torch.float64)
    base = (syn.REGULAR_TET - syn.REGULAR_TET.mean(0)) * edge
    for j in range(4):
        for k in range(3):
            T[3 * j + k] += c[k] + sum(R[k][m] * float(base[j, m]) for m in range(3))
    return T


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _context(case, V=None, F=None):
    ctx = tw.Context(torch.cuda.current_device())
    ctx.set_precision(tw.TW_PRECISION_FP32_CERTIFIED if case["precision"] == CERT
                      else tw.TW_PRECISION_FP64)
    eps = case.get("eps", 0.0)
    ctx.set_params(eps * eps, case.get("sd", eps), case.get("max_step", 15), case.get("max_it", 20))
    if V is not None:
        ctx.surface_upload(V, F)
    return ctx


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(kind=kind, n=n, host=bool(case.get("host")))
    if kind == "amips":
        s["ctx"] = _context(case)
        s["T"] = _tets(n, g)
        s["E"] = torch.empty(n, dtype=torch.float64, device="cuda")
        s["J"] = torch.empty(3, n, dtype=torch.float64, device="cuda")
        s["H"] = torch.empty(9, n, dtype=torch.float64, device="cuda")
        s["flip"] = torch.empty(n, dtype=torch.uint8, device="cuda")
        return s
    if kind == "newton":
        s["ctx"] = _context(case)
        xyz, off, tets, cen = syn.star_batch(n, seed=seed)
        s["ctx"].mesh_upload(xyz)
        s.update(off=_dev(off), tets=_dev(tets), cen=_dev(cen),
                 pos=torch.empty(n, 3, dtype=torch.float64, device="cuda"),
                 status=torch.empty(n, dtype=torch.uint8, device="cuda"))
        return s
    V, F = _surface(case, seed)
    if kind == "open":
        s["ctx"] = _context(case)
        s.update(V=V, F=F, P=_points(V, F, n, case["eps"], g).cpu().numpy())
        return s
    s["ctx"] = ctx = _context(case, V, F)
    if kind == "points":
        P = _points(V, F, n, case["eps"], g)
        s["P"] = P.cpu().numpy() if s["host"] else P
        s["out"] = None if s["host"] else torch.empty(n, dtype=torch.uint8, device="cuda")
    elif kind == "faces":
        s["tris"] = _faces(V, F, case, g)
        s["out"] = torch.empty(n, dtype=torch.uint8, device="cuda")
    else:
        xyz, off, tets, ff, cen, kinds = syn.mixed_star_batch(V, F, n, case["eps"], seed=seed)
        ctx.mesh_upload(xyz)
        if kind == "collapse":
            # the centre onto the first ring vertex; surface stars track v1 (not v2)
            v12 = np.stack([cen, tets[off[:-1], 1]], 1).astype(np.int32)
            flags = (kinds * tw.TW_CV_V1_SURFACE).astype(np.uint8)
            s.update(v12=v12, flags=flags, off=off, tets=tets, ff=ff)
        elif s["host"]:
            s.update(off=off, tets=tets, ff=ff, cen=cen, kinds=kinds)
        else:
            s.update(off=_dev(off), tets=_dev(tets), ff=_dev(ff), cen=_dev(cen), kinds=_dev(kinds),
                     pos=torch.empty(n, 3, dtype=torch.float64, device="cuda"),
                     status=torch.empty(n, dtype=torch.uint8, device="cuda"))
    return s


def run(s):
    ctx, kind, n = s["ctx"], s["kind"], s["n"]
    if kind == "points" and s["host"]:
        return ctx.envelope_points(s["P"])
    if kind == "points":
        ctx.envelope_points_device(s["P"].data_ptr(), n, s["out"].data_ptr())
        ctx.synchronize()
        return s["out"]
    if kind == "faces":
        ctx.envelope_faces_device(s["tris"].data_ptr(), n, s["out"].data_ptr())
        ctx.synchronize()
        return s["out"]
    if kind == "amips":
        ctx.amips_device(s["T"].data_ptr(), n, tw.TW_ENERGY_QUALITY, s["E"].data_ptr(),
                         s["J"].data_ptr(), s["H"].data_ptr(), s["flip"].data_ptr())
        ctx.synchronize()
        return [s["E"], s["J"], s["H"], s["flip"]]
    if kind == "newton":
        ctx.newton_stars_device(s["off"].data_ptr(), s["tets"].data_ptr(), s["cen"].data_ptr(), n,
                                s["pos"].data_ptr(), s["status"].data_ptr())
        ctx.synchronize()
        return [s["pos"], s["status"]]
    if kind == "smooth" and s["host"]:
        return list(ctx.smooth_stars(s["off"], s["tets"], s["cen"], s["ff"], s["kinds"]))
    if kind == "smooth":
        ctx.smooth_stars_device(s["off"].data_ptr(), s["tets"].data_ptr(), s["ff"].data_ptr(),
                                s["cen"].data_ptr(), s["kinds"].data_ptr(), n, len(s["tets"]),
                                s["pos"].data_ptr(), s["status"].data_ptr())
        ctx.synchronize()
        return [s["pos"], s["status"]]
    if kind == "collapse":
        return ctx.collapse_check(s["v12"], s["flags"], s["off"], s["tets"], s["ff"])
    ctx.surface_upload(s["V"], s["F"])
    return ctx.envelope_points(s["P"])


def _surface_sizes(case):
    d = case["detail"]
    if case["surface"] == "sphere":
        r = max(4, d // 5)
        return d * r + 2, 2 * d * r
    if case["surface"] == "icosphere":
        return 10 * 4 ** d + 2, 20 * 4 ** d
    return d * max(8, d // 2), 2 * d * max(8, d // 2)


def work(case):
    """Bytes: inputs once, outputs once.  flops: the arithmetic of the query itself (one
    point-triangle distance a point or sample, the closed-form E / J / H a tet)."""
    kind, n = case["kind"], case["n"]
    if kind == "points":
        return dict(bytes=25 * n, flops=60 * n)
    if kind == "amips":
        return dict(bytes=201 * n, flops=250 * n)
    if kind == "faces":
        edge = math.sqrt(case["edge_lo"] * case["edge_hi"])
        samples = 3 + 0.43 * edge * edge / (0.87 * case["sd"] ** 2)
        return dict(bytes=73 * n, flops=80 * samples * n)
    if kind == "open":
        nv, nf = _surface_sizes(case)
        return dict(bytes=24 * nv + 12 * nf + 25 * n, flops=100 * nf)
    per_tet, verts = 24, 14   # tets and vertices of a star, Poisson(24) tets
    star = 24 * verts + 17 * per_tet + 30
    if kind == "collapse":
        return dict(bytes=star * n, flops=200 * per_tet * n)
    steps = min(case["max_step"], 5)
    return dict(bytes=star * n, flops=400 * per_tet * steps * n)


def exact(case, seed):
    """E, J and H of the conformal AMIPS energy in closed form, in 64 bits (D < 0: a positively
    oriented tet); the other kinds
    answer with decisions (whole numbers) or with the end of an iteration whose every accepted
    step a rounding may decide."""
    if case["kind"] != "amips":
        return None
    T = prepare_tets(case, seed)
    p0, p1, p2, p3 = T[0:3], T[3:6], T[6:9], T[9:12]
    wb, wc = 1 / math.sqrt(3.0), 1 / math.sqrt(6.0)
    a = p0 - p3
    b = ((p0 - p1) + (p3 - p1)) * wb
    c = ((p0 - p2) + (p1 - p2) + (p3 - p2)) * wc
    cross = lambda u, v: torch.linalg.cross(u, v, dim=0)  # noqa: E731
    bc = cross(b, c)
    N = (a * a).sum(0) + (b * b).sum(0) + (c * c).sum(0)
    D = (a * bc).sum(0)
    g = bc + wb * cross(c, a) + wc * cross(a, b)
    gN = 2 * (a + wb * b + wc * c)
    r = (D * D) ** (-1.0 / 3.0)
    E = torch.where(D < 0, N * r, torch.full_like(N, tw.MAX_ENERGY))
    J = r * (gN - (2.0 / 3.0) * N / D * g)
    s1, s2 = (2.0 / 3.0) * r / D, (10.0 / 9.0) * N * r / (D * D)
    H = torch.empty(9, case["n"], dtype=torch.float64, device="cuda")
    for i in range(3):
        for j in range(3):
            H[3 * i + j] = (3 * r if i == j else 0.0) - s1 * (gN[i] * g[j] + g[i] * gN[j]) \
                + s2 * g[i] * g[j]
    return [E, J, H, None]


def prepare_tets(case, seed):
    return _tets(case["n"], torch.Generator(device="cuda").manual_seed(seed))
