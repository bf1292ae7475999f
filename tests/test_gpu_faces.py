"""Face envelope through the cut (regions of a face known to lie inside as a whole):
every decision equals the oracle's in both precision modes.  The faces cross the lines
of the dispatch: slivers and degenerate faces (never cut), faces below the sample
spacing (vertices only), no second cut and each size of it, faces that one warp samples
and faces that a block shares, vertices and interior samples just inside and just outside
eps, a vertex of many facets, a mesh far finer than the face, batches of one face and of
odd counts."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _faces(V, F, n, eps, rng, lo, hi, thin):
    """Near-tangent triangles at random surface points, circumradius lo..hi eps; `thin` of them
    squeezed to slivers; heights up to and slightly past eps."""
    i = rng.integers(0, len(F), n)
    T = V[F[i]]
    c = np.einsum("ij,ijk->ik", rng.dirichlet([1, 1, 1], n), T)
    nrm = np.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0])
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-300)
    t1 = np.cross(nrm, rng.normal(size=(n, 3)))
    t1 /= np.linalg.norm(t1, axis=1, keepdims=True)
    t2 = np.cross(nrm, t1)
    t2[rng.random(n) < thin] *= 10.0 ** rng.uniform(-8, -2)
    r = np.exp(rng.uniform(np.log(lo * eps), np.log(hi * eps), n))[:, None]
    out = []
    for k in range(3):
        a = 2 * np.pi * (k + rng.uniform(-0.45, 0.45, (n, 1))) / 3
        h = eps * rng.choice([0.0, 0.3, 0.9, 1 - 1e-7, 1 + 1e-7, 1.2], (n, 1),
                             p=[0.2, 0.3, 0.2, 0.15, 0.1, 0.05]) * rng.choice([-1, 1], (n, 1))
        out.append(c + r * (np.cos(a) * t1 + np.sin(a) * t2) + h * nrm)
    return np.hstack(out)


def _both(ctx, tris):
    out = []
    for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
        ctx.set_precision(prec)
        try:
            out.append(ctx.envelope_faces(tris))
        finally:
            ctx.set_precision(tw.TW_PRECISION_FP64)
    return out


@pytest.mark.parametrize("surface", ["sphere", "coarse", "fan", "fine"])
@pytest.mark.parametrize("spacing", [0.5, 2.4])
@pytest.mark.parametrize("size", [(0.2, 3.0), (3.0, 30.0)])
def test_cut_faces_match_oracle(ctx, oracle, surface, spacing, size):
    V, F = {"sphere": lambda: syn.displaced_sphere(2, n_lon=150, n_rings=40),
            "coarse": lambda: syn.icosphere(2),
            "fan": lambda: syn.displaced_sphere(3, n_lon=500, n_rings=6),
            "fine": lambda: syn.icosphere(6)}[surface]()
    eps = 3e-3
    rng = np.random.default_rng(int(10 * spacing + size[0]) + 100 * len(surface))
    tris = _faces(V, F, 1001, eps, rng, *size, thin=0.1)
    tris[::97, 6:9] = tris[::97, 3:6]          # degenerate: a repeated vertex
    if surface == "fan":                       # faces over the pole's many facets
        tris[:60] = _faces(V, F[-2:], 60, eps, rng, 2.0, 10.0, 0.0)
        tris[:60] += np.tile(V[-2] - tris[:60].reshape(60, 3, 3).mean(1), (1, 3))
    ctx.set_params(eps * eps, spacing * eps)
    ctx.surface_upload(V, F)
    want = oracle.surface(V, F).faces_out(tris, eps * eps, spacing * eps, nthreads=8)
    for got in _both(ctx, tris):
        assert np.array_equal(got, want)
    for n in (1, 3, 129):
        for got in _both(ctx, tris[:n]):
            assert np.array_equal(got, want[:n])
    assert 0 < want.sum() < len(want)


def test_cut_far_from_origin(ctx, oracle):
    """Coordinates far larger than eps: the cut's margin (2^-17 of the largest coordinate)
    exceeds eps, and the faces fall back to their samples."""
    V, F = syn.icosphere(3)
    shift = np.array([400.0, -300.0, 500.0])
    for eps in (2e-2, 2e-3):
        tris = _faces(V, F, 301, eps, np.random.default_rng(5), 0.5, 12.0, 0.05) + np.tile(shift, 3)
        ctx.set_params(eps * eps, eps)
        ctx.surface_upload(V + shift, F)
        want = oracle.surface(V + shift, F).faces_out(tris, eps * eps, eps, nthreads=8)
        for got in _both(ctx, tris):
            assert np.array_equal(got, want)
