"""Nearest facets with leaves culled by certified bounds: closest point, squared distance
and facet equal the oracle's in both precision modes, over cells of many leaves (the pole of
a lat-long sphere, slivers and a degenerate facet), at equal distances (vertices, edge
points) and for points around eps."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _slivers(rng):
    V, F = [np.zeros(3)], []
    for k in range(120):
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        e = np.cross(d, rng.normal(size=3))
        V += [0.3 * d, 0.3 * d + 10.0 ** rng.uniform(-7, -2) * e / np.linalg.norm(e)]
        F.append((0, 2 * k + 1, 2 * k + 2))
    F.append((0, 1, 1))
    return np.asarray(V), np.asarray(F, np.int32)


@pytest.mark.parametrize("surface", ["pole", "slivers", "coarse"])
def test_nearest_culled_matches_oracle(ctx, oracle, surface):
    rng = np.random.default_rng(3)
    V, F = {"pole": lambda: syn.displaced_sphere(4, n_lon=400, n_rings=20),
            "slivers": lambda: _slivers(rng), "coarse": lambda: syn.icosphere(1)}[surface]()
    eps = 5e-3
    f = rng.integers(0, len(F), 4001)
    w = rng.random((4001, 3)) ** 3
    w[::5] = np.eye(3)[rng.integers(0, 3, len(w[::5]))]          # vertices
    w[1::5, 0] = 0.0                                             # edge points
    w /= w.sum(1, keepdims=True)
    P = np.einsum("ij,ijk->ik", w, V[F[f]])
    d = rng.normal(size=P.shape)
    d *= eps * rng.choice([0.0, 0.5, 0.999, 1.5], (4001, 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    P += d
    if surface == "pole":
        P[:1000] = V[-2] + rng.normal(size=(1000, 3)) * 0.5 * eps
    ctx.set_params(eps * eps, eps)
    ctx.surface_upload(V, F)
    wq, wd, wf = oracle.surface(V, F).nearest(P)
    for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
        ctx.set_precision(prec)
        try:
            q, dd, ff = ctx.nearest_points(P)
        finally:
            ctx.set_precision(tw.TW_PRECISION_FP64)
        assert np.array_equal(dd, wd) and np.array_equal(ff, wf) and np.array_equal(q, wq)
