"""Grid and bin-index build (32 leaves a warp, slabs per leaf, mask columns): point decisions
at eps (1 -+ 1e-7) of random facet points equal the oracle's for facet counts around a warp's
and a block's share, facets of very different sizes (one spanning too many cells or bins for
the index: the grid or the tree serves), needle and degenerate facets, axis-aligned facets
(axes that do not depend on z) and a box flat in each direction."""
import numpy as np
import pytest

import tetwild_gb300 as tw

pytestmark = pytest.mark.gpu


def _soup(n, rng, size, flat=None, aligned=False):
    T = rng.random((n, 1, 3)) + (rng.random((n, 3, 3)) - 0.5) * size
    if aligned:
        k = rng.integers(0, 3, n)
        T[np.arange(n), 1:, k] = T[np.arange(n), :1, k]
    T[::7, 2] = T[::7, 1] + 1e-7 * rng.normal(size=T[::7, 1].shape)   # needles
    T[3::11, 2] = T[3::11, 0]                                          # degenerate
    if flat is not None:
        T[..., flat] = 0.3 + 1e-3 * T[..., flat]
    return T.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(n, 3)


@pytest.mark.parametrize("n,size,flat,aligned", [
    (1, 0.5, None, False), (31, 0.2, None, False), (33, 0.2, 0, True), (127, 0.1, 1, False),
    (129, 0.1, 2, True), (1500, 0.05, None, True), (1500, 0.05, None, False)])
@pytest.mark.parametrize("big", [False, True])
def test_index_of_soups(ctx, oracle, n, size, flat, aligned, big):
    rng = np.random.default_rng(n + 7 * big)
    V, F = _soup(n, rng, size, flat, aligned)
    if big:   # facets far larger than the others
        V = np.vstack([V, [[-40.0, -40, -40], [60, -40, 10], [10, 60, 40.0]]])
        F = np.vstack([F, [[3 * n, 3 * n + 1, 3 * n + 2]]]).astype(np.int32)
    eps = 4e-3
    w = rng.random((6000, 3)) ** 3
    w /= w.sum(1, keepdims=True)
    X = np.einsum("ij,ijk->ik", w, V[F[rng.integers(0, len(F), 6000)]])
    d = rng.normal(size=X.shape)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    P = X + d * (eps * np.where(rng.random(6000) < 0.5, 1 - 1e-7, 1 + 1e-7))[:, None]
    P[::9] = rng.uniform(-1, 2, P[::9].shape)
    want = oracle.surface(V, F).points_out(P, eps * eps, nthreads=8)
    ctx.set_params(eps * eps, eps)
    try:
        for bins in (0.25, 3.0, 0.0):
            ctx.set_tuning(tw.Context.TUNE_BIN_CELL, bins)
            ctx.surface_upload(V, F)
            for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
                ctx.set_precision(prec)
                assert np.array_equal(ctx.envelope_points(P), want), (bins, prec)
    finally:
        ctx.set_precision(tw.TW_PRECISION_FP64)
        ctx.set_tuning(tw.Context.TUNE_BIN_CELL, 0.25)
