"""Surfaces for which the grid or only the bin index is unsuitable (a leaf over too many cells or
bins, found while the leaves are counted): what is unsuitable is left out, the answers are the
oracle's in both modes, and a suitable surface uploaded next gets both again."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

EPS = 2e-3


def _with(V, F, tri):
    return np.vstack([V, tri]), np.vstack([F, [[len(V), len(V) + 1, len(V) + 2]]]).astype(np.int32)


def _held(V, F, bins):
    with tw.Context(0) as c:
        c.set_tuning(tw.Context.TUNE_BIN_CELL, bins)
        c.set_params(EPS * EPS, EPS)
        c.surface_upload(V, F)
        return c.memory_used()


@pytest.mark.parametrize("what", ["bins", "grid", "all sizes"])
def test_unsuitable_index_is_left_out(oracle, what):
    rng = np.random.default_rng(6)
    V0, F0 = syn.displaced_sphere(6, n_lon=200, n_rings=40)
    ext = np.ptp(V0[F0], axis=1).max(1).mean()
    if what == "bins":     # 20 bins a side: over 4096; 25 cells a side: below 65536
        V, F = _with(V0, F0, 0.2 + ext * np.array([[0, 0, 0], [5, 5, 0], [0, 5, 5.0]]))
    elif what == "grid":
        V, F = _with(V0, F0, 0.2 + ext * np.array([[0, 0, 0], [60, 60, 0], [0, 60, 60.0]]))
    else:
        V = (rng.normal(size=(3000, 1, 3))
             + rng.normal(size=(3000, 3, 3)) * 10.0 ** rng.uniform(-4, 0.3, (3000, 1, 1)))
        V, F = V.reshape(-1, 3), np.arange(9000, dtype=np.int32).reshape(-1, 3)
    suitable = _held(V0, F0, 0.25)
    with_bins, without = _held(V, F, 0.25), _held(V, F, 0.0)
    assert with_bins == without and suitable > _held(V0, F0, 0.0)
    P = np.vstack([V, V[F].mean(1)]) + EPS * rng.normal(size=(len(V) + len(F), 3))
    want = oracle.surface(V, F).points_out(P, EPS * EPS, nthreads=8)
    for mode in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
        with tw.Context(0) as c:
            c.set_precision(mode)
            c.set_params(EPS * EPS, EPS)
            for _ in range(3):
                c.surface_upload(V, F)
            assert np.array_equal(c.envelope_points(P), want)
            c.surface_upload(V0, F0)
            P0 = V0 * (1 + 0.8 * EPS)
            assert np.array_equal(c.envelope_points(P0), oracle.surface(V0, F0).points_out(P0, EPS * EPS))
