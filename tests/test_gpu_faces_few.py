"""Batches of few faces: a face a warp in the cut and a face a block in the sampling, with and
without a grid, at the sizes where the launches change (one face, the warps of a block, one
block a face on every SM and one more); answers equal the oracle's in both modes.  A large face
that is out is found so by its first samples."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

EPS, SD = 2e-3, 1e-3
MODES = [tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED]


def _surface(grid):
    V, F = syn.icosphere(3, seed=2)
    if not grid:   # a facet over too many cells
        V = np.vstack([V, [[-1e3, 3, 0], [1e3, 3, 0], [0, 3, 1e3]]])
        F = np.vstack([F, [[len(V) - 3, len(V) - 2, len(V) - 1]]]).astype(np.int32)
    return V, F


def _faces(V, F, n, rng):
    f = rng.integers(0, 1280, n)
    A, B, C = V[F[f, 0]], V[F[f, 1]], V[F[f, 2]]
    N = np.cross(B - A, C - A)
    N /= np.linalg.norm(N, axis=1, keepdims=True)
    cen = (A + B + C) / 3
    grow = 10.0 ** rng.uniform(-2.5, 0.2, (n, 1))    # a vertex alone to hundreds of samples
    off = EPS * rng.choice([0.0, 0.9, 0.99999, 1.5], (n, 1)) * N
    return np.hstack([cen + grow * (X - cen) + off for X in (A, B, C)])


@pytest.mark.parametrize("grid", [True, False])
@pytest.mark.parametrize("n", [1, 4, 9, 608, 609, 2433])
def test_few_faces_match_oracle(oracle, grid, n):
    V, F = _surface(grid)
    tris = _faces(V, F, n, np.random.default_rng(n))
    want = oracle.surface(V, F).faces_out(tris, EPS * EPS, SD, nthreads=8)
    for mode in MODES:
        with tw.Context(0) as c:
            c.set_precision(mode)
            c.set_params(EPS * EPS, SD)
            c.surface_upload(V, F)
            for _ in range(2):
                assert np.array_equal(c.envelope_faces(tris), want)


@pytest.mark.parametrize("mode", MODES)
def test_a_large_face_that_is_out_is_probed_first(mode):
    V, F = _surface(False)
    tri = np.array([[3.0, 0.0, 0.0, 3.1, 0.0, 0.0, 3.0, 0.1, 0.0]])   # some 5000 samples
    with tw.Context(0) as c:
        c.set_precision(mode)
        c.set_params(EPS * EPS, SD)
        c.surface_upload(V, F)
        c.reset_stats()
        assert c.envelope_faces(tri).tolist() == [1]
        assert 0 < c.stats()["env_queries"] <= 32
