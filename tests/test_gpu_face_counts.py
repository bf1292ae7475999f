"""The statistics of envelope queries count points and samples of faces, not the pieces by which
faces are decided as a whole."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

EPS = 2e-3
MODES = [tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED]


def _faces(V, F, push):
    A, B, C = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    n = np.cross(B - A, C - A)
    n *= push / np.linalg.norm(n, axis=1, keepdims=True)
    return np.hstack([A + n, B + n, C + n])


@pytest.mark.parametrize("mode", MODES)
def test_face_statistics_count_samples(oracle, mode):
    V, F = syn.icosphere(2, seed=3)
    with tw.Context(0) as c:
        c.set_precision(mode)
        c.set_params(EPS * EPS, EPS)
        c.surface_upload(V, F)
        # the surface itself: pieces decide every face, no sample is queried
        tris = _faces(V, F, 0.0)
        c.reset_stats()
        assert not c.envelope_faces(tris).any()
        st = c.stats()
        assert st["env_queries"] == 0 and st["env_facet_tests"] == 0
        # eps away: pieces decide nothing, the samples do (the vertices once more, where the
        # pieces looked for one that is out)
        tris = _faces(V, F, EPS * (1 - 1e-9))
        c.reset_stats()
        out = c.envelope_faces(tris)
        assert np.array_equal(out, oracle.surface(V, F).faces_out(tris, EPS * EPS, EPS))
        samples = sum(len(oracle.sample_triangle(t, EPS)) for t in tris)
        st = c.stats()
        assert len(tris) < st["env_queries"] <= samples + 3 * len(tris)
        assert st["env_facet_tests"] >= st["env_queries"] - 3 * len(tris)
