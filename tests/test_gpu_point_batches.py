"""Point queries at the sizes where the host call changes its route (one staged copy up to
256 KB of points and answers, the pipeline above), and where the batch is sorted (from 4096
points on), with points on and beside the surface, far out and NaN: the oracle's answers in
both precision modes, in a context with a memory budget (sorted by index) and without (sorted
records), and the same counters of work either way."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 37, 4095, 4096, 4129, 8190, 8191, 70001])
def test_point_batches_match_oracle(oracle, n):
    rng = np.random.default_rng(n)
    V, F = syn.displaced_sphere(6, n_lon=120, n_rings=24)
    eps = 2e-3
    f = rng.integers(0, len(F), n)
    w = rng.dirichlet([1.0, 1.0, 1.0], n)
    P = np.einsum("ij,ijk->ik", w, V[F[f]])
    d = rng.normal(size=P.shape)
    P += d * (eps * rng.uniform(0, 2, (n, 1)) / np.linalg.norm(d, axis=1, keepdims=True))
    P[5::97] *= 40.0
    P[11::301, 1] = np.nan
    ok = ~np.isnan(P).any(1)
    want = np.ones(n, np.uint8)   # no facet is within eps of a NaN
    want[ok] = oracle.surface(V, F).points_out(P[ok], eps * eps, nthreads=4)
    for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
        tests = []
        for budget in (0, 4 << 30):
            with tw.Context(0, budget) as c:
                c.set_precision(prec)
                c.set_params(eps * eps, eps)
                c.surface_upload(V, F)
                c.reset_stats()
                for _ in range(2):
                    assert np.array_equal(c.envelope_points(P), want)
                tests.append(c.stats()["env_facet_tests"])
        assert tests[0] == tests[1]
