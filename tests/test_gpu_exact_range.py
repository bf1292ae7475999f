"""Signs, gradients and Hessians over the whole range of binary64 coordinates, far beyond the
range of binary32: tets whose coordinates along one axis are 2^-95 or smaller beside ones up
to 2^48 along the others, and tets whose edges differ by factors up to 2^250."""
import numpy as np
import pytest

import tetwild_gb300 as tw

pytestmark = pytest.mark.gpu


def _flat_axis(rng, n):
    P = rng.normal(size=(n, 4, 3)) * 2.0 ** rng.integers(0, 49, (n, 1, 1))
    k = rng.integers(0, 3, n)
    P[np.arange(n), :, k] = rng.normal(size=(n, 4)) * 2.0 ** rng.integers(-170, -94, (n, 1))
    return np.ascontiguousarray(P.reshape(n, 12).T)


def _short(rng, n):
    """Coordinates of few bits, a quarter of them zero."""
    P = np.round(rng.normal(size=(n, 4, 3)) * 4) / 4 * 2.0 ** rng.integers(-5, 5, (n, 1, 3))
    P[rng.random(P.shape) < 0.25] = 0.0
    return np.ascontiguousarray(P.reshape(n, 12).T)


@pytest.mark.parametrize("make,n", [(_flat_axis, 40_001), (_short, 400_001)])
def test_reference_form_values(ctx, oracle, make, n):
    T = make(np.random.default_rng(5), n)
    with np.errstate(all="ignore"):
        g = ctx.amips(T, tw.TW_ENERGY_RAW)
        want = oracle.amips_batch_soa(T, quality=False)
    for k, w in zip(("E", "J", "H"), want):
        same = (w == g[k]) | np.isnan(w) & np.isnan(g[k])
        assert same.all(), (k, int((~same).sum()))
