"""A surface whose bin index does not fit the context's memory budget keeps its grid: the upload
reports that memory ran out, and what follows finds the grid built."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

EPS = 2e-3


def test_grid_stays_when_the_bin_index_does_not_fit():
    V, F = syn.displaced_sphere(6, n_lon=120, n_rings=24)
    P = V * 1.001

    def build(budget, bins):
        c = tw.Context(0, budget)
        c.set_tuning(tw.Context.TUNE_BIN_CELL, bins)
        c.set_params(EPS * EPS, EPS)
        return c

    with build(0, 0.25) as c:
        c.surface_upload(V, F)
        full = c.memory_used()
        want = c.envelope_points(P)
    with build(0, 0.0) as c:
        c.surface_upload(V, F)
        grid = c.memory_used()
    # room for what stays but not for the temporaries beside it
    with build(full, 0.25) as c:
        with pytest.raises(tw.TetWildGpuError):
            c.surface_upload(V, F)
        assert c.memory_used() == grid
        c.set_params(EPS * EPS, EPS)          # the same surface and eps: nothing to build
        assert c.memory_used() == grid
        assert np.array_equal(c.envelope_points(P), want)
