"""Clearing the statistics and the error word is in order with the next call, whatever other
streams are doing."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

EPS = 2e-3
MODES = [tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED]


@pytest.mark.parametrize("mode", MODES)
def test_clears_are_in_order_with_the_next_call(mode):
    """torch's default stream is the legacy default stream: held busy here, so that a clear
    queued there would run after the calls that follow it."""
    import torch

    V, F = syn.icosphere(2, seed=3)
    P = V[:37] * 1.0005
    busy = lambda: torch.cuda._sleep(40_000_000)  # noqa: E731  (some 20 ms)
    huge = np.array([[0, 0, 0, 1e5, 0, 0, 0, 1e5, 0]], float)   # over 4e6 samples a row

    def fresh():
        c = tw.Context(0)
        c.set_precision(mode)
        c.set_params(EPS * EPS, EPS)
        c.surface_upload(V, F)
        return c

    with fresh() as c:
        want = c.envelope_points(P)
    for _ in range(5):
        torch.cuda.synchronize()
        busy()
        with fresh() as c:                     # counters cleared on creation
            assert np.array_equal(c.envelope_points(P), want)
            torch.cuda.synchronize()
            assert c.stats()["env_queries"] == len(P)
            busy()
            c.reset_stats()
            assert np.array_equal(c.envelope_points(P), want)
            torch.cuda.synchronize()
            assert c.stats()["env_queries"] == len(P)
            busy()
            with pytest.raises(tw.TetWildGpuError, match="sample bound"):
                c.envelope_faces(huge)
            assert np.array_equal(c.envelope_points(P), want)   # no error left over
            with pytest.raises(tw.TetWildGpuError, match="sample bound"):
                c.envelope_faces(huge)                           # nor one wiped
            torch.cuda.synchronize()
