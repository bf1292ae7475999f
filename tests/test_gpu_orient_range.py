"""Orientation signs of tets whose edges differ by up to 2^250 in length, against exact
integer arithmetic, in both precision modes: products of such edges leave the normal range of
binary32 while the determinant lies well inside it."""
import numpy as np
import pytest

import tetwild_gb300 as tw

pytestmark = pytest.mark.gpu


def _sign(d):
    """The sign of det(d), d of shape (3, 3), in whole numbers."""
    a = [[int(x * 2.0 ** 300) for x in row] for row in d]   # exact: 2^-260 <= |x| < 2^101
    det = (a[0][0] * (a[1][1] * a[2][2] - a[1][2] * a[2][1])
           - a[0][1] * (a[1][0] * a[2][2] - a[1][2] * a[2][0])
           + a[0][2] * (a[1][0] * a[2][1] - a[1][1] * a[2][0]))
    return (det > 0) - (det < 0)


def test_signs_of_long_and_short_edges(ctx):
    rng = np.random.default_rng(8)
    n = 30_000
    d = rng.uniform(-1, 1, (n, 3, 3))
    e = rng.integers(-60, 60, (n, 3))
    e[:, 0] = rng.integers(-155, -145, n)          # one short edge
    e[:, 1:] = rng.integers(0, 100, (n, 2))        # two long ones,
    near = rng.random(n) < 0.7                     # nearly parallel in most
    d[near, 2] = d[near, 1] + d[near, 2] * 0.5 ** rng.integers(1, 20, (int(near.sum()), 1))
    d = np.ldexp(d, e[:, :, None])
    roll = rng.integers(0, 3, n)
    d = np.stack([np.roll(d[i], roll[i], axis=0) for i in range(n)])
    want = np.array([_sign(m) for m in d])
    T = np.zeros((12, n))                          # from the origin: the differences are exact
    T[3:] = d.reshape(n, 9).T
    for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
        ctx.set_precision(prec)
        try:
            flip = ctx.amips(T, tw.TW_ENERGY_RAW, jacobian=False, hessian=False)["flip"]
        finally:
            ctx.set_precision(tw.TW_PRECISION_FP64)
        assert np.array_equal(flip, (want != 1).astype(np.uint8)), int((flip != (want != 1)).sum())
