"""The reference-form E / J / H in fewer binary64 instructions (corrections rounded from
binary32, doubled linear forms, quotients from one reciprocal): bit for bit the oracle's, at
scales where the short paths apply and where they must give way -- coordinates beyond
2^+-400, tets far smaller than their coordinates, flat and repeated vertices, zeros,
determinants that are powers of two, infinities and NaN."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _tets(n, edge, offset, rng):
    T = np.empty((12, n))
    R = syn.random_rotations(rng, n)
    base = syn.REGULAR_TET - syn.REGULAR_TET.mean(0)
    sig = np.where(rng.random((n, 1, 1)) < 0.3, 0.6, 0.1)
    P = edge * (np.einsum("nij,kj->nki", R, base) + sig * rng.normal(size=(n, 4, 3)))
    T[:] = (P + offset * rng.random((n, 1, 3))).reshape(n, 12).T
    return T


def _check(ctx, oracle, T, quality):
    g = ctx.amips(T, tw.TW_ENERGY_QUALITY if quality else tw.TW_ENERGY_RAW)
    E, J, H, F = oracle.amips_batch_soa(T, quality=quality)
    for k, want in (("E", E), ("J", J), ("H", H)):
        assert np.array_equal(g[k], want, equal_nan=True), k
    assert np.array_equal(g["flip"], F)


@pytest.mark.parametrize("edge,offset", [(1e-2, 1.0), (1e-2, 100.0), (1.0, 0.0), (1e-6, 1.0),
                                         (1e-9, 1.0), (1e-40, 0.0), (1e-125, 0.0), (1e40, 0.0),
                                         (1e125, 0.0)])
@pytest.mark.parametrize("quality", [False, True])
def test_reference_form_scales(ctx, oracle, edge, offset, quality):
    T = _tets(40_001, edge, offset, np.random.default_rng(11))
    with np.errstate(all="ignore"):
        _check(ctx, oracle, T, quality)


def test_reference_form_special_tets(ctx, oracle):
    rng = np.random.default_rng(12)
    T = _tets(20_000, 1.0, 0.0, rng)
    T[:, 0:2000] = np.round(T[:, 0:2000] * 4) / 4              # short significands, exact quotients
    T[3:6, 2000:2500] = T[0:3, 2000:2500]                       # repeated vertex
    T[2::3, 2500:3000] = 0.0                                    # flat
    T[rng.integers(0, 12, 2000), np.arange(3000, 5000)] = 0.0
    T[:, 5000:6000] = 0.0
    unit = np.array([0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1.0])
    T[:, 5000:5200] = unit[:, None] * 2.0 ** rng.integers(-60, 60, 200)
    T[rng.integers(0, 12, 200), np.arange(6000, 6200)] = rng.choice([np.inf, -np.inf, np.nan], 200)
    with np.errstate(all="ignore"):
        _check(ctx, oracle, T, True)
        keep = np.isfinite(T).all(0)
        _check(ctx, oracle, np.ascontiguousarray(T[:, keep]), False)
