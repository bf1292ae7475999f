"""Newton steps of many stars in flight per block: positions and flags equal the oracle's
bit for bit in both precision modes, over stars of 0 to 600 tets (rounds that split a star),
caps of 0 and up, both energy forms, batches from one star to more than the slots of the
GPU, stars whose binary32 energies cannot decide a trial (far smaller than their
coordinates, converged, or with flat and inverted tets)."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _join(parts):
    xyz, off, tets, cen = [], [0], [], []
    nv = nt = 0
    for x, o, t, c in parts:
        xyz.append(x)
        tets.append(t + nv)
        cen.append(c + nv)
        off.extend((o[1:] + nt).tolist())
        nv += len(x)
        nt += len(t)
    return (np.vstack(xyz), np.asarray(off, np.int32), np.vstack(tets).astype(np.int32),
            np.concatenate(cen).astype(np.int32))


def _batch(n, seed):
    rng = np.random.default_rng(seed)
    parts = [syn.star_batch(n, seed=seed),
             syn.star_batch(3, seed=seed + 1, mean_tets=600, lo=560, hi=600, radius=0.05),
             syn.star_batch(n // 4 + 1, seed=seed + 2, radius=2e-7),            # far below M
             syn.star_batch(n // 4 + 1, seed=seed + 3, jitter_rel=0.5),         # inverted tets
             syn.star_batch(n // 4 + 1, seed=seed + 4, jitter_rel=1e-9)]        # at the optimum
    xyz, off, tets, cen = _join(parts)
    # some flat stars, a star of one tet and empty stars among the others
    flat = rng.choice(len(cen), max(1, len(cen) // 50), replace=False)
    for s in flat:
        xyz[np.unique(tets[off[s]:off[s + 1]]), 2] = 0.25
    keep = np.diff(off)
    keep[rng.choice(len(cen), max(1, len(cen) // 20), replace=False)] = 0
    keep[0] = 1
    sel = np.concatenate([np.arange(o, o + k) for o, k in zip(off[:-1], keep)])
    return xyz, np.concatenate([[0], np.cumsum(keep)]).astype(np.int32), tets[sel], cen


@pytest.mark.parametrize("n,max_step,max_it", [(1, 15, 20), (40, 15, 20), (40, 0, 5), (40, 3, 0),
                                               (40, 2, 1), (30_000, 1, 8)])
def test_newton_stars_match_oracle(ctx, oracle, n, max_step, max_it):
    xyz, off, tets, cen = _batch(n, seed=n + max_step)
    want, wmoved = oracle.newton_stars(xyz, off, tets, cen, max_step, max_it, nthreads=8)
    wpos, wst = oracle.smooth_stars(xyz, off, tets, cen, max_step=max_step, max_it=max_it,
                                    nthreads=8)
    ctx.set_params(1e-6, 1e-3, max_step, max_it)
    ctx.mesh_upload(xyz)
    try:
        for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
            ctx.set_precision(prec)
            pos, moved = ctx.newton_stars(off, tets, cen)
            assert np.array_equal(moved, wmoved) and np.array_equal(pos, want, equal_nan=True)
            pos, st = ctx.smooth_stars(off, tets, cen)
            assert np.array_equal(st.astype(np.int8), wst) and np.array_equal(pos, wpos)
    finally:
        ctx.set_precision(tw.TW_PRECISION_FP64)


def test_newton_closed_form_same_in_both_modes(ctx):
    xyz, off, tets, cen = _batch(200, seed=9)
    ctx.set_params(1e-6, 1e-3, 15, 20)
    ctx.mesh_upload(xyz)
    got = []
    try:
        ctx.set_energy_form(tw.TW_ENERGY_FORM_CLOSED)
        for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
            ctx.set_precision(prec)
            got.append(ctx.newton_stars(off, tets, cen))
    finally:
        ctx.set_energy_form(tw.TW_ENERGY_FORM_REFERENCE)
        ctx.set_precision(tw.TW_PRECISION_FP64)
    assert np.array_equal(got[0][1], got[1][1])
    assert np.array_equal(got[0][0], got[1][0], equal_nan=True)
