"""The Newton autotuner times each configuration of the kernel once: shapes that launch the
same kernel in the same way share a time, and among them the lanes a star of the stages around
it are kept."""
import numpy as np
import pytest

import tetwild_gb300 as tw
from tetwild_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

TWINS = [(0, 2, 5), (3, 6, 9)]   # 128 threads and 256, each with 32 stars in flight


@pytest.mark.parametrize("start", [0, 5, 6, 9])
def test_newton_autotune_times_twins_once(ctx, start):
    import torch

    n = 2_001
    xyz, off, tets, cen = syn.star_batch(n, seed=4)
    ctx.set_params(1e-6, 1e-3, 4, 8)
    ctx.mesh_upload(xyz)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (off, tets, cen)]
    out = torch.empty(n, 3, dtype=torch.float64, device="cuda")
    mov = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.set_newton_shape(start)
    try:
        best, ms = ctx.newton_autotune_device(*(a.data_ptr() for a in d), n, out.data_ptr(),
                                              mov.data_ptr())
    finally:
        ctx.set_newton_shape(5)
        ctx.set_params(1e-6, 1e-3)
    assert len(ms) == tw.Context.NEWTON_SHAPES and min(ms) > 0 and ms[best] == min(ms)
    for twins in TWINS:
        assert len({ms[k] for k in twins}) == 1
        if best in twins and start in twins:
            assert best == start
