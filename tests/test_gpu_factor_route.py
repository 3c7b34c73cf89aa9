"""Which systems k_ilu_cluster factorises: levels short for the rows' kind.  Both routes give the same
factor, bit for bit (test_gpu_chain_factor.py); longer levels measured sooner on the whole grid."""
import numpy as np
import pytest

import test_stream_plan_long_levels as shapes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw, rows, cluster", [
    (dict(precond="ilu0"), 600, True), (dict(precond="ilu0"), 900, False),
    (dict(precond="ilut", ilut_entries=60, ilut_drop=1e-7), 60, True), (dict(precond="ilut", ilut_entries=60, ilut_drop=1e-7), 400, False),
])
def test_route(gpu_ctx, kw, rows, cluster):
    import torch
    from torch.profiler import ProfilerActivity, profile
    rp, ci, v, _ = shapes._levels([rows] * 40)
    n = len(rp) - 1
    S = gpu_ctx.system(rp, ci, v, np.ones(n), trsv="per_system", ordering="natural", tol=1e-10, **kw)
    try:
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            x, st = S.solve()
            torch.cuda.synchronize()
    finally:
        S.free()
    assert st["status"] == 0
    names = [e.key for e in p.key_averages()]
    assert any("k_ilu_cluster" in k for k in names) == cluster
    assert any("k_ilu0" in k for k in names) != cluster
