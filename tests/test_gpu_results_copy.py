"""x_full of more than 64 MB into pageable memory (pages faulted in by several threads ahead of the copies)
and into pinned memory (one copy): the same values."""
import ctypes as C

import numpy as np
import pytest

from vshe import devices as D
from vshe import gpu

pytestmark = pytest.mark.gpu


def test_pageable_and_pinned():
    import torch
    from torch.profiler import ProfilerActivity, profile
    dev, cfg = D.config2(100, 25, 240, 3)
    ctx = gpu.Context(0)
    try:
        P = gpu.SheProblem(ctx, dev, cfg, precond="block_ilu0", ordering="multicolor", fill_level=0, tol=1e-3)
        P.run()
        n = P.info["n_even"] + P.info["n_odd"]
        pinned = torch.empty(n, dtype=torch.float64).pin_memory()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            ctx._check(gpu._she_lib().vshe_she_results(ctx.h, P.h, C.cast(pinned.data_ptr(), C.POINTER(C.c_double)), None, None))
            torch.cuda.synchronize()
        copies = sum(e.count for e in p.key_averages() if "DtoH" in e.key)
        x, _, _ = P.results()
        assert x.nbytes > 64 << 20 and np.any(x != 0.0)
        assert np.array_equal(x, pinned.numpy())
        assert copies == 1
    finally:
        ctx.close()
