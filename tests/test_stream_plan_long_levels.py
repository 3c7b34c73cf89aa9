"""Streams (k_trsv_stream) of systems with a level of several chunks between short ones: the values a
chunk gathers from global memory must lie in chunks that every warp has left when it is fetched, whatever
the level's length.  A plan is either refused or runs like the level sweep (host only)."""
import numpy as np
import pytest

from vshe import gpu
import test_local_plan as plans


def _levels(sizes, width=1):
    """A symmetric pattern with the given levels, forward and backward: every row is coupled to `width`
    rows or more of the level before and of the one after."""
    start = np.concatenate([[0], np.cumsum(sizes)])
    a, b = [], []
    for k in range(len(sizes) - 1):
        m, q = sizes[k], sizes[k + 1]
        j = np.arange(max(m, q))
        for u in range(width):
            a.append(start[k] + (j * m // len(j) + u) % m)
            b.append(start[k + 1] + (j * q // len(j) + u) % q)
    a, b = np.concatenate(a), np.concatenate(b)
    n = int(start[-1])
    pairs = np.unique(np.concatenate([a * n + b, b * n + a, np.arange(n) * (n + 1)]))
    row, ci = pairs // n, (pairs % n).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int64)
    return rp, ci, np.where(ci == row, 40.0, -1.0), None


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("width", [1, 3])
@pytest.mark.parametrize("long", [4000, 6000, 7000, 7700, 8000, 8192, 8193])
def test_level_of_several_chunks(long, width, precision):
    make = lambda: _levels([600] * 16 + [long] + [600] * 16, width)
    kw = dict(plans.NAT, trsv="per_system")
    rp, ci, v, _ = make()
    if gpu.stream_plan(rp, ci, None, precision=precision, **kw) is None:
        return
    plans.STREAMS["long level"] = (make, kw, precision, 1)
    try:
        plans.test_stream_runs_like_the_level_sweep("long level")
    finally:
        del plans.STREAMS["long level"]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("long", [4000, 7000, 8000, 8193])
def test_same_x_as_task(long, precision):
    import test_gpu_local_sweeps as sweeps
    rp, ci, v, _ = _levels([600] * 16 + [long] + [600] * 16, 3)
    b = np.random.default_rng(1).uniform(-1.0, 1.0, len(rp) - 1)
    assert sweeps._both((rp, ci, v, b), precision, **dict(plans.NAT, trsv="per_system")) == 3
