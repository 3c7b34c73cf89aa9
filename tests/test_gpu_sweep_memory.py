"""The sweeps' own copies of the factor (streams, records of the local tasks) are optional memory: a budget
that holds the systems without them takes the systems, whose x is the same with them and without; a SHE problem
with them stays within its bound."""
import numpy as np
import pytest

from vshe import devices as D
from vshe import gpu
import test_gpu_local_sweeps as sweeps

pytestmark = pytest.mark.gpu

OFFSETS = [-700, -3, -2, -1, 1, 2, 3, 700]
KW = {"streams": dict(precond="ilu0", ordering="natural", trsv="per_system", tol=1e-11),
      "local": dict(precond="block_ilu0", ordering="multicolor", fill_level=1, trsv="per_block", blocks=np.arange(0, 40001, 8000), tol=1e-11)}


def _bound(A):
    """vshe_system_create's bound of a system."""
    n, nnz = len(A[0]) - 1, len(A[1])
    return nnz * 56 + n * 168


@pytest.mark.parametrize("kind", sorted(KW))
def test_tables_give_way_to_systems(kind):
    A = sweeps._csr(40000, [-100, 100] if kind == "streams" else OFFSETS)

    def held(budget):
        ctx = gpu.Context(0, budget)
        try:
            S = ctx.system(*A, **KW[kind])
            assert S.solve()[1]["status"] == 0
            return ctx.bytes_in_use()
        finally:
            ctx.close()

    full, bare = held(0), held(_bound(A))
    assert bare < full, "the smallest budget that takes the system leaves no room for tables"
    # the first system with its tables, and the bound of a second one that fits only without them
    ctx = gpu.Context(0, bare + _bound(A) + (full - bare) // 2)
    try:
        S = ctx.system(*A, **KW[kind])
        S.solve()
        x = S.x()
        with_tables = ctx.bytes_in_use()
        T = ctx.system(*A, **KW[kind])
        assert ctx.bytes_in_use() < with_tables + bare
        assert all(s["status"] == 0 for s in ctx.batch_solve([S, T]))
        assert np.array_equal(S.x(), x) and np.array_equal(T.x(), x)
        S.solve()
        assert np.array_equal(S.x(), x)
    finally:
        ctx.close()
    assert with_tables == full


def test_bounds_hold_with_tables(gpu_ctx):
    for dev, cfg, o in [(*D.config1(), dict(precond="ilu0", ordering="natural")),
                        (*D.config2(60, 20, 60, 1), dict(precond="block_ilu0", ordering="multicolor", fill_level=1)),
                        (*D.config2(40, 12, 60, 3), dict(precond="block_ilu0", ordering="multicolor", fill_level=1))]:
        for precision in ("mixed", "fp64"):
            before = gpu_ctx.bytes_in_use()
            P = gpu.SheProblem(gpu_ctx, dev, cfg, precision=precision, tol=1e-8, max_iters=2000, **o)
            try:
                P.run()
                held = gpu_ctx.bytes_in_use() - before
                assert 0 < held <= P.info["bytes_estimate"]
            finally:
                P.free()
