"""A batch of whole systems (streams) and block tasks (local ones, or some too large to be local), whose
sweeps run side by side: every member's x is the one of its own solve, bit for bit, on the captured
chunk, launched directly under profiling, and after the tables are gone."""
import numpy as np
import pytest

from vshe import gpu
import test_gpu_local_sweeps as sweeps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("sizes", [[1000, 700, 900], [30000, 700]])
def test_members_as_alone(sizes, precision):
    blocks = np.concatenate([[0], np.cumsum(sizes)])
    chain = [sweeps._csr(n, [-40, 40, -41]) for n in (3000, 900)]
    A = sweeps._csr(int(blocks[-1]), [-60, -3, 3, 60])
    o = dict(precision=precision, tol=1e-11, max_iters=400)
    ctx = gpu.Context(0)
    try:
        S = [ctx.system(*c, precond="ilu0", ordering="natural", trsv="per_system", **o) for c in chain]
        S.insert(1, ctx.system(*A, precond="block_ilu0", ordering="multicolor", fill_level=1, blocks=blocks, trsv="per_block", **o))
        alone = [s.solve()[0] for s in S]
        for profiling in (False, True, False):
            ctx.set_profiling(profiling)
            assert all(s["status"] == 0 for s in ctx.batch_solve(S))
            for k in range(3):
                assert np.array_equal(S[k].x(), alone[k])
        ctx.set_task_sweep(0)
        ctx.batch_solve(S)
        for k in range(3):
            assert np.array_equal(S[k].x(), alone[k])
    finally:
        ctx.close()
