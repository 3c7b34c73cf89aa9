"""Factorisation of a system with short levels on one thread-block cluster (k_ilu_cluster) against the
grid-wide factorisation of the same system, which the grid-wide sweep modes take: the same factor
values, bit for bit.  Rows at the edges of the caches (64 entries without dropping, 256 with ILUT's), levels
of one row and of more rows than a cluster has groups, and a batch of both kinds of member.  A wait
that runs out in the sweep of such a system leaves the context usable."""
import numpy as np
import pytest

from vshe import gpu

pytestmark = pytest.mark.gpu


def _csr(n, offsets, seed=3):
    rng = np.random.default_rng(seed)
    cols = np.arange(n)[:, None] + np.array(sorted(set(offsets) | {0}))[None, :]
    keep = (cols >= 0) & (cols < n)
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(keep.sum(1))
    ci = cols[keep].astype(np.int32)
    row = np.repeat(np.arange(n), keep.sum(1))
    v = rng.uniform(-1.0, 1.0, len(ci))
    v[ci == row] = 0.7 * len(set(offsets)) + 1.0
    return rp, ci, v, rng.uniform(-1.0, 1.0, n)


def _factor(ctx, A, trsv, **kw):
    S = ctx.system(*A, trsv=trsv, ordering="natural", precision="fp64", **kw)
    try:
        return S.factor_values()
    finally:
        S.free()


@pytest.mark.parametrize("kw", [dict(precond="ilu0"), dict(precond="ilu0", fill_level=1),
                                dict(precond="ilut", ilut_entries=7, ilut_drop=1e-3), dict(precond="ilut", ilut_entries=40, ilut_drop=1e-8)])
@pytest.mark.parametrize("n, offsets", [(1, []), (65, [-1, 1]), (1500, [-1, 1, -40, 40]), (1200, list(range(-31, 32))), (1200, list(range(-32, 33))),
                                        (700, list(range(-127, 128))), (700, list(range(-128, 129))), (4000, [-900, -1, 900])])
def test_cluster_factor_equals_grid_factor(gpu_ctx, kw, n, offsets):
    A = _csr(n, offsets)
    assert np.array_equal(_factor(gpu_ctx, A, "per_system", **kw), _factor(gpu_ctx, A, "persistent", **kw))


def test_batch_of_both_kinds(gpu_ctx):
    mats = [_csr(3000, [-1, 1, -40, 40], seed=k) for k in range(3)]
    modes = ["per_system", "persistent", "per_system"]
    alone = []
    for A, m in zip(mats, modes):
        S = gpu_ctx.system(*A, trsv=m, precond="ilu0", ordering="natural", tol=1e-11)
        alone.append(S.solve()[0])
        S.free()
    S = [gpu_ctx.system(*A, trsv=m, precond="ilu0", ordering="natural", tol=1e-11) for A, m in zip(mats, modes)]
    try:
        st = gpu_ctx.batch_solve(S)
        assert all(s["status"] == 0 for s in st)
        for k in range(3):
            assert np.array_equal(S[k].x(), alone[k])
    finally:
        for s in S:
            s.free()


@pytest.mark.parametrize("precond, trsv", [("ilu0", "per_system"), ("block_ilu0", "per_block")])
def test_context_survives_a_sweep_wait_that_runs_out(precond, trsv):
    A = _csr(20000, [-1, 1, -100, 100])
    kw = dict(precond=precond, trsv=trsv, ordering="natural", tol=1e-11, max_iters=200)
    if precond == "block_ilu0":
        kw["blocks"] = np.arange(0, 20001, 4000)
    ctx = gpu.Context(0)
    try:
        ctx.set_spin_limit(1)
        with pytest.raises(gpu.VsheError) as e:
            ctx.solve_csr(*A, **kw)
        assert e.value.code == -10
        ctx.set_spin_limit(0)
        x, st = ctx.solve_csr(*A, **kw)
        assert st["status"] == 0
    finally:
        ctx.close()
    rows = np.repeat(np.arange(20000), np.diff(A[0]))
    r = A[3] - np.bincount(rows, A[2] * x[A[1]], 20000)
    assert np.linalg.norm(r) <= 2e-11 * np.linalg.norm(A[3])
