"""The sweeps that keep solved values in shared memory (k_trsv_stream for whole systems, k_trsv_local
for block tasks) against k_trsv_task on the same systems: the same x, bit for bit, and the same
iterations.  Sizes where their tables can go wrong: one row, a partial slice, one row per level, slices of
every stored width and wider, entries far older than the ring, blocks of one row and of one slice,
tasks of several blocks, and blocks just below and above what fits shared memory."""
import numpy as np
import pytest

from vshe import gpu

pytestmark = pytest.mark.gpu


def _csr(n, offsets, seed=3):
    """Rows with the given column offsets (those in range), diagonally dominant, random values."""
    rng = np.random.default_rng(seed)
    cols = np.arange(n)[:, None] + np.array(sorted(set(offsets) | {0}))[None, :]
    keep = (cols >= 0) & (cols < n)
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(keep.sum(1))
    ci = cols[keep].astype(np.int32)
    row = np.repeat(np.arange(n), keep.sum(1))
    v = rng.uniform(-1.0, 1.0, len(ci))
    v[ci == row] = 1.2 * len(set(offsets)) + 1.0
    return rp, ci, v, rng.uniform(-1.0, 1.0, n)


def _both(A, precision, **kw):
    out = []
    # one context: the reduction tiles are tuned once per size class, and x depends on them
    ctx = gpu.Context(0)
    try:
        for kernel in (-1, 0):
            ctx.set_task_sweep(kernel)
            try:
                x, st = ctx.solve_csr(*A, precision=precision, tol=1e-11, max_iters=300, **kw)
                out.append((x, st["iterations"], st["sweep_mode"]))
            except gpu.VsheError as e:
                # Jacobi blocks can break the recurrence down; both kernels then have to
                out.append((np.zeros(1), e.code, 5))
                assert e.code == -5
    finally:
        ctx.close()
    assert out[0][2] == out[1][2] and out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0])
    return out[0][2]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n, offsets", [
    (1, []), (2, [-1, 1]), (31, [-1, 1]), (33, [-1, 1]), (500, [-1, 1]),            # one row per level
    (3000, [-40, 40]), (3001, [-37, -36, 36, 37]), (2000, [-50, -49, -48, 50, 51, 52]),  # widths 1, 2, 3
    (2000, list(range(-44, -40)) + [41]), (2000, list(range(-45, -40)) + [41]), (2000, list(range(-46, -40)) + [41]),
    (2000, list(range(-48, -40)) + [41]), (2500, list(range(-61, -40)) + [41, 42]),  # widths 4, 5, 6, 8, 21
    (30000, [-100, -20000, 100]), (30000, [-100, 100, 11000]), (17000, [-300, -8191, -8192, -8193, -8500, 300]),  # older than the ring
    (6000, [-700, 700]),                                                             # 22 slices a level
])
def test_stream_equals_task(precision, n, offsets):
    assert _both(_csr(n, offsets), precision, precond="ilu0", ordering="natural", trsv="per_system") == 3


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("sizes, offsets", [
    ([1] * 40, [-1, 1]), ([32] * 40, [-1, 1]), ([33, 1, 7, 64, 500] * 9, [-3, -1, 1, 3]),
    ([3000] * 170, [-60, -1, 1, 60]),                                   # more blocks than tasks
    ([16384, 16385, 200, 16000], [-128, -1, 1, 128]),                   # long levels: k_trsv_task
    # below and above what fits shared memory
    *[(sizes, [-700, -251, -250, -126, -125, -3, -2, -1, 1, 2, 3, 125, 126, 250, 251, 700]) for sizes in ([12200, 9000], [12400, 9000], [18700, 16000], [18900, 16000])],
])
def test_local_equals_task(precision, sizes, offsets):
    blocks = np.concatenate([[0], np.cumsum(sizes)])
    A = _csr(int(blocks[-1]), offsets)
    assert _both(A, precision, precond="block_ilu0", ordering="multicolor", fill_level=1, blocks=blocks, trsv="per_block") == 5


def test_ilut_stream_equals_task():
    A = _csr(4000, [-60, -59, -1, 1, 58, 61])
    assert _both(A, "mixed", precond="ilut", ordering="natural", ilut_entries=60, ilut_drop=1e-9, trsv="per_system") == 3
