"""vshe_csr_residual_noalloc where its tiles can go wrong: row counts around a tile of 256 rows and
around one tile for every resident block, rows longer than a staged chunk, tiles averaging more
than 32 entries a row (summed by warps), empty rows and empty matrices, and column and value
arrays aligned to their elements only.  Reference: numpy in extended precision; each row's sum may
differ by its rounding bound, (entries + 2) eps (|b| + sum |a||x|)."""
import ctypes as C

import numpy as np
import pytest

from vshe import gpu

pytestmark = pytest.mark.gpu


def _lengths(kind, n, rng):
    if kind == "short":
        return rng.integers(0, 13, n)
    if kind == "empty":
        return np.zeros(n, np.int64)
    if kind == "wide":
        return rng.integers(30, 90, n)
    k = rng.integers(5, 12, n)  # "dense": a few rows longer than a chunk among short ones
    k[n // 3] = 9000
    k[n - 1] = 3073
    return k


@pytest.mark.parametrize("kind", ["short", "empty", "wide", "dense"])
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1000, 189440, 189441 + 256])
def test_residual_edges(gpu_ctx, kind, n):
    import torch
    if n == 1 and kind == "dense":
        kind = "wide"
    rng = np.random.default_rng(n)
    k = _lengths(kind, n, rng)
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(k)
    nnz = int(rp[-1])
    ci = rng.integers(0, n, nnz).astype(np.int32)
    v = rng.standard_normal(nnz)
    x, b = rng.standard_normal(n), rng.standard_normal(n)
    prod = v.astype(np.longdouble) * x[ci]
    cs = np.concatenate([[0], np.cumsum(prod)])
    ref = b - (cs[rp[1:]] - cs[rp[:-1]])
    mag = np.concatenate([[0], np.cumsum(np.abs(prod))])
    # the running sums of the reference carry 1e-19 of the whole sum, far below the bound
    bound = (k + 2) * np.finfo(float).eps * (np.abs(b) + (mag[rp[1:]] - mag[rp[:-1]])) + 1e-17 * mag[-1]
    cuda = torch.device("cuda", 0)
    d_rp = torch.from_numpy(rp).to(cuda)
    # one element past a 256-byte aligned allocation: aligned to the element only
    d_ci = torch.from_numpy(np.concatenate([[0], ci]).astype(np.int32)).to(cuda)[1:]
    d_v = torch.from_numpy(np.concatenate([[0.0], v])).to(cuda)[1:]
    d_x, d_b = torch.from_numpy(x).to(cuda), torch.from_numpy(b).to(cuda)
    L = gpu.lib()
    L.vshe_csr_residual_noalloc.argtypes = [C.c_int64, C.c_int64] + [C.c_void_p] * 8
    for call in range(2):
        d_r = torch.full((n,), float("nan"), dtype=torch.float64, device=cuda)
        d_n2 = torch.full((2,), float("nan"), dtype=torch.float64, device=cuda)
        torch.cuda.synchronize()
        rc = L.vshe_csr_residual_noalloc(n, nnz, d_rp.data_ptr(), d_ci.data_ptr(), d_v.data_ptr(), d_x.data_ptr(), d_b.data_ptr(),
                                         d_r.data_ptr(), d_n2.data_ptr(), None)
        assert rc == 0, L.vshe_errstr(rc)
        torch.cuda.synchronize()
        r = d_r.cpu().numpy()
        assert np.all(np.abs(r - ref) <= bound), (call, float(np.max(np.abs(r - ref) - bound)))
        n2 = np.array([np.sum(r.astype(np.longdouble) ** 2), np.sum(b.astype(np.longdouble) ** 2)], np.float64)
        assert np.all(np.abs(d_n2.cpu().numpy() - n2) <= 1e-12 * n2)
