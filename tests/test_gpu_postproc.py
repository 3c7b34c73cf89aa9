"""Carrier densities and terminal currents of the device pass (k_density: one warp per cell;
k_terminal_currents: one block per contact) against the oracle's sums over the same solution, at
energy counts around the 32 terms a warp sums at once and contacts of one facet, of fewer and of
more facets than a block has warps."""
import numpy as np
import pytest

from vshe import devices as D
from vshe import gpu
import oracle_api as O
import cases

pytestmark = pytest.mark.gpu


def _case(name):
    if name.startswith("diode"):  # one facet per contact
        return cases.diode_small(L=1, boxes=20, bias=0.2, n_energy_range=float(name[5:]))
    ny, ne = (int(v) for v in name.split("x"))
    return cases.bar_small(L=1, nx=6, ny=ny, n_energies=ne)


@pytest.mark.parametrize("name", ["diode0.1", "diode0.5", "2x33", "5x34", "5x35", "33x36", "64x40"])
def test_densities_and_currents_match_oracle(gpu_ctx, name):
    dev, cfg = _case(name)
    P = cases.oracle_problem(dev, cfg)
    S = gpu.SheProblem(gpu_ctx, dev, cfg, coupling=O.golden_coupling(cfg.max_expansion_order), precision="fp64", precond="ilu0", tol=1e-10,
                       max_iters=4000)
    try:
        S.run()
        x, dens, cur = S.results()
        s, sf = S.scaling()
    finally:
        S.free()
    # the reduced solution the device finished from, to rounding
    _, dens_r, cur_r, _ = P.finish(x[:len(s)] / (s * sf))
    # rounding of the division above and of sums of up to 40 energies and 64 facets: a few 1e-15 of
    # the largest term; a net current is a cancellation of one-way fluxes
    assert np.max(np.abs(dens - dens_r)) <= 1e-13 * np.max(np.abs(dens_r))
    assert len(cur) == len(cur_r)
    assert np.max(np.abs(cur - cur_r)) <= 1e-11 * cases.current_scale(dens_r, cur_r)


def test_large_result_arrives_whole():
    """x_full of 74 MB, downloaded in parts by several threads: the residual of the full system, from
    the exported matrix, is the one the device reports (both FP64 sums over the rows; a part that
    is missing or misplaced changes it by orders of magnitude)."""
    dev, cfg = D.config2(100, 25, 240, 3)
    ctx = gpu.Context(0)
    try:
        G = gpu.SheProblem(ctx, dev, cfg, precond="block_ilu0", ordering="multicolor", fill_level=0, tol=1e-4)
        full_residual = G.run()[1]
        rp, ci, val, rhs = G.export("full")
        for _ in range(2):  # allocates the staging buffers, then uses them again
            x = G.results()[0]
            assert x.nbytes > 64 << 20
            r = np.linalg.norm(np.add.reduceat(val * x[ci], rp[:-1]) - rhs) / np.linalg.norm(rhs)
            assert r == pytest.approx(full_residual, rel=1e-6)
    finally:
        ctx.close()
