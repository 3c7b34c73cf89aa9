"""The tables of the sweeps that keep solved values in shared memory: k_trsv_local's plan for block
tasks (vshe_layout_local_plan) and k_trsv_stream's for whole systems (vshe_layout_stream_plan), host
only.  What the kernels' copies, rings and barriers rely on is checked by running the plans on the
CPU as the kernels do -- the copies of every chunk into a stage with bounds and alignment checked, the
slices of every warp from the stage alone, the solved values in the ring -- and comparing the result
bit for bit with the level by level sweep of the same SELL slices:
* stage, ring and static shared memory fit one CTA; copies are 16-byte aligned, inside their source
  arrays (8 padding entries past n) and the stage, and do not overlap;
* a value a row reads from the ring is the one it names, of an earlier level, and no row of the
  reader's own level overwrites it; one read from global memory (by streams) is at
  least three steps old;
* block tasks: a warp's slices come in level order, and every chunk's barrier count lets the warps
  still in it reach their levels;
* streams: every warp has a slice (the chunk's empty one where it has none) in every step, and the
  descriptors reach two steps past the end;
* over all tasks every row is solved once forward and once backward."""
import numpy as np
import pytest

from vshe import devices as D
from vshe import gpu
import oracle_api as O

SMEM = 232448 - 1024  # opt-in limit of a CTA less what the system and the kernel hold statically
PAD = 0x7FFFFFFF


def _system(make):
    dev, cfg = make()
    P = O.OracleProblem(dev, cfg, O.golden_coupling(cfg.max_expansion_order))
    A = P.matrix(3)
    return A.rp, A.ci, A.v, P.blocks()


def _poisson():
    dev = D.nin_bar_2d(nx=60, ny=21, bias=0.8)
    M = O.poisson_assemble(dev, D.facet_centres(dev), dev.potential, dev.doping_n, dev.doping_n * 0 + 1)
    return M.rp, M.ci, M.v, None


def _tri(n=70):
    """Tridiagonal: one row per level, a single slice of one row at a time."""
    rp = np.zeros(n + 1, np.int64)
    rows = [[j for j in (i - 1, i, i + 1) if 0 <= j < n] for i in range(n)]
    rp[1:] = np.cumsum([len(r) for r in rows])
    ci = np.concatenate(rows).astype(np.int32)
    v = np.where(ci == np.repeat(np.arange(n), np.diff(rp)), 4.0, -1.0)
    return rp, ci, v, None


def _far(n, far, width=1):
    """Rows that read `width` columns from i - far on, and their neighbours at 100."""
    off = np.array(sorted({-100, 0, 100} | set(range(-far, -far + width))))
    cols = np.arange(n)[:, None] + off[None, :]
    keep = (cols >= 0) & (cols < n)
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(keep.sum(1))
    ci = cols[keep].astype(np.int32)
    return rp, ci, np.where(ci == np.repeat(np.arange(n), keep.sum(1)), 40.0, -1.0), None


BLK = dict(precond="block_ilu0", ordering="multicolor", fill_level=1)
NAT = dict(precond="ilu0", ordering="natural")
BLOCKS = {
    "bar_blocks_mixed": (lambda: _system(lambda: D.config2(40, 10, 48, 3)), BLK, "mixed", 2),
    "bar_blocks_fp64": (lambda: _system(lambda: D.config2(40, 10, 48, 3)), BLK, "fp64", 2),
    "bar_blocks_L1": (lambda: _system(lambda: D.config2(37, 9, 55, 1)), dict(BLK, fill_level=0), "mixed", 2),
}
STREAMS = {
    "diode_mixed": (lambda: _system(D.config1), NAT, "mixed", 1),
    "diode_fp64": (lambda: _system(D.config1), NAT, "fp64", 1),
    "diode_L3": (lambda: _system(lambda: D.config3()[8]), NAT, "mixed", 1),
    "bar_natural": (lambda: _system(lambda: D.config2(50, 20, 60, 1)), NAT, "mixed", 1),
    "ilut": (lambda: _system(lambda: D.config2(8, 4, 36, 5, 0.1)), dict(precond="ilut", ordering="natural", ilut_entries=40, ilut_drop=1e-3), "mixed", 1),
    "poisson": (_poisson, NAT, "fp64", 1),
    "tridiagonal": (_tri, dict(NAT, trsv="per_system"), "mixed", 1),
    "one_row": (lambda: _tri(1), dict(NAT, trsv="per_system"), "fp64", 1),
    "two_rows": (lambda: _tri(2), dict(NAT, trsv="per_system"), "mixed", 1),
    "old_values": (lambda: _far(30000, 20000), dict(NAT, trsv="per_system"), "mixed", 1),
    "wide_rows": (lambda: _far(4000, 61, 21), dict(NAT, trsv="per_system"), "fp64", 1),
}


def _sweep_reference(lay, lval, uval, udinv, x):
    n = lay["n"]
    y, z = np.zeros(n + 1), np.zeros(n + 1)
    for off, col, val, r0, lower in ((lay["loff"], lay["lcol"], lval, lay["lrow0"], True), (lay["uoff"], lay["ucol"], uval, lay["uslot0"], False)):
        src = y if lower else z
        for j in range(len(off) - 1):
            nr, w = int(r0[j + 1] - r0[j]), int(off[j + 1] - off[j]) // 32
            c, a = col[off[j]:off[j + 1]].reshape(w, 32)[:, :nr], val[off[j]:off[j + 1]].reshape(w, 32)[:, :nr]
            s = np.zeros(nr)
            for k in range(w):
                s = s + a[k] * src[c[k]]
            if lower:
                y[r0[j]:r0[j + 1]] = x[r0[j]:r0[j + 1]] - s
            else:
                rows = lay["urow"][r0[j]:r0[j + 1]]
                z[rows] = (y[rows] - s) * udinv[r0[j]:r0[j + 1]]
    return y[:n], z[:n]


def _make(case):
    make, kw, precision, kind = case
    rp, ci, v, blocks = make()
    kw = dict(kw, precision=precision)
    if kw["precond"].startswith("block"):
        kw["blocks"] = blocks
    vals = v if kw["precond"] == "ilut" else None
    lay = gpu.layout(rp, ci, vals, **kw)
    assert gpu.sweep_plan(rp, ci, vals, **kw)["kind"] == kind
    vt = np.float32 if precision == "mixed" else np.float64
    rng = np.random.default_rng(3)
    n = lay["n"]
    fill = lambda m: np.where(m >= 0, rng.uniform(-0.4, 0.4, len(m)), 0.0).astype(vt)
    # factor values at the layout's slots (padding 0), inverse diagonals, an input
    lval, uval = fill(np.where(lay["lcol"] < n, 0, -1)), fill(np.where(lay["ucol"] < n, 0, -1))
    udinv = np.concatenate([rng.uniform(0.5, 2.0, n), np.zeros(8)]).astype(vt)
    x = np.concatenate([rng.standard_normal(n), np.zeros(8)])
    slot = np.zeros(n + 8, np.int32)
    slot[lay["urow"]] = np.arange(n)
    ref = _sweep_reference(lay, lval.astype(float), uval.astype(float), udinv.astype(float), x)
    return rp, ci, vals, kw, lay, vt, lval, uval, udinv, x, slot, ref


@pytest.mark.parametrize("name", sorted(STREAMS))
def test_stream_runs_like_the_level_sweep(name):
    rp, ci, vals, kw, lay, vt, lval, uval, udinv, x, slot, (y_ref, z_ref) = _make(STREAMS[name])
    P = gpu.stream_plan(rp, ci, vals, **kw)
    n, ring, nw = lay["n"], P["ring"], P["nwarp"]
    assert 1 <= nw <= 15 and ring & (ring - 1) == 0
    assert P["smem"] == 8 * ring + 128 + 3 * P["stage"] and P["smem"] + 256 <= SMEM
    assert (8 * ring + 128) % 128 == 0 and P["stage"] % 128 == 0, "copies into the stages are 16-byte aligned"
    eb = 8 if vt == np.float32 else 16
    # the device arrays as k_stream_fill and k_stream_patch write them: entry offset / value, row
    # position / target / diagonal; and the number each entry names (-1: padding)
    nent, nrow = int(P["chunks"][:, 4].sum()) // eb, int(P["chunks"][:, 5].sum()) // 16
    ent_at, ent_v, ent_num = np.full(nent, -1, np.int64), np.zeros(nent), np.full(nent, -1)
    row_pos, row_dst, row_inv, row_num = np.zeros(nrow, np.int64), np.full(nrow, -2), np.ones(nrow), np.full(nrow, -1)
    seen = {True: np.zeros(len(lay["loff"]) - 1, int), False: np.zeros(len(lay["uoff"]) - 1, int)}
    for ent, row, j, width, lower in P["recs"].tolist():
        lower = bool(lower)
        e, k = ent // eb, row // 16
        assert ent % (32 * eb) == 0 and row % 512 == 0
        assert np.all(ent_at[e:e + 32 * width] == -1) and np.all(row_dst[k:k + 32] == -2), "slices of the stream do not overlap"
        ent_at[e:e + 32 * width], row_dst[k:k + 32] = 8 * ring, -1
        if j < 0:  # an empty slice
            continue
        off, col, val, r0 = (lay["loff"], lay["lcol"], lval, lay["lrow0"]) if lower else (lay["uoff"], lay["ucol"], uval, lay["uslot0"])
        w, nr = int(off[j + 1] - off[j]) // 32, int(r0[j + 1] - r0[j])
        assert width >= w
        seen[lower][j] += 1
        c = col[off[j]:off[j + 1]].astype(np.int64)
        num = np.where(c < n, c if lower else slot[np.minimum(c, n - 1)], -1)
        ent_at[e:e + 32 * w] = np.where(num < 0, 8 * ring, 8 * (num & (ring - 1)))
        ent_num[e:e + 32 * w], ent_v[e:e + 32 * w] = num, val[off[j]:off[j + 1]]
        q = np.arange(r0[j], r0[j] + nr)
        row_pos[k:k + nr], row_num[k:k + nr], row_dst[k:k + nr] = 8 * (q & (ring - 1)), q, slot[q] if lower else lay["urow"][q]
        if not lower:
            row_inv[k:k + nr] = udinv[q]
    assert np.all(seen[True] == 1) and np.all(seen[False] == 1)
    assert len(np.unique(P["patch"][:, 0])) == len(P["patch"])
    ent_at[P["patch"][:, 0]] = P["patch"][:, 1]
    yslot, out = np.full(n + 8, np.nan), np.full(n, np.nan)
    # shared memory by 8-byte word: value, number it is of, step it was written in
    words = P["smem"] // 8
    win, tag, tlev = np.full(words, np.nan), np.full(words, -1), np.full(words, -1)
    win[ring] = 0.0
    tag[ring] = -1
    level, writes, head, starts, kept = 0, [], 0, [], {}
    for g, (h, ent, row, hb, ebytes, rb, op0, nop, nstep, old0, nold) in enumerate(P["chunks"].tolist()):
        lower = g < P["nfwd"]
        if g == P["nfwd"]:
            starts, kept = [], {}
            tag[:], tlev[:], win[:ring] = -1, -1, np.nan  # nothing of the forward sweep is read again
        assert nstep % 2 == 0 and h == 16 * head and hb == 16 * nw * (nstep + 2) and ebytes % 16 == 0 and rb % 16 == 0 and nold % 2 == 0
        ops = hb + ebytes + rb + 8 * nold
        assert op0 % 4 == 0 and nop % 4 == 0 and ops + 8 * nop <= P["stage"] and 0 <= op0 and op0 + nop <= n + 8 and 0 < ops + 8 * nop < 1 << 20
        # the producer gathers the older values when every warp is through chunk g - 3
        stage0 = 8 * ring + 128 + (g % 3) * P["stage"]
        finished = starts[-2] if len(starts) >= 2 else 0
        for i in range(nold):
            q = int(P["olds"][old0 + i])
            assert P["keep"][0 if lower else 1] and 0 <= q < finished, "an older value is written before its chunk is fetched"
            at = (stage0 + hb + ebytes + rb) // 8 + i
            win[at], tag[at], tlev[at] = kept[q], q, -1
        st = P["steps"][head:head + nw * (nstep + 2)].reshape(nstep + 2, nw, 4)
        head += nw * (nstep + 2)
        src = x if lower else yslot
        first = n
        for step in range(nstep + 2):
            # the barrier before the step: what earlier steps wrote is visible
            for l_, p_, q_, v_ in writes:
                win[p_], tag[p_], tlev[p_] = v_, q_, l_
                kept[q_] = v_
            writes, level = [], level + (step < nstep)
            for warp, (e, r, op, w) in enumerate(st[step].tolist()):
                want = int(P["widths"][0 if lower else 1][warp])
                assert (w >= want if want <= 8 else w >= 8) and e >= hb and r >= hb + ebytes and op >= ops and op + 256 <= P["stage"]
                assert e + 32 * w * eb <= hb + ebytes and r + 512 <= hb + ebytes + rb
                k0, r0 = (ent + e - hb) // eb, (row + r - hb - ebytes) // 16
                if row_dst[r0] < 0:
                    assert np.all(row_dst[r0:r0 + 32] == -1) and np.all(ent_at[k0:k0 + 32 * w] == 8 * ring)
                    continue
                assert step < nstep and (w == want or want > 8)
                at, v = ent_at[k0:k0 + 32 * w].reshape(w, 32), ent_v[k0:k0 + 32 * w].reshape(w, 32)
                num = ent_num[k0:k0 + 32 * w].reshape(w, 32)
                lanes = row_dst[r0:r0 + 32] >= 0
                nr = int(lanes.sum())
                q = row_num[r0:r0 + nr]
                first = min(first, int(q[0]))
                assert lanes[:nr].all() and op0 + (op - ops) // 8 == q[0]
                s = np.zeros(nr)
                for u in range(w):
                    a = at[u, :nr] // 8
                    assert np.all(tag[a] == num[u, :nr]) and np.all(tlev[a] < level), "the value is the one the row names, of an earlier step"
                    # rows of the reader's own step (and of later ones of its level) do not overwrite it
                    s = s + v[u, :nr] * win[a]
                base = src[q]
                z = base - s if lower else (base - s) * row_inv[r0:r0 + nr]
                (yslot if lower else out)[row_dst[r0:r0 + nr]] = z
                writes += [(level, int(p_) // 8, int(t), float(v_)) for p_, t, v_ in zip(row_pos[r0:r0 + nr], q, z)]
            pos = [p_ for _, p_, _, _ in writes]
            assert len(set(pos)) == len(pos)
            written = set(pos)
            for e, r, op, w in st[step].tolist():
                k0 = (ent + e - hb) // eb
                assert not written.intersection((ent_at[k0:k0 + 32 * w] // 8).tolist()), "no row of a step overwrites what another of it reads"
        starts.append(first)
        if g == P["nfwd"] - 1:
            assert not np.isnan(yslot[:n]).any()
    assert np.array_equal(yslot[slot[:n]], y_ref)
    assert np.array_equal(out, z_ref)


@pytest.mark.parametrize("name", sorted(BLOCKS))
def test_local_plan_runs_like_the_level_sweep(name):
    rp, ci, vals, kw, lay, vt, lval, uval, udinv, x, slot, (y_ref, z_ref) = _make(BLOCKS[name])
    P = gpu.local_plan(rp, ci, vals, **kw)
    n, ring, C = lay["n"], P["ring"], P["consumers"]
    assert len(P["tasks"]) > 0 and P["rest"] == 0
    assert C in (3, 7, 15, 31) and ring & (ring - 1) == 0
    assert 8 * ring + 128 + 3 * P["stage"] + 256 <= SMEM
    assert (8 * ring + 128) % 128 == 0 and P["stage"] % 128 == 0, "copies into the stages are 16-byte aligned"
    fm, bm = np.append(P["fmap"], PAD), np.append(P["bmap"], PAD)
    arrays = {0: P["heads"], 1: fm[lay["lcol"]].astype(np.int32), 2: lval, 3: x, 4: slot, 5: bm[lay["ucol"]].astype(np.int32), 6: uval,
              7: np.full(n + 8, np.nan), 8: np.concatenate([lay["urow"], np.zeros(8, np.int32)]), 9: udinv}
    vb = vt().itemsize
    out = np.full(n, np.nan)
    fwd_seen, bwd_seen = np.zeros(n, int), np.zeros(n, int)
    for sys_, c0, nfwd, nchunk, nlevF, m, tring, _ in P["tasks"].tolist():
        assert tring == ring and m <= ring
        win, tlev = np.full(ring, np.nan), np.full(ring, -1)
        passed = 0
        writes = []  # (level, number, value): applied when their level closes
        for g in range(c0, c0 + nchunk):
            lower = g - c0 < nfwd
            if g - c0 == nfwd:
                win[:], tlev[:] = np.nan, -1  # nothing of the forward sweep is read again
            rec0, nrec, nlate, nbytes, late = P["chunks"][g].tolist()
            stage, used = np.zeros(P["stage"], np.uint8), np.zeros(P["stage"], bool)
            tot = [0, 0]
            for k in range(rec0, rec0 + nrec):
                src, dst, arr, size = P["copies"][k].tolist()
                b = arrays[arr].view(np.uint8)
                assert src % 16 == 0 and dst % 16 == 0 and size % 16 == 0 and size > 0
                assert src + size <= len(b) and dst + size <= P["stage"] and not used[dst:dst + size].any()
                is_late = k >= rec0 + nrec - nlate
                assert is_late == (arr == 7)
                stage[dst:dst + size], used[dst:dst + size] = b[src:src + size], True
                tot[is_late] += size
            assert tot == [nbytes, late]
            i32 = stage.view(np.int32)
            offA, offB, offC, offD, npass = i32[:5].tolist()
            wptr = i32[8:8 + C + 1]
            ns = int(wptr[C])
            desc = i32[offD // 4:offD // 4 + 8 * ns].reshape(ns, 8)
            assert wptr[0] == 0 and np.all(np.diff(wptr) >= 0) and offD + 32 * ns <= offA
            for w in range(C):
                assert np.all(np.diff(desc[wptr[w]:wptr[w + 1], 5]) >= 0), "a warp's slices come in level order"
            lmax = int(desc[:, 5].max())
            assert npass == (nlevF if g - c0 == nfwd - 1 else lmax)
            for d in desc[np.argsort(desc[:, 4], kind="stable")]:
                col, val, op, wnr, loc0, lev = d[:6].tolist()
                width, nr = wnr >> 6, wnr & 63
                if lev > passed:  # the level barrier: what earlier levels wrote is visible
                    for l_, num, value in writes:
                        win[num], tlev[num] = value, l_
                    writes, passed = [], lev
                c = i32[col // 4:col // 4 + 32 * width].reshape(width, 32)[:, :nr]
                a = stage[val:val + 32 * width * vb].view(vt).reshape(width, 32)[:, :nr].astype(float)
                s = np.zeros(nr)
                for k in range(width):
                    q = c[k]
                    near = q < m
                    assert np.all(q[near] < loc0) and np.all(tlev[q[near]] < lev) and np.all(tlev[q[near]] >= 0)
                    xv = np.zeros(nr)
                    xv[near] = win[q[near]]
                    s = s + a[k] * xv
                num = np.arange(loc0, loc0 + nr)
                assert loc0 + nr <= m
                base = stage[offA:].view(np.float64)[op:op + nr]
                dst = stage[offB:].view(np.int32)[op:op + nr]
                assert used[offA + 8 * op:offA + 8 * (op + nr)].all() and used[offB + 4 * op:offB + 4 * (op + nr)].all()
                if lower:
                    r = base - s
                    arrays[7][dst] = r
                    fwd_seen[dst] += 1
                else:
                    r = (base - s) * stage[offC:].view(vt)[op:op + nr].astype(float)
                    out[dst] = r
                    bwd_seen[dst] += 1
                writes += [(lev, t, value) for t, value in zip(num.tolist(), r.tolist())]
            if g - c0 == nfwd - 1:
                writes, passed = [], nlevF
    assert np.all(fwd_seen == 1) and np.all(bwd_seen == 1)
    assert np.array_equal(arrays[7][slot[:n]], y_ref)
    assert np.array_equal(out, z_ref)
