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
* block tasks: a warp's chunks follow each other, and each is copied whole into a slot that its reader
  has left;
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
def _many_blocks(size=310, count=170):
    """More blocks than CTAs: tasks of two blocks."""
    n = size * count
    rp, ci, v, _ = _far(n, 61)
    return rp, ci, v, np.arange(0, n + 1, size)


BLOCKS["tasks_of_two_blocks"] = (_many_blocks, dict(BLK, trsv="per_block"), "mixed", 2)
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


@pytest.mark.parametrize("num_sms", [148, 20])
@pytest.mark.parametrize("name", sorted(BLOCKS))
def test_local_plan_runs_like_the_level_sweep(name, num_sms):
    rp, ci, vals, kw, lay, vt, lval, uval, udinv, x, slot, (y_ref, z_ref) = _make(BLOCKS[name])
    P = gpu.local_plan(rp, ci, vals, num_sms=num_sms, **kw)
    n, ring, nw, slots, sb = lay["n"], P["ring"], P["nwarp"], P["slots"], P["slot_bytes"]
    vb = np.dtype(vt).itemsize
    assert 1 <= nw <= 15 and slots == 3 and ring % 16 == 0 and ring < 1 << 16 and sb % 16 == 0
    assert 8 * ring + 128 + nw * slots * sb + 1024 <= SMEM
    assert len(P["tasks"]) and P["rest"] == 0 and len(P["warps"]) == nw * len(P["tasks"])
    # the chunks and records as k_local_fill writes them, by offset; they follow each other without a gap
    recs, chunks, end, left, cols = {}, {}, 0, 0, 8
    seen = {True: np.zeros(len(lay["lcol"]) // 32, int), False: np.zeros(len(lay["ucol"]) // 32, int)}
    rows = {True: np.zeros(n, int), False: np.zeros(n, int)}
    for off, j, u0, ncol, lower, loc0, lev, groups, nr in P["recs"].tolist():
        assert off == end and off % 16 == 0
        if j < 0:
            assert left == 0 and loc0 > 0
            head, left, end = off, loc0, off + 16
            chunks[head] = [16, lev, []]
            continue
        lower, back, nr = bool(lower), nr >= 64, nr % 64
        size = 16 + 128 * groups * (2 + vb) + (32 * (2 + vb) if back else 0)
        end, left = off + size, left - 1
        chunks[head][0] += size
        chunks[head][2].append(off)
        assert size % 16 == 0 and chunks[head][0] <= sb
        so, col, val, r0 = (lay["loff"], lay["lcol"], lval, lay["lrow0"]) if lower else (lay["uoff"], lay["ucol"], uval, lay["uslot0"])
        w = int(so[j + 1] - so[j]) // 32
        last = u0 + ncol == w
        assert 0 <= ncol <= cols and u0 % cols == 0 and (nr > 0) == last and (last or ncol == cols)
        assert back == (last and not lower) and 4 * groups - ncol in (0, 1, 2, 3)
        a, b = so[j] + 32 * u0, so[j] + 32 * (u0 + ncol)
        seen[lower][a // 32:b // 32] += 1
        q = np.arange(r0[j], r0[j + 1])
        if last:
            assert nr == len(q)
            rows[lower][q] += 1
        c = col[a:b].reshape(ncol, 32).astype(np.int64)
        num = np.where(c < n, P["num"][np.minimum(c, n - 1)], ring)
        assert np.all(num[c < n] < ring)
        loc = P["num"][q if lower else lay["urow"][q]]
        assert not lower or np.array_equal(loc, loc0 + np.arange(len(q)))
        recs[off] = (loc, nr, lev, lower, q, num, val[a:b].reshape(ncol, 32), np.where(c < n, c, -1))
    assert end == P["bytes"] and left == 0
    assert all(np.all(k == 1) for k in seen.values()) and all(np.all(k == 1) for k in rows.values())
    out = np.full(n, np.nan)
    for sys, nlevF, nlev, m, w0, run0 in P["tasks"].tolist():
        assert 0 < m <= ring and 0 < nlevF < nlev
        W = P["warps"][w0:w0 + nw].tolist()
        # entry i: value, row, forward result (1) or backward (2)
        win, who, kind = np.full(ring + 1, np.nan), np.full(ring + 1, -1), np.zeros(ring + 1, int)
        win[ring] = 0.0
        runs = P["runs"][run0:run0 + nlevF]
        for (row, num), stop in zip(runs, np.append(runs[1:, 1], m)):
            who[num:stop] = np.arange(row, row + stop - num)
            win[num:stop] = x[who[num:stop]]
        assert np.all(who[:m] >= 0) and np.array_equal(P["num"][who[:m]], np.arange(m))
        nxt, held, todo, done = [w[0] for w in W], [[None] * slots for _ in W], [[] for _ in W], [0] * nw
        acc = [np.zeros(32) for _ in W]

        def issue(k, to, size):
            assert held[k][to] is None and size == chunks[nxt[k]][0], "a whole chunk into a free slot"
            held[k][to] = nxt[k]
            nxt[k] += size

        for k, w in enumerate(W):
            for i in range(min(slots - 1, w[1])):
                issue(k, i, w[2 + i])
        # between two barriers the warps run in any order: what they write is not read by others before the
        # next; the results are read after the last
        for passed in range(nlev):
            if passed == nlevF:
                assert np.all(kind[:m] == 1), "the forward sweep ends before this barrier"
            writes = []
            for k in range(nw):
                while True:
                    if not todo[k]:
                        # the chunk before this one is read to its end: its slot is free
                        if done[k]:
                            held[k][(done[k] - 1) % slots] = None
                        if done[k] == W[k][1]:
                            break
                        size, ahead, todo[k] = chunks[held[k][done[k] % slots]]
                        todo[k] = list(todo[k])
                        if ahead:
                            issue(k, (done[k] + slots - 1) % slots, ahead)
                        done[k] += 1
                    loc, nr, lev, lower, q, num, v, named = recs[todo[k][0]]
                    if lev != passed:
                        assert lev > passed
                        break
                    todo[k].pop(0)
                    assert lower == (passed < nlevF)
                    used = named >= 0
                    assert np.array_equal(who[num[used]], named[used]), "the value is the one the row names, of this task"
                    assert np.all(kind[num[used]] == (1 if lower else 2)), "and of an earlier level of this sweep"
                    for u in range(v.shape[0]):
                        acc[k] = acc[k] + v[u] * win[num[u]]
                    if nr == 0:
                        continue
                    assert np.all(kind[loc] == (0 if lower else 1))
                    z = win[loc] - acc[k][:nr] if lower else (win[loc] - acc[k][:nr]) * udinv[q]
                    acc[k] = np.zeros(32)
                    writes += list(zip(loc.tolist(), z, [1 if lower else 2] * nr))
            assert len({p_ for p_, _, _ in writes}) == len(writes)
            for p_, v_, f_ in writes:
                win[p_], kind[p_] = v_, f_
            if passed == nlevF - 1:
                assert np.array_equal(win[:m], y_ref[who[:m]])
        assert done == [w[1] for w in W] and not any(todo) and np.all(kind[:m] == 2)
        out[who[:m]] = win[:m]
    assert np.array_equal(out, z_ref)
