"""k_trsv_local's copies where a warp's first chunk holds a single record (slots of about one record beside
a block of many rows, and a warp without a slice in level 0).  On the CPU: the kernel's order of loads,
work and copies on the plan's records -- a record is loaded before the one ahead of it is worked on, and
one pending copy is issued after the work -- finds every chunk whole in its slot.  On the GPU: the same x
as k_trsv_task, bit for bit."""
import numpy as np
import pytest

from vshe import gpu
import test_gpu_local_sweeps as sweeps

OFFSETS = [-700, -251, -250, -126, -125, -3, -2, -1, 1, 2, 3, 125, 126, 250, 251, 700]
SIZES = [[18700, 2000], [16000, 800], [16000, 16000, 2000]]
BLK = dict(precond="block_ilu0", ordering="multicolor", fill_level=1, trsv="per_block")


def _system(sizes):
    blocks = np.concatenate([[0], np.cumsum(sizes)])
    return sweeps._csr(int(blocks[-1]), OFFSETS), blocks


@pytest.mark.parametrize("sizes", SIZES)
def test_every_chunk_is_copied(sizes):
    (rp, ci, _, _), blocks = _system(sizes)
    P = gpu.local_plan(rp, ci, precision="mixed", blocks=blocks, **BLK)
    slots, chunks = P["slots"], {}
    for off, j, _, _, _, a, b, _, _ in P["recs"].tolist():
        if j < 0:
            chunks[off] = (a, b)  # records, size of the chunk slots - 1 further on
    starts = sorted(chunks) + [P["bytes"]]
    size = dict(zip(starts, np.diff(starts)))
    single = 0
    for off, nchunk, *sizes3 in P["warps"].tolist():
        if nchunk == 0:
            continue
        single += nchunk >= 3 and chunks[off][0] == 1
        slot_of, nxt = {}, off

        def issue(slot, nbytes):
            nonlocal nxt
            assert slot_of.get(slot) is None and nbytes == size[nxt], "a whole chunk into a free slot"
            slot_of[slot], nxt = nxt, nxt + nbytes

        for i in range(min(slots - 1, nchunk)):
            issue(i, sizes3[i])
        # records as (chunk, is its last); `ahead` the pending copy
        chunk, slot, left, ahead, at = -1, -1, 0, 0, off

        def load():
            nonlocal chunk, slot, left, ahead, at
            if left == 0:
                chunk += 1
                if chunk == nchunk:
                    return None
                slot = (slot + 1) % slots
                assert slot_of.get(slot) == at, "the chunk is in the slot its reader waits for"
                left, ahead = chunks[at]
                at += size[at]
            left -= 1
            return slot, left == 0

        def copy_ahead():
            nonlocal ahead
            if ahead:
                to = (slot - 1) % slots
                issue(to, ahead)
                ahead = 0

        held = load()
        copy_ahead()
        while held is not None:
            after = load()
            if held[1]:
                slot_of[held[0]] = None  # its last record is worked on: the slot is free
            copy_ahead()
            held = after
        assert chunk == nchunk and nxt == at
    assert single, "the plan has a first chunk of one record"


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", SIZES)
def test_local_equals_task(sizes):
    A, blocks = _system(sizes)
    assert sweeps._both(A, "mixed", blocks=blocks, **BLK) == 5
