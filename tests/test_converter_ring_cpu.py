"""CPU: how deep the packed-weight ring of the int4 / MXFP4 converters has to be.

A converter set takes every `sets`-th block of the ring and waits for a stage's fill by parity, so it takes
an unfinished fill for a finished one if the fill before that may still be on its way.  The protocol is
searched in full for the depth from which that cannot happen, and the kernels must refuse to compile below it.
The first search is the protocol of gemm_tc_dq.cu (one issuer, which frees operands in order).  gemm_tc_i4.cu has two
issuers, and there a hand-over stands for all that it implies: the second search is its ring, operands and
accumulators, the third its groups of token scales and sums.  Both are wider than the kernel (each leaves out the
waits of the other), so what they do not reach the kernel does not reach."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import PKG_DIR

CSRC = PKG_DIR / "csrc"


def _reads_a_block_that_has_not_landed(stages, sets, operands):
    """Every interleaving of: loads issued in order into free stages and landing in any order; converter set
    k reading block k, k + sets, .. and storing it to operand stage block % operands; the MMA taking blocks in
    order.  True if some set gets past its wait for a block that is not there."""
    blocks = 2 * stages + sets
    # state: loads issued, mask of landed blocks, per set (its block, 1 = read but not stored), blocks multiplied
    start = (0, 0, tuple((k, 0) for k in range(sets)), 0)
    seen, todo = {start}, [start]
    while todo:
        issued, landed, conv, done = todo.pop()
        stored = lambda j: any(j % sets == k and (b > j) for k, (b, _) in enumerate(conv))
        read = lambda j: any(j % sets == k and (b > j or (b == j and r)) for k, (b, r) in enumerate(conv))
        after = []
        if issued < blocks and (issued < stages or (read(issued - stages) and done > issued - stages)):
            after.append((issued + 1, landed, conv, done))
        for j in range(issued):
            if not landed >> j & 1:
                after.append((issued, landed | 1 << j, conv, done))
        for k, (b, r) in enumerate(conv):
            if b >= blocks:
                continue
            step = lambda new: (issued, landed, conv[:k] + (new,) + conv[k + 1:], done)
            if not r:
                fills = sum(landed >> j & 1 for j in range(b % stages, blocks, stages))
                if (fills - b // stages) % 2:          # the wait for fill number b // stages by parity
                    if not landed >> b & 1:
                        return True
                    after.append(step((b, 1)))
            elif b < operands or done > b - operands:
                after.append(step((b + sets, 0)))
        if done < blocks and landed >> done & 1 and stored(done):
            after.append((issued, landed, conv, done + 1))
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


@pytest.mark.parametrize("sets,operands", [(2, 2), (2, 4), (3, 3), (3, 4)])
def test_ring_depth_that_parity_waits_need(sets, operands):
    need = sets + operands
    assert not any(_reads_a_block_that_has_not_landed(n, sets, operands) for n in (need, need + 1))
    # one less fails, but for multiples of `sets`: there a stage is always read by the same set
    assert _reads_a_block_that_has_not_landed(need - 1, sets, operands) == ((need - 1) % sets != 0)


def _search(start, steps):
    """Every state that `steps(state)` (new states, or a text: what went wrong) leads to; the first fault, or None."""
    seen, todo = {start}, [start]
    while todo:
        for s in steps(todo.pop()):
            if isinstance(s, str):
                return s
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def _passes(completed, wanted):
    """A wait by parity for completion number `wanted` (0: the barrier's start) of a barrier that has seen `completed`."""
    return (completed - wanted) % 2 == 0


def _int4_ring(stages, sets, slots, issuers, released_by=None):
    """Blocks through ring, operand slots and accumulators.  A stage is free for the next load when the set that reads
    it has read it and when the block `released_by` (slots) further on has been stored.  A load lands at the latest
    when its block is read; it may be late if the stage's last reader was another set.  MMAs of an issuer complete in
    order, those of two issuers in any."""
    ahead = slots if released_by is None else released_by
    blocks = 2 * max(stages, slots) + sets

    def upto(n, first, step, b):       # of the blocks < n with block % step == first: how many share b's slot
        return sum(1 for j in range(first, n, step) if j % slots == b % slots)

    def steps(state):
        issued, conv, mma, done, promo = state     # next load; per set (block, 1 = read); per issuer next and completed; next promoted
        read = lambda j: any(j % sets == k and (b > j or (b == j and r)) for k, (b, r) in enumerate(conv))
        stored = lambda j: conv[j % sets][0] > j
        complete = lambda j: done[j % issuers] > j
        full = lambda b: sum(complete(j) for j in range(b % slots, blocks, slots))       # acc_full of b's slot
        out, waits = [], 0
        if issued < blocks:
            old = issued - stages
            if old < 0 or (read(old) and stored(old + ahead)):
                if old >= 0 and not complete(old):
                    return ["a load overwrites tokens that an MMA reads"]
                out.append((issued + 1, conv, mma, done, promo))
            waits += 1
        for k, (b, r) in enumerate(conv):
            if b >= blocks:
                continue
            waits += 1
            put = lambda new: (issued, conv[:k] + (new,) + conv[k + 1:], mma, done, promo)
            if not r:
                if b >= stages and not read(b - stages):
                    return ["a set takes the fill before for its own"]
                if b < issued:
                    out.append(put((b, 1)))
            elif _passes(full(b), b // slots):
                if b >= slots and not complete(b - slots):
                    return ["a set overwrites an operand in use"]
                out.append(put((b + sets, 0)))
        for i, b in enumerate(mma):
            if b < blocks:
                waits += 1
                have = sum(stored(j) for j in range(b % slots, blocks, slots))
                drained = sum(1 for j in range(b % slots, promo, slots))
                if _passes(have, b // slots + 1) and _passes(drained, b // slots):
                    if not stored(b) or not (b < slots or promo > b - slots):
                        return ["an MMA without its operand, or on an accumulator in use"]
                    out.append((issued, conv, mma[:i] + (b + issuers,) + mma[i + 1:], done, promo))
            if done[i] < mma[i]:
                out.append((issued, conv, mma, done[:i] + (done[i] + issuers,) + done[i + 1:], promo))
        if promo < blocks:
            waits += 1
            if _passes(full(promo), promo // slots + 1):
                if not complete(promo):
                    return ["an accumulator is read before its MMAs are complete"]
                out.append((issued, conv, mma, done, promo + 1))
        return out if out or not waits else ["nobody can go on"]

    return _search((0, tuple((k, 0) for k in range(sets)), tuple(range(issuers)), tuple(range(issuers)), 0), steps)


def _int4_scales(num_kb, slots=6, issuers=2, group=4, ring=3, waits_for=None):
    """Groups of `group` blocks' scales and sums (the last one of a tile may be shorter) through a ring of `ring` slots.  An
    issuer waits for a group with the first `waits_for` (issuers) blocks of it only."""
    waits_for = issuers if waits_for is None else waits_for
    of, pos = [], []                    # group of a block, place in it
    while len(of) < 4 * ring * group or len(of) % num_kb:
        kb = len(of) % num_kb
        pos.append(kb % group)
        of.append(0 if not of else of[-1] + (kb % group == 0))
    blocks, groups = len(of), of[-1] + 1
    last = {g: b for b, g in enumerate(of)}

    def steps(state):
        written, mma, done, promo = state
        complete = lambda j: done[j % issuers] > j
        finished = promo and of[promo - 1] + (last[of[promo - 1]] == promo - 1)     # groups handed back
        in_slot = lambda n, g: sum(1 for j in range(g % ring, n, ring))
        out, waits = [], 0
        if written < groups:
            waits += 1
            if _passes(in_slot(finished, written), written // ring):
                old = written - ring
                if old >= 0 and not (finished > old and all(complete(b) for b in range(blocks) if of[b] == old)):
                    return ["scales are overwritten in use"]
                out.append((written + 1, mma, done, promo))
        for i, b in enumerate(mma):
            if b < blocks:
                waits += 1
                g = of[b]
                drained = sum(1 for j in range(b % slots, promo, slots))
                if (pos[b] >= waits_for or _passes(in_slot(written, g), g // ring + 1)) and _passes(drained, b // slots):
                    if written <= g:
                        return ["an MMA without its scales"]
                    out.append((written, mma[:i] + (b + issuers,) + mma[i + 1:], done, promo))
            if done[i] < mma[i]:
                out.append((written, mma, done[:i] + (done[i] + issuers,) + done[i + 1:], promo))
        if promo < blocks:
            waits += 1
            if _passes(sum(complete(j) for j in range(promo % slots, blocks, slots)), promo // slots + 1):
                if not complete(promo) or written <= of[promo]:
                    return ["sums are read that are not there"]
                out.append((written, mma, done, promo + 1))
        return out if out or not waits else ["nobody can go on"]

    return _search((0, tuple(range(issuers)), tuple(range(issuers)), 0), steps)


def _i4_constant(name):
    return int(re.search(rf"constexpr int {name} = (\d+);", (CSRC / "gemm_tc_i4.cu").read_text()).group(1))


@pytest.mark.parametrize("stages", [9, 12])
def test_int4_ring_operands_and_accumulators(stages):
    sets, slots, issuers = (_i4_constant(n) for n in ("kI4Sets", "kI4Conv", "kI4Issuers"))
    assert stages % sets == 0 and stages <= _i4_constant("kI4MaxStages")
    assert _int4_ring(stages, sets, slots, issuers) is None


@pytest.mark.parametrize("what,kw", [("takes the fill before", dict(stages=8, sets=3, slots=6, issuers=2)),
                                     ("nobody can go on", dict(stages=6, sets=3, slots=6, issuers=2)),
                                     ("tokens that an MMA reads", dict(stages=6, sets=3, slots=6, issuers=2, released_by=3))])
def test_the_search_finds_what_the_int4_ring_must_not_be(what, kw):
    assert what in (_int4_ring(**kw) or "")


@pytest.mark.parametrize("num_kb", [1, 2, 3, 4, 5, 6, 7, 8, 9])
def test_int4_groups_of_scales(num_kb):
    kw = dict(slots=_i4_constant("kI4Conv"), issuers=_i4_constant("kI4Issuers"), group=_i4_constant("kI4Group"), ring=_i4_constant("kI4Slots"))
    assert _int4_scales(num_kb, **kw) is None
    if num_kb % kw["group"] not in (1,):     # one issuer that does not wait for a group's scales
        assert _int4_scales(num_kb, **kw, waits_for=1) is not None


@pytest.mark.parametrize("source,planted", [
    ("gemm_tc_i4.cu", ("constexpr int kI4MaxStages = 12;", "constexpr int kI4MaxStages = 6;")),
    ("gemm_tc_dq.cu", ("kDqMaxRaw = 12,", "kDqMaxRaw = 8,")),
])
def test_kernels_with_a_shorter_ring_do_not_compile(tmp_path, source, planted):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    text = (CSRC / source).read_text()
    assert text.count(planted[0]) == 1
    (tmp_path / source).write_text(text.replace(*planted))
    res = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(CSRC), "-ptx",
                          "-o", str(tmp_path / "out.ptx"), str(tmp_path / source)], capture_output=True, text=True)
    assert res.returncode != 0 and "ring depth" in res.stderr, res.stderr[-500:]
