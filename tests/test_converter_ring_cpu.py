"""CPU: how deep the packed-weight ring of the int4 / MXFP4 converters has to be.

A converter set takes every `sets`-th block of the ring and waits for a stage's fill by parity, so it takes
an unfinished fill for a finished one if the fill before that may still be on its way.  The protocol is
searched in full for the depth from which that cannot happen, and the kernels must refuse to compile below it."""
import os
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
