"""CPU: hand-overs between the warps of the grouped GEMMs, read from the sources (a missing one is a race
that no run shows reliably)."""
import re

import pytest

from conftest import PKG_DIR

SOURCES = sorted((PKG_DIR / "csrc").glob("gemm_tc*.cu"))


def _statements(path):
    """(line number, code without comments) of the non-empty lines."""
    for i, line in enumerate(path.read_text().splitlines(), 1):
        code = line.split("//")[0].strip()
        if code:
            yield i, code


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_lane_0_arrives_for_its_warp_after_a_warp_barrier(path):
    """An arrival by lane 0 alone says that all lanes have read (or written) what the barrier guards:
    only a __syncwarp directly before it orders their accesses."""
    before, arrivals = "", 0
    for i, code in _statements(path):
        if re.search(r"mbar_arrive\w*\(.*", code) and "lane == 0" in code:
            arrivals += 1
            assert before == "__syncwarp();", f"{path.name}:{i}: {code}"
        before = code
    assert arrivals > 0


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_tensor_memory_waits_name_the_registers_they_wait_for(path):
    """A tcgen05.ld fills its registers after the statement; only a wait that takes them as operands keeps
    the compiler from using them earlier.  (A wait without any is for leaving: nothing is used.)"""
    loads = [code for _, code in _statements(path) if "tmem_ld_32x" in code]
    waits = [code for _, code in _statements(path) if re.search(r"tmem_wait_ld\w*\(", code)]
    assert loads and waits
    assert not [w for w in waits if "tmem_wait_ld()" in w and "break;" not in w]
