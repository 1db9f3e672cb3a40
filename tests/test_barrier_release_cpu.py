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
