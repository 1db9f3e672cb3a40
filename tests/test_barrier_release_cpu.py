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


@pytest.mark.parametrize("name,kernel,seen", [("gemm_tc_fp8t.cu", "grouped_gemm_fp8t256_kernel", "sf_full0"),
                                              ("gemm_tc_i4.cu", "grouped_gemm_i4_kernel", "sf_full0")])
def test_promotion_warps_acquire_what_they_read_from_shared_memory(name, kernel, seen):
    """Scales and sums are written with ordinary stores by warps that only the issuer waits for.  A
    tcgen05.commit orders the tensor core's work, not those stores: the issuer has to arrive on the
    accumulator's barrier itself, after its own wait for them and before (or beside) the commit."""
    text = (PKG_DIR / "csrc" / name).read_text()
    code = "\n".join(c for c in (line.split("//")[0].rstrip() for line in text[text.index(kernel):].splitlines()) if c.strip())
    assert re.search(r"mbar_init\(&ctrl->acc_full\[a\], 2\);", code)
    issuer = code[code.index("umma_commit(acc_full0"):]           # behind: the promotion warps take the accumulator alone
    assert seen not in issuer[issuer.index("setmaxnreg_inc"):]
    before = code[:code.index("umma_commit(acc_full0")]
    wait = before.rindex("mbar_wait_s(" + seen)
    free = before.rindex("mbar_wait_s(acc_empty0")                # (not before the phase before is over)
    assert before.rfind("mbar_arrive_s(acc_full0") > max(wait, free)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_a_proxy_fence_lies_between_ordinary_stores_and_the_tensor_core(path):
    """Scale words and partial weight blocks are stored by warps and read by tcgen05.cp / tcgen05.mma, and finished
    rows by TMA, through the async proxy.  Either the writer fences before it arrives, or the issuer does between its
    wait for them and its first use."""
    text = "\n".join(code for _, code in _statements(path))
    fences = text.count("ptx::fence_proxy_async();")
    uses = {"gemm_tc_i4.cu": 1, "gemm_tc_mx.cu": 2, "gemm_tc_fp8t.cu": 1}.get(path.name, 0)
    assert fences == uses
    if path.name == "gemm_tc_i4.cu":      # the preparer, before it hands a group over
        assert "ptx::fence_proxy_async();\n__syncwarp();\nif (lane == 0) ptx::mbar_arrive_s(sf_full0" in text
    if path.name == "gemm_tc_mx.cu":      # the partial block's writers; the issuer, for the scale words
        assert "ptx::fence_proxy_async();\n__syncwarp();\nif (lane == 0) ptx::mbar_arrive(&ctrl->tail_full);" in text
        assert re.search(r"mbar_wait_s\(sf_full0 [^\n]*\n *ptx::fence_proxy_async\(\);", text)
    if path.name == "gemm_tc_fp8t.cu":    # finished rows, before their TMA store
        assert re.search(r"ptx::fence_proxy_async\(\);\n__syncwarp\(\);\nif \(lane == 0\) \{\nptx::tma_store_2d", text)
