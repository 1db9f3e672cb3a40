"""CPU: a kernel that is launched while its predecessor still runs must not read what that one writes through the
non-coherent path (__ldg: read-only for the kernel's whole life, free to move ahead of the wait).  Read from the
sources."""
import re

from conftest import PKG_DIR

SOURCES = sorted(p for p in (PKG_DIR / "csrc").glob("*.cu*") if "pdl_wait()" in p.read_text())


def _code(path):
    return "\n".join(line.split("//")[0] for line in path.read_text().splitlines())


def test_only_weights_are_read_through_the_non_coherent_path():
    """Token scales and sums, rows and their positions come from the kernel ahead."""
    weights = {"gemm_tc_mx.cu": ["src", "src + 1"], "gemm_tc_fp8t.cu": ["w0 + kb", "w0 + w1 + kb"],
               "gemm_tc_i4.cu": ["reinterpret_cast<const uint2*>(srow + kb0)", "srow + g"],
               "gemm_tc_dq.cu": ["s16 + ((kb * 128) >> p.group_shift)", "s16 + g", "srow + kb * 4 + u"]}
    for path in SOURCES:
        found = re.findall(r"__ldg\(((?:[^()]|\((?:[^()]|\([^()]*\))*\))*)\)", _code(path))
        assert found == weights.get(path.name, []), path.name


def test_row_counts_are_read_with_plain_loads():
    """Counts come from the sort ahead: no __ldg, and no __restrict__, by which a compiler may make one."""
    for path in SOURCES:
        code = _code(path)
        assert not re.search(r"__ldg\([^)]*rows_per_(segment|expert)", code), path.name
        assert not re.search(r"const int32_t\* __restrict__ rows_per_(segment|expert)", code), path.name
