"""Block-scaled fp8 GEMM around the lines between its token tiles (16 up to 6 rows per expert, 64 up to 11 where K
is 2048 or more, else 128): segments that fill, split and miss a tile, empty experts, both weight layouts."""
import pytest
import torch

from gpu_utils import DEV, grouped_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("K", [1920, 2048, 2176])
@pytest.mark.parametrize("rows", [[6] * 8, [7] * 8, [11] * 8, [12] * 8, [64, 0, 0, 1, 0, 0, 0, 0], [65, 1, 0, 0, 3, 0, 0, 16, 0, 0],
                                  [1, 0, 0, 0, 0, 0, 0, 0, 0, 129, 0, 0, 0, 63], [7]])
def test_fp8_tile_lines(native, layout, K, rows):
    E, M, N = len(rows), sum(rows), 384
    g = torch.Generator().manual_seed(K + M)
    w = torch.randint(0, 256, (E, N, K), generator=g, dtype=torch.int32).to(torch.uint8)
    w[(w & 0x7f) == 0x7f] = 0x38
    a = (torch.randn(M, K, generator=g) * 40).to(torch.float8_e4m3fn)
    sa, sw = torch.rand(M, K // 128, generator=g), torch.rand(E, N // 128, K // 128, generator=g)
    af = a.float() * sa.repeat_interleave(128, 1)
    wf = w.view(torch.float8_e4m3fn).float() * sw.repeat_interleave(128, 1).repeat_interleave(128, 2)
    ref = torch.cat([x @ wf[e].T for e, x in enumerate(af.split(rows))])
    wd = w if layout == 1 else w.transpose(1, 2).contiguous()
    out = grouped_gemm(a.to(DEV), sa.to(DEV), wd.view(torch.float8_e4m3fn).to(DEV), sw.to(DEV), None,
                       torch.tensor(rows, dtype=torch.int32, device=DEV), N, K, layout=layout)
    assert not out.isnan().any()
    # bfloat16 results: relative rounding at most 2^-9, 2^-9 / sqrt(3) of the norm
    assert (out.cpu().float() - ref).norm() / ref.norm() < 2 ** -9
