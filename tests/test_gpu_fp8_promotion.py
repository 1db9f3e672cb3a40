"""Token-major fp8 GEMM (12 and more rows per expert): scale groups of four K blocks and their
remainders, several tiles per CTA (tile and scale rings go round), feature tiles of one and a half
blocks, empty experts, both weight layouts, and an expert count whose tile walk costs a pipeline stage."""
import pytest
import torch

from gpu_utils import DEV, grouped_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("N,K,rows", [(256, 128, [256, 256]), (384, 256, [1, 128, 129]), (512, 640, [300, 0, 257, 13]),
                                      (1024, 1152, [700, 5, 255, 511, 64]), (2048, 384, [260] * 24),
                                      (256, 128, [12 + i % 3 for i in range(900)])])
def test_fp8_scale_groups(native, layout, N, K, rows):
    E, M = len(rows), sum(rows)
    g = torch.Generator().manual_seed(N + K)
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
    assert (out.cpu().float() - ref).norm() / ref.norm() < 3e-3
