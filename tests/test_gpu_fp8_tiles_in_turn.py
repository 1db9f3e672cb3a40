"""Block-scaled fp8 GEMM with few rows per expert and a short K loop: two sets of epilogue warps take tiles in turn.
K of one block to 31 and, as before, 32; grids from one CTA (all tiles in one stream) to one tile a CTA; both
weight layouts, a bias; the sums are the same bits whatever the grid."""
import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("blocks", [1, 2, 3, 5, 6, 8, 16, 31, 32])
@pytest.mark.parametrize("rows", [[3, 0, 6, 1, 16, 17, 0, 2], [1]])
def test_tiles_in_turn(native, rows, blocks, layout):
    E, M, N, K = len(rows), sum(rows), 640, 128 * blocks
    g = torch.Generator().manual_seed(K + M)
    w = (torch.randn(E, N, K, generator=g) * 20).to(torch.float8_e4m3fn)
    a = (torch.randn(M, K, generator=g) * 40).to(torch.float8_e4m3fn)
    sa, sw = torch.rand(M, blocks, generator=g) * 0.02, torch.rand(E, N // 128, blocks, generator=g) * 0.02
    bias = torch.randn(E, N, generator=g).to(torch.bfloat16)
    af = a.double() * sa.double().repeat_interleave(128, 1)
    wf = w.double() * sw.double().repeat_interleave(128, 1).repeat_interleave(128, 2)
    ref = torch.cat([x @ wf[e].T + bias[e].double() for e, x in enumerate(af.split(rows))])
    # one rounding to bf16 and fp32 sums of K terms
    bound = 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * (af.abs() @ wf.abs().amax(0).T + 1)
    wd = (w if layout == 1 else w.transpose(1, 2).contiguous()).to(DEV)
    outs = []
    for ctas in [1, 2, 3, 5, 8, 17, 0]:
        d = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        torch.ops._xpu_C.b200_grouped_gemm(a.to(DEV), sa.to(DEV), wd, sw.to(DEV), bias.to(DEV), d,
                                           torch.tensor(rows, dtype=torch.int32, device=DEV), N, K, E, layout, 0, 1.702, 7.0,
                                           0.0, 0, ctas)
        outs.append(d.cpu())
        assert ((outs[-1].double() - ref).abs() <= bound).all(), ctas
    assert all(torch.equal(o.view(torch.int16), outs[0].view(torch.int16)) for o in outs)
