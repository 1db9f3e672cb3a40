"""Token-major fp8 GEMM, 256-feature tiles: rows leave 32 at a time by TMA and the rest of an expert from the
registers, so segments end at every place around 32 and 128 rows; K of one block (a tile per block), of
three (scale groups span tiles); N of one and a half tiles; bias; float16; a D that begins on a 16-byte boundary."""
import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu

ROWS = [31, 0, 32, 33, 64, 127, 128, 129, 160, 1, 95, 97]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,K,offset", [(256, 128, 0), (384, 384, 8), (640, 128, 0), (1024, 640, 8)])
def test_fp8_rows_end_anywhere(native, dtype, N, K, offset):
    E, M = len(ROWS), sum(ROWS)
    g = torch.Generator().manual_seed(N + K)
    w = (torch.randn(E, N, K, generator=g) * 20).to(torch.float8_e4m3fn)
    a = (torch.randn(M, K, generator=g) * 40).to(torch.float8_e4m3fn)
    sa, sw = torch.rand(M, K // 128, generator=g) * 0.02, torch.rand(E, N // 128, K // 128, generator=g) * 0.02
    bias = torch.randn(E, N, generator=g).to(dtype)
    af = a.double() * sa.double().repeat_interleave(128, 1)
    wf = w.double() * sw.double().repeat_interleave(128, 1).repeat_interleave(128, 2)
    ref = torch.cat([x @ wf[e].T + bias[e].double() for e, x in enumerate(af.split(ROWS))])
    # D between guards: `offset` elements before it, 40 rows behind it
    mem = torch.full((offset + (M + 40) * N,), float("nan"), dtype=dtype, device=DEV)
    d = mem[offset:offset + M * N].view(M, N)
    torch.ops._xpu_C.b200_grouped_gemm(a.to(DEV), sa.to(DEV), w.to(DEV), sw.to(DEV), bias.to(DEV), d,
                                       torch.tensor(ROWS, dtype=torch.int32, device=DEV), N, K, E, 1)
    assert mem[:offset].isnan().all() and mem[offset + M * N:].isnan().all()
    out = d.cpu().double()
    # one rounding to the 16-bit type (half an ulp: 2^-8 / 2^-11 of the value) and fp32 sums of K terms
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    bound = half_ulp * ref.abs() + K * 2.0 ** -24 * (af.abs() @ wf.abs().amax(0).T + 1)
    assert not out.isnan().any()
    assert ((out - ref).abs() <= bound).all()
