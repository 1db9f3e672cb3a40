"""int4 GEMM where the kernel takes 16- or 32-token tiles by the rows that it finds: each choice gives what the kernel with
16-token tiles alone gives (asked for by a small rows hint), bit for bit, and the 64-bit result within one rounding."""
import ctypes as ct

import pytest
import torch

from conftest import PKG_DIR
from gemm_args import GemmArgs
from gpu_utils import DEV

pytestmark = pytest.mark.gpu

F16, BF16, X2, X3, INT4_NK = 1, 2, 9, 11, 7

# (rows per expert, 9 or 10 on average; then 11 to 13 for float16): all within one tile, some beyond, most beyond, empty ones
COUNTS = [[16, 2, 13, 9], [10, 10, 10, 10], [17, 3, 12, 8], [40, 0, 0, 0], [0, 33, 0, 5], [31, 1, 1, 3] * 20, [9, 10] * 200]
COUNTS_F16 = [[13, 13, 12], [16, 17, 3, 16], [0, 26, 26, 0], [50, 1, 0, 1], [11] * 9 + [0, 32]]


@pytest.mark.parametrize("ctas", [0, 1, 5])
@pytest.mark.parametrize("unused", [0, 3])
@pytest.mark.parametrize("rows_ready", [0, 1])
@pytest.mark.parametrize("N,K", [(136, 128), (264, 640)])
@pytest.mark.parametrize("planes,counts", [(2, c) for c in COUNTS] + [(3, c) for c in COUNTS + COUNTS_F16])
def test_either_tile_gives_the_same(native, counts, planes, N, K, rows_ready, unused, ctas):
    if ctas == 1 and len(counts) > 20:
        ctas = 7
    dtype, type16, a_dtype = (torch.float16, F16, X3) if planes == 3 else (torch.bfloat16, BF16, X2)
    E, M = len(counts), sum(counts) + unused
    g = torch.Generator().manual_seed(M + K)
    w = torch.randint(0, 256, (E, N, K // 2), generator=g, dtype=torch.int32).to(torch.uint8)
    ws = (torch.rand(E, N, K // 128, generator=g) * K ** -0.5).to(dtype)
    bias = torch.randn(E, N, generator=g).to(dtype).to(DEV)
    # small whole numbers as codes of the first plane with scales of 1
    x = torch.randint(-16, 17, (M, K), generator=g).float()
    a = torch.zeros(planes, M, K, dtype=torch.uint8)
    a[0] = x.to(torch.float8_e4m3fn).view(torch.uint8)
    words = torch.full((planes, K // 128, M), 0x7f7f7f7f, dtype=torch.int32)
    sums = x.view(M, K // 128, 128).sum(-1).t().contiguous().view(torch.int32)
    a, scale, wd, wsd = a.to(DEV), torch.cat((words, sums.unsqueeze(0))).to(DEV), w.to(DEV), ws.to(DEV)
    rows = torch.tensor(counts, dtype=torch.int32, device=DEV)
    lib = ct.CDLL(str(PKG_DIR / "vllm_xpu_kernels" / "libb200moe.so"))
    lib.b200moe_last_error.restype = ct.c_char_p

    def gemm(hint):
        d = torch.full((M, N), float("nan"), dtype=dtype, device=DEV)
        args = GemmArgs(a=a.data_ptr(), a_dtype=a_dtype, a_scale=scale.data_ptr(), w=wd.data_ptr(), w_format=INT4_NK,
                        w_scale=wsd.data_ptr(), bias=bias.data_ptr(), d=d.data_ptr(), d_dtype=type16,
                        rows_per_expert=rows.data_ptr(), m=M, n=N, k=K, num_experts=E, group_size=128, max_ctas=ctas,
                        rows_ready=rows_ready, rows_hint=hint)
        rc = lib.b200moe_grouped_gemm(ct.byref(args), ct.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, lib.b200moe_last_error()
        return d
    used = M - unused
    got, plain = gemm(0), gemm(1)
    assert torch.equal(got[:used], plain[:used]) and got[used:].isnan().all()
    u = torch.stack((w & 15, w >> 4), -1).flatten(-2).int()
    exact_w = ((u ^ 8) - 8).double() * ws.double().repeat_interleave(128, -1)
    at = 0
    for e, n in enumerate(counts):
        want = x[at:at + n].double() @ exact_w[e].t() + bias[e].cpu().double()
        err = (got[at:at + n].cpu().double() - want).abs()
        # one rounding to the 16-bit type, and fp32 sums of up to five blocks of a few hundred
        assert (err <= want.abs() * torch.finfo(dtype).eps / 2 * 1.001 + 1e-3).all()
        at += n
