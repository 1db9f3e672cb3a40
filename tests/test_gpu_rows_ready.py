"""b200moe_gemm_args.rows_ready by itself, through the C ABI: the weights' prefetch ahead of the kernel's wait
(16-bit, fp8 in both tile forms, int4 planes) leaves the result as it is, bit for bit, and another value than 1
is no request for it."""
import ctypes as ct

import pytest
import torch

from conftest import PKG_DIR
from gemm_args import GemmArgs
from gpu_utils import DEV

pytestmark = pytest.mark.gpu

F16, BF16, E4M3, E4M3_X2 = 1, 2, 3, 9
W16_KN, W16_NK, FP8_BLOCK_NK, FP8_BLOCK_KN, INT4_NK = 0, 1, 3, 4, 7


@pytest.fixture(scope="module")
def lib(native):
    so = ct.CDLL(str(PKG_DIR / "vllm_xpu_kernels" / "libb200moe.so"))
    so.b200moe_last_error.restype = ct.c_char_p
    return so


@pytest.mark.parametrize("fmt", [W16_KN, W16_NK, FP8_BLOCK_NK, FP8_BLOCK_KN, INT4_NK])
@pytest.mark.parametrize("rows", [[3, 0, 5, 1], [40, 0, 129, 7], [0, 0, 0, 1]])
def test_result_does_not_depend_on_it(lib, fmt, rows):
    E, M, N, K = len(rows), sum(rows), 384, 640
    g = torch.Generator(device=DEV).manual_seed(fmt + M)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x = rnd(M, K).to(torch.bfloat16)
    st = torch.cuda.current_stream().cuda_stream
    a, a_scale, w_scale, a_dtype = x, None, None, BF16
    if fmt in (W16_KN, W16_NK):
        w = (rnd(E, K, N) if fmt == W16_KN else rnd(E, N, K)).to(torch.bfloat16)
    elif fmt == INT4_NK:
        w = torch.randint(0, 256, (E, N, K // 2), generator=g, device=DEV, dtype=torch.uint8)
        w_scale = torch.rand(E, N, K // 128, generator=g, device=DEV).to(torch.bfloat16)
        a = torch.empty(2, M, K, dtype=torch.uint8, device=DEV)
        a_scale, a_dtype = torch.empty(3, K // 128, M, dtype=torch.int32, device=DEV), E4M3_X2
        assert lib.b200moe_quant_mxfp8_ex(ct.c_void_p(x.data_ptr()), BF16, ct.c_void_p(a.data_ptr()),
                                          ct.c_void_p(a_scale.data_ptr()), ct.c_int64(M), K, 2, 1, 0, ct.c_void_p(st)) == 0
    else:
        w = rnd(*((E, N, K) if fmt == FP8_BLOCK_NK else (E, K, N))).to(torch.float8_e4m3fn)
        w_scale = torch.rand(E, N // 128, K // 128, generator=g, device=DEV)
        a, a_scale, a_dtype = x.to(torch.float8_e4m3fn), torch.rand(M, K // 128, generator=g, device=DEV), E4M3
    counts = torch.tensor(rows, dtype=torch.int32, device=DEV)
    outs = []
    for ready in (0, 1, 0x5a5a5a5a, -1):
        d = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        args = GemmArgs(a=a.data_ptr(), a_dtype=a_dtype, a_scale=a_scale.data_ptr() if a_scale is not None else None,
                        w=w.data_ptr(), w_format=fmt, w_scale=w_scale.data_ptr() if w_scale is not None else None,
                        d=d.data_ptr(), d_dtype=BF16, rows_per_expert=counts.data_ptr(), m=M, n=N, k=K, num_experts=E,
                        group_size=128, rows_ready=ready)
        torch.cuda.synchronize()      # the counts are complete
        rc = lib.b200moe_grouped_gemm(ct.byref(args), ct.c_void_p(st))
        assert rc == 0, lib.b200moe_last_error()
        torch.cuda.synchronize()
        outs.append(d)
    assert not outs[0].isnan().any()
    assert all(torch.equal(outs[0], d) for d in outs[1:])
