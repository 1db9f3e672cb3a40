"""The activation planes of an int4 GEMM at the C ABI: codes in their own order, as the types X2 and X3 say (a caller may
make them itself), and in the order that the types ..._EVENS_FIRST name.  The quantisers write either, with the same scale
words and sums, and the GEMM gives the same bits for both, in each of its tiles."""
import ctypes as ct

import pytest
import torch

from conftest import PKG_DIR
from gemm_args import GemmArgs
from gpu_utils import DEV

pytestmark = pytest.mark.gpu

F16, BF16, E4M3_X2, E4M3_X3, X2_EVENS_FIRST, X3_EVENS_FIRST, I32, INT4_NK = 1, 2, 9, 11, 12, 13, 5, 7
IN_ORDER, EVENS_FIRST = 0, 16
ORDER = [0, 2, 4, 6, 1, 3, 5, 7]


@pytest.fixture(scope="module")
def lib(native):
    so = ct.CDLL(str(PKG_DIR / "vllm_xpu_kernels" / "libb200moe.so"))
    so.b200moe_last_error.restype = ct.c_char_p
    return so


def _ptr(t):
    return ct.c_void_p(t.data_ptr())


def _stream():
    return ct.c_void_p(torch.cuda.current_stream().cuda_stream)


def _quantise(lib, x, planes, order, gated=0, block_sums=1):
    rows, cols = x.shape[0], x.shape[1] // (2 if gated else 1)
    q = torch.empty(planes, rows, cols, dtype=torch.uint8, device=DEV)
    s = torch.empty(planes + 1, (cols + 127) // 128, rows, dtype=torch.int32, device=DEV)
    rc = lib.b200moe_quant_mxfp8_ex(_ptr(x), F16 if x.dtype == torch.float16 else BF16, _ptr(q), _ptr(s), ct.c_int64(rows), cols,
                                    planes + order, block_sums, gated, _stream())
    assert rc == 0, lib.b200moe_last_error()
    return q, s


def _gemm(lib, a, a_scale, a_dtype, w, w_scale, counts, M, N, K, dtype):
    d = torch.full((M, N), float("nan"), dtype=dtype, device=DEV)
    args = GemmArgs(a=a.data_ptr(), a_dtype=a_dtype, a_scale=a_scale.data_ptr(), w=w.data_ptr(), w_format=INT4_NK,
                    w_scale=w_scale.data_ptr(), d=d.data_ptr(), d_dtype=F16 if dtype == torch.float16 else BF16,
                    rows_per_expert=counts.data_ptr(), m=M, n=N, k=K, num_experts=counts.numel(), group_size=128)
    assert lib.b200moe_grouped_gemm(ct.byref(args), _stream()) == 0, lib.b200moe_last_error()
    return d


def _weights(g, E, N, K, dtype):
    w = torch.randint(0, 256, (E, N, K // 2), generator=g, dtype=torch.int32).to(torch.uint8)
    s = (torch.rand(E, N, K // 128, generator=g) * K ** -0.5).to(dtype)
    u = torch.stack((w & 15, w >> 4), -1).flatten(-2).int()
    return w.to(DEV), s.to(DEV), ((u ^ 8) - 8).double() * s.double().repeat_interleave(128, -1)


@pytest.mark.parametrize("dtype,planes", [(torch.bfloat16, 2), (torch.float16, 3)])
@pytest.mark.parametrize("rows", [[3, 0, 5, 1], [16, 30, 40, 1]])
def test_planes_that_the_caller_made(lib, rows, dtype, planes):
    """Small whole numbers as e4m3 codes with scales of 1, the other planes zero, sums of the blocks behind the words."""
    E, M, N, K = len(rows), sum(rows), 264, 256
    g = torch.Generator().manual_seed(M)
    w, ws, exact_w = _weights(g, E, N, K, dtype)
    x = torch.randint(-16, 17, (M, K), generator=g).float()
    a = torch.zeros(planes, M, K, dtype=torch.uint8)
    a[0] = x.to(torch.float8_e4m3fn).view(torch.uint8)
    words = torch.full((planes, K // 128, M), 0x7f7f7f7f, dtype=torch.int32)
    sums = x.view(M, K // 128, 128).sum(-1).t().contiguous().view(torch.int32)
    scale = torch.cat((words, sums.unsqueeze(0))).to(DEV)
    counts = torch.tensor(rows, dtype=torch.int32, device=DEV)
    got = _gemm(lib, a.to(DEV), scale, E4M3_X3 if planes == 3 else E4M3_X2, w, ws, counts, M, N, K, dtype)
    e_of = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))
    want = torch.einsum("mk,mnk->mn", x.double(), exact_w[e_of])
    # one rounding to the 16-bit type, and fp32 sums of two blocks
    assert ((got.cpu().double() - want).abs() <= want.abs() * torch.finfo(dtype).eps / 2 * 1.001 + 1e-4).all()
    # ... and the same codes in the other order
    b = a.view(planes, M, K // 8, 8)[..., ORDER].reshape(planes, M, K).contiguous()
    other = _gemm(lib, b.to(DEV), scale, X3_EVENS_FIRST if planes == 3 else X2_EVENS_FIRST, w, ws, counts, M, N, K, dtype)
    assert torch.equal(got, other)


@pytest.mark.parametrize("gated", [0, 1])
@pytest.mark.parametrize("dtype,planes", [(torch.bfloat16, 2), (torch.float16, 3), (torch.bfloat16, 1)])
@pytest.mark.parametrize("rows,cols", [(1, 32), (7, 160), (33, 640)])
def test_quantiser_writes_both_orders(lib, rows, cols, dtype, planes, gated):
    g = torch.Generator().manual_seed(cols)
    x = torch.randn(rows, cols * (1 + gated), generator=g).to(dtype).to(DEV)
    q, s = _quantise(lib, x, planes, IN_ORDER, gated)
    for other in (2, 16, -1):                            # any value but zero asks for the sums, and for nothing else
        again = _quantise(lib, x, planes, IN_ORDER, gated, other)
        assert torch.equal(q, again[0]) and torch.equal(s, again[1])
    q2, s2 = _quantise(lib, x, planes, EVENS_FIRST, gated)
    assert torch.equal(s, s2)
    assert torch.equal(q.view(planes, rows, cols // 8, 8)[..., ORDER].reshape_as(q), q2)
    # the planes add up to the values, in order
    if not gated:
        byte = s[:planes].contiguous().view(torch.uint8).view(planes, -1, rows, 4).permute(0, 2, 1, 3).reshape(planes, rows, -1)
        scale = torch.exp2(byte.double() - 127).repeat_interleave(32, -1)[..., :cols]
        value = (q.view(torch.float8_e4m3fn).double() * scale).sum(0)
        # (each plane leaves half a step, 2^-4, of what the one before left, or less)
        bound = x.double().abs().view(rows, cols // 32, 32).amax(-1).repeat_interleave(32, -1) * 2.0 ** (-4 * planes)
        assert ((value - x.double()).abs() <= bound).all()


@pytest.mark.parametrize("dtype,planes", [(torch.bfloat16, 2), (torch.float16, 3)])
def test_remap_and_quantise_as_the_quantiser_does(lib, dtype, planes):
    T, K, E, H = 37, 2, 4, 256
    g = torch.Generator().manual_seed(4)
    x = torch.randn(T, H, generator=g).to(dtype).to(DEV)
    ids = torch.stack([torch.randperm(E, generator=g)[:K] for _ in range(T)]).int().to(DEV)
    order = torch.sort(ids.flatten(), stable=True).indices
    for codes, block_sums in ((IN_ORDER, 1), (IN_ORDER, 2), (EVENS_FIRST, 1)):
        want_q, want_s = _quantise(lib, x[order // K].contiguous(), planes, codes)
        q, s = torch.empty_like(want_q), torch.empty_like(want_s)
        rows, row_map = torch.empty(E, dtype=torch.int32, device=DEV), torch.empty(T, K, dtype=torch.int32, device=DEV)
        rc = lib.b200moe_remap_quant_mxfp8(_ptr(x), F16 if dtype == torch.float16 else BF16, _ptr(q), _ptr(s), planes + codes,
                                           block_sums, None, _ptr(rows), _ptr(row_map), _ptr(ids), I32, ct.c_int64(T), H, K, E, E, None,
                                           ct.c_size_t(0), _stream())
        assert rc == 0, lib.b200moe_last_error()
        assert torch.equal(q, want_q) and torch.equal(s, want_s)


def test_other_weights_refuse_the_order(lib):
    a = torch.zeros(4, 256, dtype=torch.uint8, device=DEV)
    for a_dtype in (X2_EVENS_FIRST, X3_EVENS_FIRST):
        args = GemmArgs(a=a.data_ptr(), a_dtype=a_dtype, a_scale=a.data_ptr(), w=a.data_ptr(), w_format=5, w_scale=a.data_ptr(),
                        d=a.data_ptr(), d_dtype=BF16, rows_per_expert=a.data_ptr(), m=1, n=64, k=128, num_experts=1)
        assert lib.b200moe_grouped_gemm(ct.byref(args), _stream()) == -1


@pytest.mark.parametrize("terms,block_sums", [(EVENS_FIRST + 2, 0), (EVENS_FIRST, 1), (EVENS_FIRST + 4, 1), (4, 1), (0, 1), (-14, 1)])
def test_quantiser_refuses_other_plane_counts(lib, terms, block_sums):
    x = torch.zeros(4, 256, dtype=torch.bfloat16, device=DEV)
    q, s = torch.empty(5, 4, 256, dtype=torch.uint8, device=DEV), torch.empty(5, 2, 4, dtype=torch.int32, device=DEV)
    assert lib.b200moe_quant_mxfp8_ex(_ptr(x), BF16, _ptr(q), _ptr(s), ct.c_int64(4), 256, terms, block_sums, 0, _stream()) == -1
