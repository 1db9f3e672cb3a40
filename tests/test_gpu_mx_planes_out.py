"""MXFP4 layers with SwigluOAI and up to 64 routed rows: gemm1 writes gemm2's input as e4m3 planes.  Bit for bit what
its 16-bit output through the quantiser gives, on both sides of the rule: one and several tiles an expert, widths
whose last scale word is padded and whose last feature tile is half a tile, both 16-bit types, biases."""
import pytest
import torch

from gpu_utils import DEV, grouped_gemm, quant_mxfp8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("planes,how", [(2, "mxfp8x2"), (1, "mxfp8")])
@pytest.mark.parametrize("T,H,I,E", [(1, 128, 320, 8), (3, 192, 192, 4), (17, 256, 320, 8), (32, 128, 128, 4), (31, 192, 448, 2),
                                     (25, 320, 192, 3), (33, 128, 192, 4), (300, 192, 448, 4)])
def test_layer_is_gemm_quantise_gemm(native, T, H, I, E, planes, how, dtype):
    K = 2
    g = torch.Generator().manual_seed(T + I)
    some = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=g, dtype=torch.int32).to(torch.uint8).to(DEV)
    w13, w2 = some(0, 256, E, 2 * I, H // 2).view(torch.float4_e2m1fn_x2), some(0, 256, E, H, I // 2).view(torch.float4_e2m1fn_x2)
    s13, s2 = some(117, 124, E, 2 * I, H // 32), some(117, 124, E, H, I // 32)
    b13, b2 = (torch.randn(E, n, generator=g).to(dtype).to(DEV) for n in (2 * I, H))
    x = torch.randn(T, H, generator=g).to(dtype).to(DEV)
    tw, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=g), -1), k=K, dim=-1)
    tw, ids = tw.to(DEV), ids.int().to(DEV)
    layer = native.XpuFusedMoe(w13, s13, b13, w2, s2, b2, K, "swigluoai", E, mxfp4_activations=how)
    out = torch.empty_like(x)
    layer.apply(out, x, tw, ids)
    # the stages apart
    rows, row_map = torch.empty(E, dtype=torch.int32, device=DEV), torch.empty(T, K, dtype=torch.int32, device=DEV)
    xp = torch.empty(T * K, H, dtype=dtype, device=DEV)
    torch.ops._moe_C.remap_hidden_states(x, None, xp, None, None, rows, row_map, ids, E, E)
    mid = grouped_gemm(*quant_mxfp8(xp, planes), w13, s13, b13, rows, 2 * I, H, epilogue=2, out_dtype=dtype, rows_out=T * K)
    assert not mid.isnan().any()
    d = grouped_gemm(*quant_mxfp8(mid, planes), w2, s2, b2, rows, H, I, out_dtype=dtype, rows_out=T * K)
    want = torch.empty_like(x)
    torch.ops._moe_C.moe_gather(want, d, tw, row_map, E)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("T", [1, 9, 40])
def test_per_tensor_fp8_weights_too(native, T):
    """The same kernel's other weights: [E, K, N] e4m3 with one scale per expert."""
    E, K, H, I, dtype = 8, 2, 256, 160, torch.bfloat16
    g = torch.Generator().manual_seed(T)
    w13, w2 = ((torch.randn(E, *s, generator=g)).to(torch.float8_e4m3fn).to(DEV) for s in ((H, 2 * I), (I, H)))
    s13, s2 = ((torch.rand(E, generator=g) * 0.1 + 0.02).to(DEV) for _ in range(2))
    x = torch.randn(T, H, generator=g).to(dtype).to(DEV)
    tw, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=g), -1), k=K, dim=-1)
    tw, ids = tw.to(DEV), ids.int().to(DEV)
    layer = native.XpuFusedMoe(w13, s13, None, w2, s2, None, K, "swigluoai", E, fuse_activation=True)
    out = torch.empty_like(x)
    layer.apply(out, x, tw, ids)
    rows, row_map = torch.empty(E, dtype=torch.int32, device=DEV), torch.empty(T, K, dtype=torch.int32, device=DEV)
    xp = torch.empty(T * K, H, dtype=dtype, device=DEV)
    torch.ops._moe_C.remap_hidden_states(x, None, xp, None, None, rows, row_map, ids, E, E)
    mid = grouped_gemm(*quant_mxfp8(xp, 2), w13, s13, None, rows, 2 * I, H, epilogue=2, rows_out=T * K)
    d = grouped_gemm(*quant_mxfp8(mid, 2), w2, s2, None, rows, H, I, rows_out=T * K)
    want = torch.empty_like(x)
    torch.ops._moe_C.moe_gather(want, d, tw, row_map, E)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
