"""MXFP4 layers with SwigluOAI and up to 64 routed rows: gemm1 writes gemm2's input as e4m3 planes.  Bit for bit what
its 16-bit output through the quantiser gives, on both sides of the rule: one and several tiles an expert, one and many
tiles a CTA (the two buffers that pairs of warps exchange halves through are then written again and again), widths whose
last scale word is padded and whose last feature tile is half a tile, both 16-bit types, biases."""
import ctypes as ct

import pytest
import torch

from conftest import PKG_DIR
from gemm_args import GemmArgs
from gpu_utils import DEV, grouped_gemm, quant_mxfp8

pytestmark = pytest.mark.gpu

FP8_TENSOR_KN, MXFP4_NK, MXFP8_KN, SWIGLUOAI = 2, 5, 8, 2


@pytest.mark.parametrize("ctas", [0, 1, 2, 3])
@pytest.mark.parametrize("fmt,N,K", [(MXFP4_NK, 192, 192), (MXFP4_NK, 448, 320), (MXFP4_NK, 1088, 256), (FP8_TENSOR_KN, 320, 160),
                                     (MXFP8_KN, 320, 288)])
@pytest.mark.parametrize("planes,dtype", [(2, torch.bfloat16), (1, torch.float16)])
@pytest.mark.parametrize("counts", [[40, 0, 3, 17], [1], [0, 33, 16, 15, 0]])
def test_planes_of_the_gemm_itself(native, counts, planes, dtype, fmt, N, K, ctas):
    """The GEMM with planes asked for: up to 3 token tiles an expert, half a feature tile at the end, up to 54 tiles a CTA."""
    E, M = len(counts), sum(counts)
    g = torch.Generator().manual_seed(N + M)
    some = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=g, dtype=torch.int32).to(torch.uint8).to(DEV)
    if fmt == MXFP4_NK:
        w, ws = some(0, 256, E, N, K // 2).view(torch.float4_e2m1fn_x2), some(117, 124, E, N, K // 32)
    else:
        w = torch.randn(E, K, N, generator=g).to(torch.float8_e4m3fn).to(DEV)
        ws = some(117, 124, E, K // 32, N) if fmt == MXFP8_KN else (torch.rand(E, generator=g) * 0.1 + 0.02).to(DEV)
    bias = torch.randn(E, N, generator=g).to(dtype).to(DEV)
    rows = torch.tensor(counts, dtype=torch.int32, device=DEV)
    a, a_scale = quant_mxfp8(torch.randn(M, K, generator=g).to(dtype).to(DEV), planes)
    lib = ct.CDLL(str(PKG_DIR / "vllm_xpu_kernels" / "libb200moe.so"))
    lib.b200moe_last_error.restype = ct.c_char_p
    stream = ct.c_void_p(torch.cuda.current_stream().cuda_stream)
    a_dtype, type16 = (9 if planes == 2 else 3), (1 if dtype == torch.float16 else 2)

    def gemm(d, d_dtype, d_scale, ctas):
        args = GemmArgs(a=a.data_ptr(), a_dtype=a_dtype, a_scale=a_scale.data_ptr(), w=w.data_ptr(), w_format=fmt,
                        w_scale=ws.data_ptr(), bias=bias.data_ptr(), d=d.data_ptr(), d_dtype=d_dtype, d_scale=d_scale,
                        mid_dtype=type16, rows_per_expert=rows.data_ptr(), m=M, n=N, k=K, num_experts=E, epilogue=SWIGLUOAI,
                        act_alpha=1.702, act_limit=7.0, max_ctas=ctas)
        assert lib.b200moe_grouped_gemm(ct.byref(args), stream) == 0, lib.b200moe_last_error()
        return d
    mid = gemm(torch.full((M, N // 2), float("nan"), dtype=dtype, device=DEV), type16, None, 0)
    assert not mid.isnan().any()
    want_q, want_s = quant_mxfp8(mid, planes)
    s = torch.full_like(want_s, 0x55555555)
    q = gemm(torch.full((planes * M, N // 2), 0x55, dtype=torch.uint8, device=DEV), a_dtype, s.data_ptr(), ctas)
    assert torch.equal(q, want_q.view(torch.uint8)) and torch.equal(s, want_s)


def _launches(call):
    """Nodes of the graph that a call is captured into: its launches."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    n = ct.c_size_t()
    rt = ct.CDLL("libcudart.so.12")
    assert rt.cudaGraphGetNodes(ct.c_void_p(graph.raw_cuda_graph()), None, ct.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("ctas", [1, 2, 3])
@pytest.mark.parametrize("T,H,I,E", [(32, 192, 448, 8), (29, 128, 320, 8), (24, 256, 192, 7)])
def test_layer_with_many_tiles_a_cta(native, T, H, I, E, ctas):
    """A layer that takes the path (one launch fewer than with one expert too few for it), most rows on two experts, and
    CTAs with many tiles: what one tile a CTA gives."""
    K, dtype = 2, torch.bfloat16
    g = torch.Generator().manual_seed(T)
    some = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=g, dtype=torch.int32).to(torch.uint8).to(DEV)
    w13, w2 = some(0, 256, E, 2 * I, H // 2).view(torch.float4_e2m1fn_x2), some(0, 256, E, H, I // 2).view(torch.float4_e2m1fn_x2)
    s13, s2 = some(117, 124, E, 2 * I, H // 32), some(117, 124, E, H, I // 32)
    x = torch.randn(T, H, generator=g).to(dtype).to(DEV)
    ids = torch.tensor([[1, 2]] * (T - 4) + [[E - 1, 0]] * 4, dtype=torch.int32, device=DEV)
    tw = torch.rand(T, K, generator=g).to(DEV)
    layer = native.XpuFusedMoe(w13, s13, None, w2, s2, None, K, "swigluoai", E)
    outs = []
    for n in (0, ctas):
        layer.gemm_max_ctas = n
        outs.append(torch.full_like(x, float("nan")))
        layer.apply(outs[-1], x, tw, ids)
    assert not outs[0].isnan().any() and torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    if ctas == 1:
        few = (T * K - 1) // 8                  # experts for which T * K rows are more than 8 each
        other = native.XpuFusedMoe(w13[:few].contiguous(), s13[:few].contiguous(), None, w2[:few].contiguous(),
                                   s2[:few].contiguous(), None, K, "swigluoai", few)
        out, low = torch.empty_like(x), ids.clamp(max=few - 1)
        assert _launches(lambda: layer.apply(out, x, tw, ids)) + 1 == _launches(lambda: other.apply(out, x, tw, low))


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
