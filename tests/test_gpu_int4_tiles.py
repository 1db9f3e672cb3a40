"""INT4 layers on the two kernels that take them, against the CPU oracle: the block-scaled one (few rows
per expert, scales per 128 and 256 elements, two and three activation planes) and the one that expands
the weights into tensor memory (more rows, or finer scales).  Token tiles and their remainders, several
tiles per CTA, K down to half a block, feature tiles cut off by N."""
import pytest
import torch

from gpu_utils import DEV
from oracle import torch_oracle as to

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,H,I,group", [(1, 128, 128, 128), (9, 256, 384, 128), (33, 640, 256, 128), (70, 512, 512, 256),
                                         (150, 256, 256, 256), (401, 384, 128, 128),
                                         (3, 192, 320, 64), (70, 128, 192, 32), (640, 64, 2560, 64),
                                         (900, 192, 1536, 64), (1100, 640, 768, 128)])
def test_layer_int4(native, dtype, T, H, I, group):
    E, K = 4, 2
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, H, generator=g).to(dtype)
    w13 = torch.randint(0, 256, (E, 2 * I, H // 2), generator=g, dtype=torch.int32).to(torch.uint8)
    w2 = torch.randint(0, 256, (E, H, I // 2), generator=g, dtype=torch.int32).to(torch.uint8)
    s13 = (torch.rand(E, 2 * I, H // group, generator=g) * 0.4 + 0.1).mul(H ** -0.5).to(dtype)
    s2 = (torch.rand(E, H, I // group, generator=g) * 0.4 + 0.1).mul(I ** -0.5).to(dtype)
    b13 = torch.randn(E, 2 * I, generator=g).to(dtype)
    b2 = torch.randn(E, H, generator=g).to(dtype)
    tw, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=g), -1), k=K, dim=-1)
    ref = to.fused_moe_bf16(x, to.dequant_int4(w13, s13, group), b13, to.dequant_int4(w2, s2, group), b2, tw, ids.int(), E)
    mv = lambda t: t.to(DEV)
    layer = native.XpuFusedMoe(mv(w13), mv(s13), mv(b13), mv(w2), mv(s2), mv(b2), K, "silu", E)
    out = torch.empty_like(x, device=DEV)
    layer.apply(out, mv(x), mv(tw), mv(ids.int()))
    torch.testing.assert_close(out.cpu().float(), ref.float(), rtol=2e-2, atol=2e-2 * float(ref.float().abs().max()))
    err = (out.cpu().float() - ref.float()).norm() / ref.float().norm()
    assert err < (1e-2 if dtype == torch.bfloat16 else 2e-3), err


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,H,I", [(20, 256, 384), (21, 640, 256), (26, 384, 128), (27, 256, 640), (32, 512, 384), (30, 128, 256)])
def test_layer_int4_on_both_sides_of_the_tile_lines(native, dtype, T, H, I):
    """Rows per expert (half of T) around the lines of 10 (bfloat16) and 13 (float16), and up to the 16 at which another
    kernel takes over: 16- and 32-token tiles of two and three planes, several tiles an expert (routing as it comes)."""
    test_layer_int4(native, dtype, T, H, I, 128)


@pytest.mark.parametrize("ctas", [1, 3])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T", [24, 30])
def test_int4_tiles_that_follow_one_another(native, dtype, T, ctas):
    """Few CTAs that walk many tiles give what one tile a CTA gives, bit for bit; some experts have none, some several."""
    E, K, H, I, group = 4, 2, 384, 640, 128
    g = torch.Generator().manual_seed(T)
    w13, w2 = (torch.randint(0, 256, s, generator=g, dtype=torch.int32).to(torch.uint8).to(DEV)
               for s in ((E, 2 * I, H // 2), (E, H, I // 2)))
    s13, s2 = ((torch.rand(E, n, k // group, generator=g) * 0.2 + 0.1).mul(k ** -0.5).to(dtype).to(DEV) for n, k in ((2 * I, H), (H, I)))
    x = torch.randn(T, H, generator=g).to(dtype).to(DEV)
    ids = torch.tensor([[0, 2]] * (T - 3) + [[2, 3]] * 3, dtype=torch.int32, device=DEV)
    tw = torch.rand(T, K, generator=g).to(DEV)
    layer = native.XpuFusedMoe(w13, s13, None, w2, s2, None, K, "silu", E)
    outs = []
    for n in (0, ctas):
        layer.gemm_max_ctas = n
        outs.append(torch.full_like(x, float("nan")))
        layer.apply(outs[-1], x, tw, ids)
    assert not outs[0].isnan().any() and torch.equal(*outs)


@pytest.mark.parametrize("T", [9, 70])
@pytest.mark.parametrize("size", [1e-6, 1e-11, 1e-14])
def test_layer_int4_keeps_small_activations(native, T, size):
    """bfloat16 hidden states far below 1, whose gated product gemm2 sees squared: both kernels keep their
    relative precision (up to 16 rows per expert the activations are e4m3 planes)."""
    E, K, H, I, group = 4, 2, 256, 128, 128
    g = torch.Generator().manual_seed(T)
    x = (torch.randn(T, H, generator=g) * size).to(torch.bfloat16)
    w13 = torch.randint(0, 256, (E, 2 * I, H // 2), generator=g, dtype=torch.int32).to(torch.uint8)
    w2 = torch.randint(0, 256, (E, H, I // 2), generator=g, dtype=torch.int32).to(torch.uint8)
    s13 = (torch.rand(E, 2 * I, H // group, generator=g) * 0.4 + 0.1).mul(H ** -0.5).to(torch.bfloat16)
    s2 = (torch.rand(E, H, I // group, generator=g) * 0.4 + 0.1).mul(I ** -0.5).to(torch.bfloat16)
    tw, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=g), -1), k=K, dim=-1)
    ref = to.fused_moe_bf16(x, to.dequant_int4(w13, s13, group), None, to.dequant_int4(w2, s2, group), None, tw, ids.int(), E)
    mv = lambda t: t.to(DEV)
    layer = native.XpuFusedMoe(mv(w13), mv(s13), None, mv(w2), mv(s2), None, K, "silu", E)
    out = torch.empty_like(x, device=DEV)
    layer.apply(out, mv(x), mv(tw), mv(ids.int()))
    assert float(ref.abs().max()) > 0
    err = (out.cpu().double() - ref.double()).norm() / ref.double().norm()
    assert err < 1e-2, err


@pytest.mark.parametrize("dtype,bar", [(torch.bfloat16, 6e-3), (torch.float16, 8e-4)])
def test_int4_tokens_in_a_small_and_a_large_batch(native, dtype, bar):
    """Up to 16 rows per expert a group's scale multiplies the block's sum, above every weight is rounded
    after its scale: the same tokens come out differently, both as close to exact arithmetic as 16-bit rows
    between the stages allow (bar: sqrt(5) roundings of about 2^-9 resp. 2^-12 of their size)."""
    E, K, H, I, group, T = 4, 2, 512, 384, 128, 16
    g = torch.Generator().manual_seed(5)
    x = torch.randn(40 * T, H, generator=g).to(dtype)
    codes = [torch.randint(0, 256, s, generator=g, dtype=torch.int32).to(torch.uint8) for s in ((E, 2 * I, H // 2), (E, H, I // 2))]
    scales = [(torch.rand(E, n, k // group, generator=g) * 0.2 + 0.1).mul(k ** -0.5).to(dtype) for n, k in ((2 * I, H), (H, I))]
    tw, ids = torch.topk(torch.softmax(torch.randn(40 * T, E, generator=g), -1), k=K, dim=-1)
    layer = native.XpuFusedMoe(codes[0].to(DEV), scales[0].to(DEV), None, codes[1].to(DEV), scales[1].to(DEV), None, K, "silu", E)
    outs = []
    for n in (T, 40 * T):
        out = torch.empty(n, H, dtype=dtype, device=DEV)
        layer.apply(out, x[:n].to(DEV), tw[:n].to(DEV), ids[:n].int().to(DEV))
        outs.append(out[:T].cpu().double())
    w13, w2 = (torch.stack((c & 15, c >> 4), -1).flatten(-2).double().sub(8).mul(s.double().repeat_interleave(group, -1))
               for c, s in zip(codes, scales))
    exact = torch.zeros(T, H, dtype=torch.float64)
    for t in range(T):
        for k in range(K):
            h = w13[ids[t, k]] @ x[t].double()
            exact[t] += tw[t, k].double() * (w2[ids[t, k]] @ (torch.nn.functional.silu(h[:I]) * h[I:]))
    few, many = ((o - exact).norm() / exact.norm() for o in outs)
    apart = (outs[0] - outs[1]).norm() / exact.norm()
    print(f"{dtype}: few rows {few:.2e}, many rows {many:.2e}, apart {apart:.2e}")
    assert few < bar and many < bar and 0 < apart < 2 * bar


@pytest.mark.parametrize("act", ["silu", "swigluoai"])
@pytest.mark.parametrize("T", [5, 100])
def test_int4_layer_with_the_activation_asked_into_gemm1(native, act, T):
    """fuse_activation=True is taken at every size: the block-scaled kernel, which has no such epilogue, steps
    aside for the ones that have."""
    E, K, H, I, group = 4, 2, 256, 256, 128
    g = torch.Generator().manual_seed(T)
    w13, w2 = (torch.randint(0, 256, s, generator=g, dtype=torch.int32).to(torch.uint8).to(DEV)
               for s in ((E, 2 * I, H // 2), (E, H, I // 2)))
    s13, s2 = ((torch.rand(E, n, k // group, generator=g) * 0.2 + 0.1).mul(k ** -0.5).to(torch.bfloat16).to(DEV)
               for n, k in ((2 * I, H), (H, I)))
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    tw, ids = torch.topk(torch.softmax(torch.randn(T, E, generator=g), -1), k=K, dim=-1)
    outs = []
    for fuse in (True, False):
        layer = native.XpuFusedMoe(w13, s13, None, w2, s2, None, K, act, E, fuse_activation=fuse)
        outs.append(torch.empty_like(x))
        layer.apply(outs[-1], x, tw.to(DEV), ids.int().to(DEV))
    a, b = (o.double() for o in outs)
    assert (a - b).norm() / b.norm() < 1e-2      # (a rounding of the intermediate, at few rows of the weights too)
