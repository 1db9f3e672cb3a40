"""moe_gather: rows of a token in flight one, two or eight at a time (by how many there are), with masked slots, odd
widths, and k of one to twelve; sums in fp32, k ascending, and a masked slot's weight never touches the sum."""
import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,K,H", [(1, 1, 8), (3, 2, 2880), (40, 3, 2056), (1024, 8, 64), (1025, 8, 64), (300, 9, 40), (683, 12, 136),
                                   (5000, 2, 16), (17, 8, 12)])
def test_gather_sums_in_order(native, T, K, H, dtype):
    g = torch.Generator().manual_seed(T + K)
    src = torch.randn(T * K, H, generator=g).to(dtype)
    w = torch.rand(T, K, generator=g)
    rm = torch.randperm(T * K, generator=g).to(torch.int32).view(T, K)
    gone = torch.rand(T, K, generator=g) < 0.3
    rm[gone] = -1
    w[gone] = float("nan")
    out = torch.full((T, H), float("nan"), dtype=dtype, device=DEV)
    torch.ops._moe_C.moe_gather(out, src.to(DEV), w.to(DEV), rm.to(DEV), 16)
    acc = torch.zeros(T, H, dtype=torch.float64)
    for k in range(K):     # a fused multiply-add rounds once: in 64 bits the product is exact, the sum rounded to 32
        step = acc + src[rm[:, k].long().clamp(min=0)].double() * w[:, k:k + 1].double()
        acc = torch.where(gone[:, k:k + 1], acc, step.float().double())
    assert torch.equal(out.cpu(), acc.float().to(dtype))
