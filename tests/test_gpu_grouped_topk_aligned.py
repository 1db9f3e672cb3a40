"""Grouped top-k over 64 to 512 experts in a power-of-two number of groups (its own kernel): all group counts,
ties within and across groups, infinities and NaN, more picks than the kept groups hold; a buffer that does not
begin on a 16-byte boundary takes the general kernel.  Bit for bit the C restatement."""
import pytest
import torch

from gpu_utils import DEV
from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


def _check(scores, swb, ng, tg, K, renorm=True, shift=0):
    s, b = scores.to(DEV), swb.to(DEV)
    if shift:
        b = torch.cat([b.new_zeros(shift), b.flatten()])[shift:].view(swb.shape)
    v, i = torch.ops._moe_C.grouped_topk(s, b, ng, tg, K, renorm, 2.5)
    ov, oi = co.grouped_topk(scores, swb, ng, tg, K, renorm, 2.5)
    assert torch.equal(i.cpu(), oi)
    assert torch.equal(v.cpu().view(torch.uint8), ov.view(torch.uint8)) or torch.equal(v.cpu(), ov)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("E", [64, 128, 256, 512])
def test_all_group_counts(native, E, dtype):
    g = torch.Generator().manual_seed(E)
    scores = torch.sigmoid(torch.randn(37, E, generator=g)).to(dtype)
    swb = (scores.float() + torch.randn(E, generator=g) * 0.1).to(dtype)
    coarse = (swb.float() * 8).round().div(8).to(dtype)            # many ties
    for ng in (1, 2, 4, 8, 16, 32):
        for tg in sorted({1, max(1, ng // 2), ng}):
            for K in (1, 8, 32):
                _check(scores, swb, ng, tg, K)
                _check(scores, coarse, ng, tg, K, renorm=False)
    _check(scores, swb, 8, 4, 8, shift=1)


def test_special_values(native):
    g = torch.Generator().manual_seed(5)
    scores = torch.sigmoid(torch.randn(64, 256, generator=g))
    swb = scores + torch.randn(256, generator=g) * 0.1
    for n, x in enumerate([float("nan"), float("inf"), -float("inf"), 0.0, -0.0]):
        swb[torch.rand(64, 256, generator=g) < 0.1] = x
        _check(scores, swb, 8, 4, 8)
    swb[3] = -float("inf")
    swb[4, :200] = -float("inf")
    swb[5] = 0.0
    swb[5, ::2] = -0.0
    swb[6] = float("nan")
    for tg in (1, 3, 8):
        _check(scores, swb, 8, tg, 8)
