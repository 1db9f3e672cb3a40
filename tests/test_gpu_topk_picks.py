"""Picks of the softmax / sigmoid top-k: a lane keeps every 32nd (or group-width-th) pick, so pick counts around
that width, ties, zeros of both signs, infinities, and biases beyond the mark of a taken column.  Bit for bit
the C restatement; a row with a NaN counts as lane 0 sees it, so those are compared on the other rows."""
import pytest
import torch

from gpu_utils import DEV, topk_sigmoid, topk_softmax
from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [5, 16, 17, 32, 33, 128, 200, 1000])
@pytest.mark.parametrize("softmax", [True, False])
def test_pick_counts_ties_and_special_values(native, E, softmax):
    g = torch.Generator().manual_seed(E)
    x = torch.randn(23, E, generator=g)
    x[3] = 0.0
    x[4] = -0.0
    x[5] = (x[5] * 2).round()                   # ties
    x[6, ::3] = float("-inf")
    x[7, E // 2] = 80.0
    for bias in (None, torch.randn(E, generator=g), torch.randn(E, generator=g) * 20000, torch.zeros(E).neg()):
        for K in sorted({1, 2, min(E, 8), min(E, 31), min(E, 32), min(E, 33), min(E, 65)}):
            for renorm in (False, True):
                b = bias.to(DEV) if bias is not None else None
                if softmax:
                    w, ids, src = topk_softmax(x.to(DEV), K, renorm, b)
                    ow, oi, osrc = co.topk_gating(x, K, renorm, bias, True)
                else:
                    w, ids, src = topk_sigmoid(x.to(DEV), K, renorm, b, 2.5)
                    ow, oi, osrc = co.topk_gating(x, K, renorm, bias, False, 2.5)
                assert torch.equal(ids.cpu(), oi) and torch.equal(src.cpu(), osrc)
                assert torch.equal(w.cpu(), ow)


def test_a_row_with_a_nan_leaves_the_others_alone(native):
    g = torch.Generator().manual_seed(1)
    for E, K in ((8, 2), (128, 8), (64, 40)):
        x = torch.randn(9, E, generator=g)
        y = x.clone()
        y[4, E // 3] = float("nan")
        w, ids, _ = topk_softmax(x.to(DEV), K, True)
        wn, idsn, _ = topk_softmax(y.to(DEV), K, True)
        keep = [i for i in range(9) if i != 4]
        assert torch.equal(ids[keep], idsn[keep]) and torch.equal(w[keep], wn[keep])
        assert ((idsn >= 0) & (idsn < E)).all()
