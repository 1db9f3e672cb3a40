"""Permutation with the bookkeeping in the same launch (up to 2048 routed slots, top-k up to 8)
and the separate sort beyond: exact against the oracle's bookkeeping on both sides of each limit,
the MXFP8 form against copying and quantising in two steps."""
import pytest
import torch

from gpu_utils import DEV
from oracle import c_oracle as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,K", [(1, 1), (3, 8), (256, 8), (257, 8), (2048, 1), (2049, 1), (5, 9), (40, 32)])
@pytest.mark.parametrize("E,masked", [(8, False), (1024, False), (64, True)])
def test_positions_and_rows(native, T, K, E, masked):
    g = torch.Generator().manual_seed(T * 100 + K + E)
    ids = torch.randint(0, E, (T, K), generator=g, dtype=torch.int32)
    ids[0, 0] = -1
    local = E // 2 if masked else E
    emap = None
    if masked:
        emap = torch.full((E,), -1, dtype=torch.int32)
        emap[E - local:] = torch.arange(local, dtype=torch.int32)
    x = torch.randn(T, 64, generator=g).to(torch.bfloat16)
    rows, row_map = co.remap_bookkeeping(ids, emap, E, local)
    out = torch.zeros(T * K, 64, dtype=torch.bfloat16, device=DEV)
    r = torch.empty(local, dtype=torch.int32, device=DEV)
    m = torch.empty(T, K, dtype=torch.int32, device=DEV)
    torch.ops._moe_C.remap_hidden_states(x.to(DEV), None, out, None, emap.to(DEV) if masked else None, r, m,
                                         ids.to(DEV), E, local)
    assert torch.equal(r.cpu(), rows) and torch.equal(m.cpu(), row_map.view(T, K))
    want = torch.zeros(T * K, 64, dtype=torch.bfloat16)
    for t in range(T):
        for k in range(K):
            if row_map.view(T, K)[t, k] >= 0:
                want[row_map.view(T, K)[t, k]] = x[t]
    assert torch.equal(out.cpu(), want)


@pytest.mark.parametrize("T", [7, 300])
@pytest.mark.parametrize("planes", ["mxfp8", "mxfp8x2"])
def test_layer_quantises_rows_while_it_places_them(native, T, planes):
    """An MXFP4 layer quantises each token once and writes the codes to its K places: the same as
    quantising the placed rows, so a token's output does not depend on where its rows went."""
    E, K, H, I = 8, 8, 192, 128
    g = torch.Generator().manual_seed(T)
    w13 = torch.randint(0, 256, (E, 2 * I, H // 2), generator=g, dtype=torch.int32).to(torch.uint8).to(DEV)
    w2 = torch.randint(0, 256, (E, H, I // 2), generator=g, dtype=torch.int32).to(torch.uint8).to(DEV)
    s13 = torch.full((E, 2 * I, H // 32), 120, dtype=torch.uint8, device=DEV)
    s2 = torch.full((E, H, I // 32), 120, dtype=torch.uint8, device=DEV)
    layer = native.XpuFusedMoe(w13.view(torch.float4_e2m1fn_x2), s13, None, w2.view(torch.float4_e2m1fn_x2), s2, None, K,
                               "swigluoai", E, mxfp4_activations=planes)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    ids = torch.stack([torch.randperm(E, generator=g)[:K] for _ in range(T)]).int().to(DEV)
    w = torch.full((T, K), 1.0 / K, device=DEV)
    out, one = torch.empty_like(x), torch.empty_like(x[:1])
    layer.apply(out, x, w, ids)
    for t in (0, T - 1):
        layer.apply(one, x[t:t + 1].contiguous(), w[t:t + 1].contiguous(), ids[t:t + 1].contiguous())
        assert torch.equal(one[0], out[t])
