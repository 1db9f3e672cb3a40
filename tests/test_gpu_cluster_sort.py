"""remap_hidden_states where one cluster sorts the slots (2049 to 65536 of them, up to 360 experts) and on both sides of
its limits: positions and counts are those of a stable sort by expert, exactly."""
import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ids_dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("T,K,E", [(2048, 1, 8), (2049, 1, 1), (513, 4, 32), (1024, 8, 256), (1025, 8, 360), (1500, 6, 361),
                                   (3001, 8, 128), (7282, 9, 60), (8192, 8, 33), (65536, 1, 1), (8193, 8, 256)])
def test_positions_are_those_of_a_stable_sort(native, T, K, E, masked, ids_dtype):
    g = torch.Generator().manual_seed(T + E)
    # uneven: some experts get most of the slots, some none; a few ids that are no expert
    ids = (torch.rand(T, K, generator=g) ** 3 * E).long().clamp_(max=E - 1)
    ids[torch.rand(T, K, generator=g) < 0.01] = -1
    total = E
    emap = None
    if masked:
        total = 2 * E
        emap = torch.full((total,), -1, dtype=torch.int32)
        emap[torch.randperm(total, generator=g)[:E]] = torch.arange(E, dtype=torch.int32)
        ids = torch.where(ids >= 0, (ids * 2 + torch.randint(0, 2, (T, K), generator=g)), ids)
    bucket = ids.flatten().clone()
    if masked:
        bucket = torch.where(bucket >= 0, emap.long()[bucket.clamp(min=0)], bucket)
    live = (bucket >= 0).nonzero().flatten()
    order = live[torch.sort(bucket[live], stable=True).indices]
    want = torch.full((T * K,), -1, dtype=torch.int32)
    want[order] = torch.arange(order.numel(), dtype=torch.int32)
    H = 8
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    out = torch.zeros(T * K, H, dtype=torch.bfloat16, device=DEV)
    rows = torch.full((E,), -7, dtype=torch.int32, device=DEV)
    row_map = torch.full((T, K), -7, dtype=torch.int32, device=DEV)
    torch.ops._moe_C.remap_hidden_states(x, None, out, None, emap.to(DEV) if masked else None, rows, row_map,
                                         ids.to(ids_dtype).to(DEV), total, E)
    assert torch.equal(row_map.cpu().flatten(), want)
    assert torch.equal(rows.cpu().long(), torch.bincount(bucket[live], minlength=E))
    assert torch.equal(out[:order.numel()].cpu(), x.cpu()[order // K])


def test_captured_and_replayed_with_other_ids(native):
    T, K, E, H = 1024, 8, 64, 16
    g = torch.Generator().manual_seed(3)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    ids = torch.zeros(T, K, dtype=torch.int32, device=DEV)
    out = torch.empty(T * K, H, dtype=torch.bfloat16, device=DEV)
    rows, row_map = torch.empty(E, dtype=torch.int32, device=DEV), torch.empty(T, K, dtype=torch.int32, device=DEV)
    call = lambda: torch.ops._moe_C.remap_hidden_states(x, None, out, None, None, rows, row_map, ids, E, E)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for _ in range(2):
        new = torch.randint(0, E, (T, K), generator=g, dtype=torch.int32)
        ids.copy_(new)
        graph.replay()
        order = torch.sort(new.flatten(), stable=True).indices
        want = torch.empty(T * K, dtype=torch.int32)
        want[order] = torch.arange(T * K, dtype=torch.int32)
        assert torch.equal(row_map.cpu().flatten(), want)
        assert torch.equal(rows.cpu().long(), torch.bincount(new.flatten().long(), minlength=E))
