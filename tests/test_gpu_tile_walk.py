"""The grouped GEMMs' walk over ragged segments where most experts have no rows: compacted
prefix sums (256 experts per scan step), bisection for steps over several experts, tiles with
one and with several token tiles.  Against the plain-CUDA checking kernel."""
import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,live", [(1, 1), (255, 3), (257, 257), (1024, 40), (1024, 1)])
@pytest.mark.parametrize("most", [1, 70])
def test_sparse_segments_16bit(native, E, live, most):
    g = torch.Generator().manual_seed(E + live + most)
    rows = torch.zeros(E, dtype=torch.int32)
    rows[torch.randperm(E, generator=g)[:live]] = torch.randint(1, most + 1, (live,), generator=g, dtype=torch.int32)
    M, N, K = int(rows.sum()), 256, 128
    x = (torch.randn(M, K, generator=g)).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E, K, N, generator=g) * K ** -0.5).to(torch.bfloat16).to(DEV)
    out = [torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    for o, impl in zip(out, (0, 2)):
        torch.ops._xpu_C.b200_grouped_gemm(x, None, w, None, None, o, rows.to(DEV), N, K, E, impl=impl)
    torch.testing.assert_close(out[0].float(), out[1].float(), rtol=2e-2, atol=2e-2)
