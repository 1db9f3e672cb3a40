"""Token-major fp8 GEMM: a partly filled tile brings its rows in a box of 32, 64 or 96 rows and zeros in the box
behind it.  Last tiles of every height around the quarters, inside the matrix (the next segment's rows are NaN
codes) and at its end, plain and gated."""
import pytest
import torch

from gpu_utils import DEV, grouped_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129, 225])
def test_fp8_last_tile_heights(native, rows, gated, layout):
    N, K, counts = 512, 256, [rows, 40, rows]
    E, M = 3, sum(counts)
    g = torch.Generator().manual_seed(rows)
    w = (torch.randn(E, N, K, generator=g) * 20).to(torch.float8_e4m3fn)
    a = (torch.randn(M, K, generator=g) * 40).to(torch.float8_e4m3fn)
    a.view(torch.uint8)[rows:rows + 40] = 0x7f
    sa, sw = torch.rand(M, K // 128, generator=g) * 0.02, torch.rand(E, N // 128, K // 128, generator=g) * 0.02
    wd = (w if layout == 1 else w.transpose(1, 2).contiguous()).to(DEV)
    n_rows = torch.tensor(counts, dtype=torch.int32, device=DEV)
    live = torch.cat([torch.arange(rows), torch.arange(rows + 40, M)])
    af = a.double() * sa.double().repeat_interleave(128, 1)
    wf = w.double() * sw.double().repeat_interleave(128, 1).repeat_interleave(128, 2)
    ref = torch.cat([x @ wf[e].T for e, x in enumerate(af.split(counts))])[live]
    plain = grouped_gemm(a.to(DEV), sa.to(DEV), wd, sw.to(DEV), None, n_rows, N, K, layout=layout)
    out = plain[live.to(DEV)].cpu().double()
    # one rounding to bf16 and fp32 sums of K terms
    bound = 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * (af[live].abs() @ wf.abs().amax(0).T + 1)
    assert ((out - ref).abs() <= bound).all()
    if gated:   # the fused form is bit-exact with the plain one followed by the activation and quantisation
        q = torch.empty(M, N // 2, dtype=torch.float8_e4m3fn, device=DEV)
        qs = torch.empty(M, N // 256, dtype=torch.float32, device=DEV)
        torch.ops._xpu_C.b200_grouped_gemm(a.to(DEV), sa.to(DEV), wd, sw.to(DEV), None, q, n_rows, N, K, E, layout, 1, 1.702,
                                           7.0, 0.0, 0, 0, 0, qs, False)
        at = torch.empty(M, N // 2, dtype=torch.float8_e4m3fn, device=DEV)
        ats = torch.empty(M, N // 256, dtype=torch.float32, device=DEV)
        torch.ops._C.silu_and_mul_per_block_quant(at, plain, ats, 128, None, False, False)
        assert torch.equal(q.view(torch.uint8)[live.to(DEV)], at.view(torch.uint8)[live.to(DEV)])
        assert torch.equal(qs[live.to(DEV)], ats[live.to(DEV)])
