"""The layer's SiLU, multiply and 1x128 e4m3 quantisation (rows in use given by segments): value for value what
silu_and_mul_per_block_quant gives, for widths of a half and of several pieces of 256, row counts from none to
several passes of a full grid, and groups with infinities, NaN, zeros, subnormals and the type's extremes."""
import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,extra,hidden", [(0, 3, 128), (1, 0, 128), (7, 2, 384), (33, 0, 768), (1000, 100, 2048), (5000, 1, 128),
                                               (20001, 0, 256)])
def test_rows_as_the_op_gives_them(native, rows, extra, hidden, dtype):
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows + extra, 2 * hidden, generator=g) * torch.exp2(torch.randint(-20, 6, (rows + extra, 1), generator=g).float())
    x = x.to(dtype)
    info = torch.finfo(dtype)
    for i, v in enumerate([float("inf"), -float("inf"), float("nan"), 0.0, info.smallest_normal / 4, info.max, info.min, 100.0, -100.0]):
        if i < rows:
            x[i, 0], x[i, hidden + 1] = v, v
            x[i, 100:128] = v if i in (3, 4) else x[i, 100:128]
    if rows > 12:
        x[10] = 0
        x[11, :hidden] = info.min
        x[12, hidden:] = info.max
    x = x.to(DEV)
    seg = torch.tensor([rows // 3, 0, rows - rows // 3, -5], dtype=torch.int32, device=DEV)
    q = torch.full((rows + extra, hidden), 7, dtype=torch.uint8, device=DEV).view(torch.float8_e4m3fn)
    s = torch.full((rows + extra, hidden // 128), 7.0, device=DEV)
    torch.ops._C.b200_silu_and_mul_block_quant_rows(q, x, s, seg)
    assert (q.view(torch.uint8)[rows:] == 7).all() and (s[rows:] == 7).all()   # rows not in use stay as they are
    if rows:
        oq = torch.empty(rows, hidden, dtype=torch.float8_e4m3fn, device=DEV)
        os_ = torch.empty(rows, hidden // 128, device=DEV)
        torch.ops._C.silu_and_mul_per_block_quant(oq, x[:rows].contiguous(), os_, 128, None, False, False)
        assert torch.equal(q.view(torch.uint8)[:rows], oq.view(torch.uint8))
        assert torch.equal(s[:rows].view(torch.int32), os_.view(torch.int32))
        # ... which is SiLU times the other half, in the group's scale: against 64 bits, groups without special values
        gate, up = x[:rows].double().split(hidden, 1)
        v = (gate * torch.sigmoid(gate) * up).view(rows, -1, 128)
        top = v.abs().amax(-1)
        # (above the smallest scale, 448 / (448 * 512); gates below 32, whose product with log2 e is off by 2^-20 at most)
        plain = (top < 2.0 ** 100) & (top > 2 ** -8) & (gate.view(rows, -1, 128).abs().amax(-1) < 32)
        if plain.any():
            assert (s[:rows].double()[plain] / (top[plain] / 448) - 1).abs().max() < 1e-5
        back = q[:rows].double().view(rows, -1, 128) * s[:rows].double().unsqueeze(-1)
        # half a step of e4m3, 2^-4 of a value, or of the smallest step 2^-9 scales, and a few ulp before the rounding
        err = (back - v).abs() - (2 ** -4 + 1e-4) * v.abs() - 2 ** -10 * s[:rows].double().unsqueeze(-1) * 1.01
        assert (err[plain] <= 0).all()
