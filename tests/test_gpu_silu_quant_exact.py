"""SiLU, multiply and e4m3 quantisation against values that this repository's kernels have no part in: a group with one
value other than zero shows that value through its scale to fp32 precision, so SiLU itself is held against 64 bits for
every bfloat16 gate of a range, the division by 448 against float32's, and special values against the codes they must give."""
import pytest
import torch

from gpu_utils import DEV

pytestmark = pytest.mark.gpu


def _both(x):
    """(codes, scales) of the op and of the layer's rows kernel, which must agree."""
    rows, hidden = x.shape[0], x.shape[1] // 2
    outs = []
    for ragged in (False, True):
        q = torch.empty(rows, hidden, dtype=torch.float8_e4m3fn, device=DEV)
        s = torch.empty(rows, hidden // 128, device=DEV)
        if ragged:
            torch.ops._C.b200_silu_and_mul_block_quant_rows(q, x, s, torch.tensor([rows], dtype=torch.int32, device=DEV))
        else:
            torch.ops._C.silu_and_mul_per_block_quant(q, x, s, 128, None, False, False)
        outs.append((q.view(torch.uint8).cpu(), s.cpu()))
    (q, s), (q2, s2) = outs
    assert torch.equal(q, q2) and torch.equal(s.view(torch.int32), s2.view(torch.int32))
    return q, s


def _first_of_groups(gate, up, dtype):
    """Rows of one group of 128 whose first value is the given one and whose others are zero."""
    x = torch.zeros(gate.numel(), 256, dtype=dtype, device=DEV)
    x[:, 0], x[:, 128] = gate.to(DEV), up.to(DEV)
    return x


def test_silu_of_every_bfloat16_gate_against_64_bits(native):
    bits = torch.arange(0, 1 << 16, dtype=torch.int32).to(torch.int16)
    gate = bits.view(torch.bfloat16)
    gate = gate[(gate.float().abs() <= 100) & (gate.float().abs() >= 2.0 ** -100)]
    true = gate.double() * torch.sigmoid(gate.double())
    # a power of two that brings the product to [1, 2), as far as the type reaches
    up = torch.exp2((-torch.floor(torch.log2(true.abs()))).clamp(-120, 127)).to(torch.bfloat16)
    q, s = _both(_first_of_groups(gate, up, torch.bfloat16))
    want = true.abs() * up.double() / 448
    least = 1.0 / (448 * 512)
    zero = gate.double() < -87.4                 # the reciprocal of 1 + e^-g is subnormal: zero
    assert (s[zero, 0] == torch.tensor(least, dtype=torch.float32)).all() and (q[zero, 0] & 0x7f == 0).all()
    kept = ~zero & (gate.double() > -87.3)
    assert kept.sum() > 5000 and (want[kept] > least).all()
    # the rounded exponent's error, the two approximations and the roundings of the sum, the products and the quotient
    bound = 7.3e-8 * gate.double().abs() + 6e-7
    err = (s[:, 0].double() / want - 1).abs()
    print("worst error / bound", float((err / bound)[kept].max()))
    assert (err <= bound)[kept].all()
    assert ((q[kept, 0] & 0x7f) == 0x7e).all() and torch.equal(q[kept, 0] >= 128, (true < 0)[kept])


def test_scales_are_the_float32_quotients(native):
    """Gates of 32 and more are their own SiLU (e^-32 is far below half a unit of 1), so the product of two float16 is exact."""
    g = torch.Generator().manual_seed(1)
    n = 200000
    gate, up = ((torch.randint(1024, 2048, (n,), generator=g) / m).to(torch.float16) for m in (16, 64))   # [64, 128) and [16, 32)
    q, s = _both(_first_of_groups(gate, up, torch.float16))
    want = (gate.float() * up.float()) / torch.tensor(448.0)
    assert torch.equal(s[:, 0].view(torch.int32), want.view(torch.int32))
    assert (q[:, 0] == 0x7e).all() and (q[:, 1:] == 0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_codes_and_scales_of_special_values(native, dtype):
    """A NaN becomes 448 and does not count for the scale; an infinity takes the scale, and what it leaves is zero (the
    infinity itself times a zero reciprocal is a NaN: 448).  The lowest gates are a negative zero."""
    inf, nan, info = float("inf"), float("nan"), torch.finfo(dtype)
    least, one = 1.0 / (448 * 512), 64.0 / 448       # the scale beside a second value of 64 * 1
    # gate, up -> code of the value, scale of its group, code of the 64 beside it
    table = [(nan, 1.0, 0x7e, one, 0x7e), (1.0, nan, 0x7e, one, 0x7e), (inf, 1.0, 0x7e, inf, 0), (1.0, inf, 0x7e, inf, 0),
             (1.0, -inf, 0x7e, inf, 0), (-inf, 1.0, 0x7e, one, 0x7e), (0.0, inf, 0x7e, one, 0x7e), (0.0, 5.0, 0x00, one, 0x7e),
             (info.min, 1.0, 0x80, one, 0x7e), (info.min, -1.0, 0x00, one, 0x7e), (-100.0, 1.0, 0x80, one, 0x7e),
             (info.max, 1.0, 0x7e, info.max / 448, 0 if dtype == torch.bfloat16 else None)]
    gate, up = (torch.tensor([t[i] for t in table]).to(dtype) for i in (0, 1))
    x = _first_of_groups(gate, up, dtype)
    x[:, 1], x[:, 129] = 64.0, 1.0
    q, s = _both(x)
    for i, (a, b, code, scale, beside) in enumerate(table):
        assert q[i, 0] == code, (a, b, hex(int(q[i, 0])))
        assert s[i, 0] == torch.tensor(scale, dtype=torch.float32), (a, b, s[i, 0])
        assert beside is None or q[i, 1] == beside, (a, b, hex(int(q[i, 1])))
        assert (q[i, 2:] & 0x7f == 0).all()
    # ... and with nothing beside it
    q, s = _both(_first_of_groups(torch.tensor([nan, 0.0, info.min]).to(dtype), torch.ones(3).to(dtype), dtype))
    assert q[:, 0].tolist() == [0x7e, 0x00, 0x80] and (s == torch.tensor(least, dtype=torch.float32)).all()
