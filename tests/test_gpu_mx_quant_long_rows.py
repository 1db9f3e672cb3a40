"""MXFP8 quantiser, gated form: rows whose two halves together have 2^31 values and more."""
import ctypes as ct

import pytest
import torch

from conftest import PKG_DIR
from gpu_utils import DEV

pytestmark = pytest.mark.gpu


def _quantise(lib, x, rows, cols):
    q = torch.empty(rows, cols, dtype=torch.uint8, device=DEV)
    s = torch.empty((cols + 127) // 128, rows, dtype=torch.int32, device=DEV)
    rc = lib.b200moe_quant_mxfp8_ex(ct.c_void_p(x.data_ptr()), 2, ct.c_void_p(q.data_ptr()), ct.c_void_p(s.data_ptr()),
                                    ct.c_int64(rows), cols, 1, 0, 1, ct.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, lib.b200moe_last_error()
    return q, s


def test_second_row_of_long_gated_rows(native):
    lib = ct.CDLL(str(PKG_DIR / "vllm_xpu_kernels" / "libb200moe.so"))
    lib.b200moe_last_error.restype = ct.c_char_p
    rows, cols, n = 2, 1 << 30, 512
    x = torch.zeros(rows, 2, cols, dtype=torch.bfloat16, device=DEV)   # 8 GB
    ends = torch.randn(rows, 2, 2 * n, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    x[:, :, :n], x[:, :, -n:] = ends[:, :, :n], ends[:, :, n:]
    q, s = _quantise(lib, x, rows, cols)
    want_q, want_s = _quantise(lib, ends, rows, 2 * n)
    assert torch.equal(q[:, :n], want_q[:, :n]) and torch.equal(q[:, -n:], want_q[:, n:])
    assert torch.equal(s[:n // 128], want_s[:n // 128]) and torch.equal(s[-n // 128:], want_s[n // 128:])
    assert not q[:, n:-n].any()
