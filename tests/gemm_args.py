"""ctypes mirror of b200moe_gemm_args (include/b200moe.h); test_abi_cpu.py holds it against the compiler's layout."""
import ctypes as ct

_P, _I, _L, _F = ct.c_void_p, ct.c_int, ct.c_int64, ct.c_float


class GemmArgs(ct.Structure):
    _fields_ = [("a", _P), ("a_dtype", _I), ("a_scale", _P), ("w", _P), ("w_format", _I), ("w_scale", _P), ("bias", _P),
                ("d", _P), ("d_dtype", _I), ("rows_per_expert", _P), ("m", _L), ("n", _I), ("k", _I), ("num_experts", _I),
                ("epilogue", _I), ("act_alpha", _F), ("act_limit", _F), ("clamp_limit", _F), ("status", _P), ("impl", _I),
                ("max_ctas", _I), ("group_size", _I), ("w_experts", _I), ("d_scale", _P), ("mid_dtype", _I),
                ("rows_ready", _I), ("rows_hint", _L)]
