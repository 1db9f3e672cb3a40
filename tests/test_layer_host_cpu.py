"""CPU: host-side decisions of the layer object (no kernel runs: the object is built around CPU
tensors and only asked which form a call of a given size would take)."""
import copy
import pickle

import pytest
import torch

from oracle import workloads as wl


def _layer(native, cfg_name, dims, **kw):
    import vllm_xpu_kernels.fused_moe_interface as fmi
    cfg = wl.scaled(wl.CONFIGS[cfg_name], **dims)
    w = wl.make_weights(cfg, seed=0)
    w13, s13, w2, s2 = wl.to_op_layout(cfg, w)
    return cfg, fmi.XpuFusedMoe(w13, s13, w["w13_bias"], w2, s2, w["w2_bias"], cfg.K, cfg.activation, cfg.E, **kw)


def test_which_calls_fuse_the_activation_into_gemm1(native):
    rows = lambda layer, per_expert: layer.fuses_activation(per_expert * layer.num_experts)
    # 16-bit, SiLU, whole 128-feature tiles: fused at every size (one CTA up to 128-token tiles, a CTA pair beyond)
    _, bf16 = _layer(native, "cfg1_small_bf16", dict(H=256, I=256, E=4))
    assert [rows(bf16, r) for r in (1, 96, 97, 5000)] == ["epilogue"] * 4
    # ... other intermediate sizes: only where 128-token tiles are picked anyway
    _, odd = _layer(native, "cfg1_small_bf16", dict(H=256, I=208, E=4))
    assert [rows(odd, r) for r in (1, 96, 97, 5000)] == ["epilogue", "epilogue", None, None]
    _, off = _layer(native, "cfg1_small_bf16", dict(H=256, I=256, E=4), fuse_activation=False)
    assert rows(off, 8) is None
    # block-scaled fp8, SiLU: two kernels are never slower, so the fused form only on request
    _, fp8 = _layer(native, "cfg4_deepseek_fp8", dict(H=256, I=256, E=8))
    assert [rows(fp8, r) for r in (1, 511, 512, 4096)] == [None] * 4
    _, forced = _layer(native, "cfg4_deepseek_fp8", dict(H=256, I=256, E=8), fuse_activation=True)
    assert [rows(forced, r) for r in (11, 12)] == [None, "fp8"]
    # a hint about the rows actually in use (expert parallelism: buffers sized for the worst case) decides
    forced.rows_hint = 12 * forced.num_experts
    assert forced.fuses_activation(100 * 12 * forced.num_experts) == "fp8" and rows(forced, 1) == "fp8"
    forced.rows_hint = 11 * forced.num_experts
    assert rows(forced, 100) is None
    # MXFP4 with SwigluOAI: always in the epilogue
    _, mx = _layer(native, "cfg5_gptoss_mxfp4", dict(H=256, I=256, E=4))
    assert [rows(mx, r) for r in (1, 4096)] == ["epilogue"] * 2


def test_recipes_that_cannot_take_prequantised_inputs_say_so(native):
    _, bf16 = _layer(native, "cfg1_small_bf16", dict(H=256, I=256, E=4))
    x = torch.zeros(2, 256, dtype=torch.bfloat16)
    with pytest.raises(NotImplementedError):
        bf16.apply(torch.empty_like(x), x, torch.ones(2, 2), torch.zeros(2, 2, dtype=torch.int32),
                   a1q_scale=torch.ones(2, 2))


def test_a_used_layer_can_be_copied_and_saved(native):
    """The native plan of a layer that has been called stays behind: a copy makes its own, from its own tensors."""
    _, layer = _layer(native, "cfg1_small_bf16", dict(H=256, I=256, E=4))
    plan = layer._plan()
    for other in (copy.copy(layer), copy.deepcopy(layer), pickle.loads(pickle.dumps(layer))):
        assert layer._native_plan is plan
        assert other._native_plan is None and other._plan() is not plan
        assert torch.equal(other.w13, layer.w13) and other.recipe == layer.recipe


def test_a_layer_names_its_activation_op(native):
    _, layer = _layer(native, "cfg1_small_bf16", dict(H=256, I=256, E=4))
    assert layer.act_func is torch.ops._C.silu_and_mul
    with pytest.raises(AttributeError):
        layer.act_func = torch.ops._C.gelu_and_mul
