"""Performance cases of the fused Mixture-of-Experts layer.

One pass is what a serving program does for every MoE layer of every forward step: it routes
the router's output with one of the registered top-k ops and hands ids and weights to
``XpuFusedMoe.apply``.  The cases go over the layers of the benchmark table
(``bench_workloads.CONFIGS``) from one decoded token to a full prefill batch, an int4 layer of
one of these shapes, and one rank's share of an expert-parallel layer.

Inputs are seeded synthetic draws with the distributions the benchmark states: hidden states
and router logits ~N(0,1), weights ~N(0,1/fan_in) in the layer's storage format.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "vllm-xpu-kernels_b200"))

import vllm_xpu_kernels.fused_moe_interface as fmi  # noqa: E402

# family -> the fixed properties of its layers.  `experts` are the routed experts of the whole
# layer; one process holds experts / ep of them.
FAMILIES = {
    # the small CPU-runnable layer and other small 16-bit layers of its kind
    "small": dict(recipe="w16", hidden=2048, inter=1408, experts=8, topk=2),
    # a few large 16-bit experts, uneven load
    "mixtral": dict(recipe="w16", hidden=4096, inter=14336, experts=8, topk=2, skew=0.5),
    # the same layer with int4 weights and 16-bit scales per 128 values
    "mixtral_int4": dict(recipe="int4", hidden=4096, inter=14336, experts=8, topk=2, skew=0.5),
    # many small experts, fp8 weights with a scale per 128x128 block
    "qwen3": dict(recipe="fp8", hidden=2048, inter=768, experts=128, topk=8),
    # many large experts, fp8 block-scaled, grouped sigmoid routing
    "deepseek": dict(recipe="fp8", hidden=7168, inter=2048, experts=256, topk=8, groups=8, topk_group=4, scale=2.5),
    # one of eight ranks of that layer: 32 experts, the tokens' other experts masked
    "deepseek_ep8": dict(recipe="fp8", hidden=7168, inter=2048, experts=256, topk=8, groups=8, topk_group=4, scale=2.5,
                         ep=8),
    # MXFP4 weights, SwigluOAI with biases
    "gptoss": dict(recipe="mxfp4", hidden=2880, inter=2880, experts=128, topk=4, act="swigluoai"),
}
LARGEST = {"small": 8192, "mixtral": 4096, "mixtral_int4": 2048, "qwen3": 16384, "deepseek": 8192, "deepseek_ep8": 8192,
           "gptoss": 4096}
EP_RANK = 3


def _case(family, tokens, **other):
    f = FAMILIES[family]
    c = dict(family=family, tokens=tokens, hidden=f["hidden"], inter=f["inter"], experts=f["experts"], topk=f["topk"],
             dtype="bfloat16")
    c.update(other)
    return c


def listed():
    return [
        # a small layer with a small decode batch: launches and latency
        dict(_case("small", 64), name="small_bf16_t64"),
        # one user decoding: two experts' weights stream through
        dict(_case("mixtral", 1), name="mixtral_bf16_t1"),
        # a prefill batch on a few large experts: tensor-core work
        dict(_case("mixtral", 4096), name="mixtral_bf16_t4096"),
        # a decode batch on 4-bit weights with 16-bit activations
        dict(_case("mixtral_int4", 33), name="mixtral_int4_t33"),
        # a small decode batch over many small experts
        dict(_case("qwen3", 16), name="qwen3_fp8_t16"),
        # a mixed prefill batch of ragged size over many small experts
        dict(_case("qwen3", 3001), name="qwen3_fp8_t3001"),
        # a decode batch that touches most of 256 large experts
        dict(_case("deepseek", 64), name="deepseek_fp8_t64"),
        # the largest prefill batch of the benchmark
        dict(_case("deepseek", 8192), name="deepseek_fp8_t8192"),
        # one expert-parallel rank: all tokens of the group arrive, an eighth of the slots are local
        dict(_case("deepseek_ep8", 1024), name="deepseek_fp8_ep8_t1024"),
        # one user decoding on 4-bit experts: the shortest weight stream
        dict(_case("gptoss", 1), name="gptoss_mxfp4_t1"),
        # a decode batch of many users
        dict(_case("gptoss", 128), name="gptoss_mxfp4_t128"),
        # a prefill batch
        dict(_case("gptoss", 2048), name="gptoss_mxfp4_t2048"),
    ]


def draw(rng):
    """A layer family with a token count spread over its range on a logarithmic scale; small
    layers also in other sizes and 16-bit weights in both 16-bit types."""
    family = rng.choice(sorted(FAMILIES))
    tokens = int(round(math.exp(rng.uniform(0.0, math.log(LARGEST[family])))))
    other = {}
    if FAMILIES[family]["recipe"] in ("w16", "int4"):
        other["dtype"] = rng.choice(["bfloat16", "float16"])
    if family == "small":
        other.update(hidden=rng.choice([512, 1024, 2048, 3072]), inter=rng.choice([256, 704, 1408, 1536, 2048]),
                     experts=rng.choice([8, 16, 32, 60]), topk=rng.choice([1, 2, 4, 6]))
    return _case(family, tokens, **other)


def _fp8_blocks(g, experts, n, k):
    """[experts, n, k] e4m3 weights drawn from N(0, 1/k) and their scale per 128x128 block."""
    q = torch.empty(experts, n, k, dtype=torch.float8_e4m3fn, device="cuda")
    s = torch.empty(experts, n // 128, k // 128, dtype=torch.float32, device="cuda")
    for e in range(experts):
        w = torch.randn(n // 128, 128, k // 128, 128, generator=g, device="cuda").mul_(k ** -0.5)
        top = w.abs().amax(dim=(1, 3), keepdim=True).div_(448.0)
        q[e] = w.div_(top).view(n, k).to(torch.float8_e4m3fn)
        s[e] = top.view(n // 128, k // 128)
    return q, s


def _w16(g, experts, k, n, dtype):
    w = torch.empty(experts, k, n, dtype=dtype, device="cuda")
    for e in range(experts):
        w[e] = torch.randn(k, n, generator=g, device="cuda").mul_(k ** -0.5)
    return w


def _int4(g, experts, n, k, dtype):
    """Two uint4 codes a byte (zero point 8) of N(0, 1/k) weights, scale per 128 values."""
    q = torch.empty(experts, n, k // 2, dtype=torch.uint8, device="cuda")
    for e in range(experts):
        c = torch.randn(n, k // 2, 2, generator=g, device="cuda").mul_(2.5).round_().clamp_(-8, 7).add_(8).to(torch.uint8)
        q[e] = c[..., 0] | (c[..., 1] << 4)
    s = torch.empty(experts, n, k // 128, device="cuda").uniform_(0.3, 0.5, generator=g).mul_(k ** -0.5).to(dtype)
    return q, s


def prepare(case, seed):
    f = FAMILIES[case["family"]]
    T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "inter", "experts", "topk"))
    dtype = getattr(torch, case["dtype"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    ep = f.get("ep", 1)
    L = E // ep
    s13 = s2 = b13 = b2 = None
    if f["recipe"] == "w16":
        w13, w2 = _w16(g, L, H, 2 * I, dtype), _w16(g, L, I, H, dtype)
    elif f["recipe"] == "int4":
        w13, s13 = _int4(g, L, 2 * I, H, dtype)
        w2, s2 = _int4(g, L, H, I, dtype)
    elif f["recipe"] == "fp8":
        w13, s13 = _fp8_blocks(g, L, 2 * I, H)
        w2, s2 = _fp8_blocks(g, L, H, I)
    else:  # uniform e2m1 codes, e8m0 exponents in [-10, -4], biases ~N(0, 0.02)
        def some(lo, hi, *shape):
            return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=torch.uint8)
        w13 = some(0, 256, L, 2 * I, H // 2).view(torch.float4_e2m1fn_x2)
        w2 = some(0, 256, L, H, I // 2).view(torch.float4_e2m1fn_x2)
        s13, s2 = some(117, 124, L, 2 * I, H // 32), some(117, 124, L, H, I // 32)
        b13 = (torch.randn(L, 2 * I, generator=g, device="cuda") * 0.02).to(dtype)
        b2 = (torch.randn(L, H, generator=g, device="cuda") * 0.02).to(dtype)
    layer = fmi.XpuFusedMoe(w13, s13, b13, w2, s2, b2, K, f.get("act", "silu"), L,
                            ep_rank=EP_RANK if ep > 1 else 0, ep_size=ep)
    state = dict(layer=layer, topk=K, f=f, x=torch.randn(T, H, generator=g, device="cuda").to(dtype),
                 out=torch.empty(T, H, dtype=dtype, device="cuda"))
    logits = torch.randn(T, E, generator=g, device="cuda")
    if f.get("skew"):
        logits += torch.randn(E, generator=g, device="cuda") * f["skew"]
    if "groups" in f:  # the router hands over its sigmoid scores, plain and with the balancing bias
        state["scores"] = torch.sigmoid(logits)
        state["biased"] = state["scores"] + torch.randn(E, generator=g, device="cuda") * 0.1
    else:
        state["logits"] = logits
        state["weights"] = torch.empty(T, K, dtype=torch.float32, device="cuda")
        state["ids"] = torch.empty(T, K, dtype=torch.int32, device="cuda")
        state["source"] = torch.empty(T, K, dtype=torch.int32, device="cuda")
    return state


def run(s):
    f = s["f"]
    if "groups" in f:
        weights, ids = torch.ops._moe_C.grouped_topk(s["scores"], s["biased"], f["groups"], f["topk_group"], s["topk"],
                                                     True, f["scale"])
    else:
        weights, ids = s["weights"], s["ids"]
        torch.ops._moe_C.topk_softmax(weights, ids, s["source"], s["logits"], True, None)
    s["layer"].apply(s["out"], s["x"], weights, ids)
    return {"out": s["out"], "weights": weights, "ids": ids}


def _routed(case, f):
    """Experts of this process that one draw of the case's routing reaches, and the routed rows they get."""
    T, E, K = case["tokens"], case["experts"], case["topk"]
    g = torch.Generator().manual_seed(1)
    scores = torch.randn(T, E, generator=g)
    if f.get("skew"):
        scores += torch.randn(E, generator=g) * f["skew"]
    if "groups" in f:
        scores = torch.sigmoid(scores) + torch.randn(E, generator=g) * 0.1
        best = scores.view(T, f["groups"], -1).topk(2, dim=-1).values.sum(-1)
        kept = torch.zeros_like(best).scatter_(1, best.topk(f["topk_group"], dim=-1).indices, 1.0)
        scores = scores * kept.repeat_interleave(E // f["groups"], dim=1)
    ids = scores.topk(K, dim=-1).indices
    local = E // f.get("ep", 1)
    rows = torch.bincount(ids.flatten(), minlength=E).view(-1, local)[EP_RANK if f.get("ep", 1) > 1 else 0]
    return int((rows > 0).sum()), int(rows.sum())


def work(case):
    """Router scores and hidden states read, the weights of the experts that are active read,
    output, ids and routing weights written; two multiplications of every routed row."""
    f = FAMILIES[case["family"]]
    T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "inter", "experts", "topk"))
    active, rows = _routed(case, f)
    n = 3 * H * I
    each = {"w16": 2 * n, "fp8": n + 4 * n // 16384, "int4": n // 2 + 2 * n // 128,
            "mxfp4": n // 2 + n // 32 + 2 * (2 * I + H)}[f["recipe"]]
    scores = (2 if "groups" in f else 1) * 4 * T * E
    return {"bytes": active * each + 4 * T * H + scores + 8 * T * K, "flops": 6.0 * rows * H * I}


def tolerance(case):
    """16-bit rows between the stages everywhere; fp8 layers also round the rows of both
    multiplications to e4m3, where a rounding of the 16-bit value before it moves a few codes."""
    return {"rel": 2e-2 if FAMILIES[case["family"]]["recipe"] == "fp8" else 1e-2}
