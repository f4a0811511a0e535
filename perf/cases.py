"""Timing cases of the fused-MoE layer: what a serving program asks of it, from one decoded token
to a full prefill batch, through the calls such a program makes.

A layer pass is routing (``topk_softmax`` or ``grouped_topk``), where the program does it itself
the activation quantisation, and ``XpuFusedMoe.apply`` into the program's own output buffer.  An
operator pass is the sequence a program runs around grouped GEMMs of its own: top-k,
``moe_align_block_size``, ``silu_and_mul``, ``per_token_group_fp8_quant`` and ``moe_sum``.

The layer shapes are the benchmark configurations of this repository (``bench.py``) and one
generic layer of many small 16-bit experts.  Inputs and weights are made on the GPU from the
seed: activations and router logits N(0, 1), weights N(0, 1/fan_in) quantised per recipe, biases
N(0, 0.02); skewed routing adds 1.5 log(1/rank) per expert, a Zipf-like expert load.
"""
import math
import os
import sys

import torch

# The package of the tree this runs in (the working folder is its root).
_PKG = os.path.abspath("vllm-xpu-kernels_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
from vllm_xpu_kernels.fused_moe_interface import XpuFusedMoe  # noqa: E402  registers the operators
from vllm_xpu_kernels.moe_utils import quant_fp8_block_act  # noqa: E402

# hidden size, intermediate size, experts, experts per token, routing, activation, biases
SHAPES = {
    "tiny": dict(hidden=1024, inter=2048, experts=8, topk=2, routing="softmax", activation="silu", bias=False),
    "fine": dict(hidden=2048, inter=1024, experts=64, topk=6, routing="softmax", activation="silu", bias=False),
    "mixtral": dict(hidden=4096, inter=14336, experts=8, topk=2, routing="softmax", activation="silu", bias=False),
    "gptoss": dict(hidden=2880, inter=2880, experts=128, topk=4, routing="softmax", activation="swigluoai",
                   bias=True),
    "deepseek": dict(hidden=7168, inter=2048, experts=256, topk=8, routing="grouped", activation="silu", bias=False),
}
# recipes each shape is served with, and its largest batch
RECIPES = {
    "tiny": (("bf16", "fp16", "fp8block"), 8192),
    "fine": (("bf16", "fp16"), 8192),
    "mixtral": (("bf16", "fp8block", "fp8pow2"), 4096),
    "gptoss": (("mxfp4",), 8192),
    "deepseek": (("fp8block", "fp8pow2"), 16384),
}
N_GROUP, TOPK_GROUP, ROUTED_SCALE = 8, 4, 2.5   # of the grouped routing


def _layer(shape, recipe, tokens, skew=False, quantised=False, ep_size=1, ep_rank=0, **more):
    return dict(kind="layer", shape=shape, recipe=recipe, tokens=tokens, skew=skew, quantised=quantised,
                ep_size=ep_size, ep_rank=ep_rank, **more)


def listed():
    return [
        # a small 16-bit layer on a small batch: launches and latency
        _layer("tiny", "bf16", 64, name="tiny_bf16_t64"),
        # decode of one sequence through a layer of many small experts
        _layer("fine", "bf16", 1, name="fine_bf16_t1"),
        # prefill of a ragged batch through the same layer
        _layer("fine", "bf16", 3001, name="fine_bf16_t3001"),
        # decode of a few sequences, every large expert hit by a few rows
        _layer("mixtral", "fp8block", 16, name="mixtral_fp8_t16"),
        # prefill, large experts: the benchmark's second configuration
        _layer("mixtral", "fp8block", 4096, quantised=True, name="mixtral_fp8_t4096"),
        # decode with 4-bit weights
        _layer("gptoss", "mxfp4", 1, name="gptoss_mxfp4_t1"),
        # prefill with 4-bit weights: the third configuration
        _layer("gptoss", "mxfp4", 8192, name="gptoss_mxfp4_t8192"),
        # decode of one sequence and of a batch with skewed expert load: the decode sweep
        _layer("deepseek", "fp8block", 1, skew=True, name="deepseek_fp8_t1"),
        _layer("deepseek", "fp8block", 128, skew=True, name="deepseek_fp8_t128"),
        # one rank of eight of an expert-parallel group that all see the same odd batch;
        # power-of-two block scales
        _layer("deepseek", "fp8pow2", 4099, ep_size=8, ep_rank=3, name="deepseek_pow2_ep8_t4099"),
        # a full prefill batch, activations quantised by the program: the benchmark's headline
        _layer("deepseek", "fp8block", 16384, quantised=True, name="deepseek_fp8_t16384"),
        # the single operators around a program's own GEMMs
        dict(kind="ops", shape="fine", tokens=4096, name="ops_t4096"),
    ]


def draw(rng):
    shape = rng.choice(sorted(SHAPES) + ["deepseek", "ops"])
    if shape == "ops":
        shape = rng.choice(["tiny", "fine", "gptoss"])
        return dict(kind="ops", shape=shape, tokens=_log_int(rng, 4096))
    recipes, most = RECIPES[shape]
    recipe = rng.choice(recipes)
    ep_size = rng.choice((1, 1, 1, 8)) if shape in ("gptoss", "deepseek") else 1
    return _layer(shape, recipe, _log_int(rng, most), skew=rng.random() < 0.5,
                  quantised=recipe.startswith("fp8") and rng.random() < 0.5, ep_size=ep_size,
                  ep_rank=rng.randrange(ep_size))


def _log_int(rng, most):
    return max(1, min(most, round(math.exp(rng.uniform(0.0, math.log(most))))))


# ---- inputs --------------------------------------------------------------------------

def _expert_chunks(E, K, N):
    step = max(1, (1 << 28) // (K * N))
    for e in range(0, E, step):
        yield e, min(E, e + step)


def _fp8_weights(E, K, N, g, pow2):
    """[E, K, N] e4m3 with fp32 scales per 128x128 block, rounded up to powers of two if asked."""
    q = torch.empty(E, K, N, dtype=torch.float8_e4m3fn, device="cuda")
    s = torch.empty(E, K // 128, N // 128, device="cuda")
    for a, b in _expert_chunks(E, K, N):
        w = torch.randn(b - a, K // 128, 128, N // 128, 128, generator=g, device="cuda").mul_(K ** -0.5)
        sc = (w.abs().amax(dim=(2, 4)) / 448.0).clamp_min(1e-12)
        if pow2:
            sc = torch.exp2(torch.ceil(torch.log2(sc)))
        w.div_(sc[:, :, None, :, None]).clamp_(-448, 448)
        q[a:b] = w.view(b - a, K, N).to(torch.float8_e4m3fn)
        s[a:b] = sc
    return q, s


def _mxfp4_weights(E, K, N, g):
    """[E, N, K/2] packed e2m1 with e8m0 scales per 32 values along K."""
    q = torch.empty(E, N, K // 2, dtype=torch.uint8, device="cuda")
    s = torch.empty(E, N, K // 32, dtype=torch.uint8, device="cuda")
    for a, b in _expert_chunks(E, K, N):
        w = torch.randn(b - a, N, K // 32, 32, generator=g, device="cuda").mul_(K ** -0.5)
        e = torch.ceil(torch.log2(w.abs().amax(-1).clamp_min(1e-30) / 6.0)).clamp(-127, 127)
        w.mul_(torch.exp2(-e).unsqueeze(-1))
        mag = w.abs()
        code = torch.zeros(w.shape, dtype=torch.uint8, device="cuda")
        for bound in (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0):
            code += mag > bound
        code |= (w < 0).to(torch.uint8) << 3
        code = code.view(b - a, N, K)
        q[a:b] = (code[..., 1::2] << 4) | code[..., 0::2]
        s[a:b] = (e + 127).to(torch.uint8)
    return q.view(torch.float4_e2m1fn_x2), s


def _weights(recipe, E, K, N, g, dtype):
    if recipe in ("fp8block", "fp8pow2"):
        return _fp8_weights(E, K, N, g, recipe == "fp8pow2")
    if recipe == "mxfp4":
        return _mxfp4_weights(E, K, N, g)
    w = torch.empty(E, K, N, dtype=dtype, device="cuda")
    for a, b in _expert_chunks(E, K, N):
        w[a:b] = torch.randn(b - a, K, N, generator=g, device="cuda").mul_(K ** -0.5)
    return w, None


def _logits(case, E, g):
    x = torch.randn(case["tokens"], E, generator=g, device="cuda")
    if case.get("skew"):
        x += _skew(E)
    return x


def _skew(E, device="cuda"):
    rank = torch.randperm(E, generator=torch.Generator().manual_seed(1)) + 1
    return (1.5 * torch.log(1.0 / rank.float())).to(device)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return _prepare_ops(case, g) if case["kind"] == "ops" else _prepare_layer(case, g)


def _prepare_layer(case, g):
    c = SHAPES[case["shape"]]
    T, H, I, E, k = case["tokens"], c["hidden"], c["inter"], c["experts"], c["topk"]
    E_loc = E // case["ep_size"]
    dtype = torch.float16 if case["recipe"] == "fp16" else torch.bfloat16
    w13, s13 = _weights(case["recipe"], E_loc, H, 2 * I, g, dtype)
    w2, s2 = _weights(case["recipe"], E_loc, I, H, g, dtype)
    b13 = b2 = None
    if c["bias"]:
        b13 = torch.randn(E_loc, 2 * I, generator=g, device="cuda").mul_(0.02).to(torch.bfloat16)
        b2 = torch.randn(E_loc, H, generator=g, device="cuda").mul_(0.02).to(torch.bfloat16)
    moe = XpuFusedMoe(w13, s13, b13, w2, s2, b2, k, c["activation"], E_loc, ep_rank=case["ep_rank"],
                      ep_size=case["ep_size"])
    state = dict(moe=moe, routing=c["routing"], topk=k, quantised=case["quantised"],
                 x=torch.randn(T, H, generator=g, device="cuda").to(dtype), logits=_logits(case, E, g),
                 out=torch.empty(T, H, dtype=dtype, device="cuda"))
    if c["routing"] == "grouped":
        state["score_bias"] = torch.randn(E, generator=g, device="cuda").mul_(0.01)
    return state


def _prepare_ops(case, g):
    c = SHAPES[case["shape"]]
    T, H, I, E, k = case["tokens"], c["hidden"], c["inter"], c["experts"], c["topk"]
    numel, block = T * k, 64
    padded = numel + E * (block - 1)
    d16 = dict(dtype=torch.bfloat16, device="cuda")
    d32 = dict(dtype=torch.int32, device="cuda")
    width = I // 128 * 128
    return dict(ops=True, logits=_logits(case, E, g), experts=E, topk=k, block=block,
                gate_up=torch.randn(numel, 2 * width, generator=g, device="cuda").to(torch.bfloat16),
                rows=torch.randn(T, k, H, generator=g, device="cuda").to(torch.bfloat16),
                act=torch.empty(numel, width, **d16),
                act_q=torch.empty(numel, width, dtype=torch.float8_e4m3fn, device="cuda"),
                act_s=torch.empty(numel, width // 128, device="cuda"),
                sorted_ids=torch.zeros(padded, **d32), expert_ids=torch.zeros(-(-padded // block), **d32),
                post_pad=torch.zeros(1, **d32), out=torch.empty(T, H, **d16))


# ---- one pass ------------------------------------------------------------------------

def _topk_softmax(logits, k):
    T = logits.shape[0]
    w = torch.empty(T, k, dtype=torch.float32, device=logits.device)
    ids = torch.empty(T, k, dtype=torch.int32, device=logits.device)
    src = torch.empty(T, k, dtype=torch.int32, device=logits.device)
    torch.ops._moe_C.topk_softmax(w, ids, src, logits, True, None, None)
    return w, ids


def run(state):
    return _run_ops(state) if "ops" in state else _run_layer(state)


def _run_layer(s):
    moe, x, scales = s["moe"], s["x"], None
    if s["routing"] == "grouped":
        w, ids = torch.ops._moe_C.grouped_topk(s["logits"], N_GROUP, TOPK_GROUP, s["topk"], True, ROUTED_SCALE,
                                               s["score_bias"], 1)
    else:
        w, ids = _topk_softmax(s["logits"], s["topk"])
    if s["quantised"]:
        x, scales = quant_fp8_block_act(x, moe.act_scales_pow2)
    moe.apply(s["out"], x, w, ids, a1q_scale=scales)
    return dict(out=s["out"], weights=w, ids=ids)


def _run_ops(s):
    w, ids = _topk_softmax(s["logits"], s["topk"])
    torch.ops._moe_C.moe_align_block_size(ids, s["experts"], s["block"], s["sorted_ids"], s["expert_ids"],
                                          s["post_pad"], None)
    torch.ops._C.silu_and_mul(s["act"], s["gate_up"])
    torch.ops._C.per_token_group_fp8_quant(s["act"], s["act_q"], s["act_s"], 128, 1e-10, -448.0, 448.0, False,
                                           False, False)
    torch.ops._moe_C.moe_sum(s["rows"], s["out"], None, None)
    keys = ("act", "act_q", "act_s", "sorted_ids", "expert_ids", "post_pad", "out")
    return dict({key: s[key] for key in keys}, weights=w, ids=ids)


# ---- what a pass cannot do without ---------------------------------------------------

def _experts_hit(case, E, E_loc, k):
    """Local experts that get a row, of a simulated batch (beyond 512 tokens: no more)."""
    if case["tokens"] * k >= 64 * E and not case["skew"]:
        return E_loc
    logits = torch.randn(min(case["tokens"], 512), E, generator=torch.Generator().manual_seed(0))
    if case["skew"]:
        logits += _skew(E, "cpu")
    ids = logits.topk(k, dim=1).indices.unique()
    first = E_loc * case["ep_rank"]
    return max(1, int(((ids >= first) & (ids < first + E_loc)).sum()))


def work(case):
    c = SHAPES[case["shape"]]
    T, H, I, E, k = case["tokens"], c["hidden"], c["inter"], c["experts"], c["topk"]
    route = T * E * 4 + T * k * 8
    if case["kind"] == "ops":
        width = I // 128 * 128
        align = T * k * 4 + (T * k + E * 63) * 4
        act = T * k * (2 * width * 2 + width * 2)
        quant = T * k * (width * 2 + width + width // 128 * 4)
        return {"bytes": route + align + act + quant + T * (k + 1) * H * 2, "flops": 0}
    per_weight = {"bf16": 2.0, "fp16": 2.0, "fp8block": 1.0, "fp8pow2": 1.0, "mxfp4": 0.5 + 1 / 32}[case["recipe"]]
    hit = _experts_hit(case, E, E // case["ep_size"], k)
    return {"bytes": route + hit * 3 * H * I * per_weight + 2 * T * H * 2,
            "flops": 6.0 * T * k * H * I / case["ep_size"]}


def tolerance(case):
    if case["kind"] == "ops":
        # SiLU and sums in fp32 rounded to bf16; e4m3 codes and indices follow the same rounding
        return {"rel": 4e-3, "differ": 0.0}
    # bf16 outputs of fp32 sums; with quantised recipes a sum in another order can move a value
    # of the intermediate activation to the neighbouring code.  Expert ids are exact.
    return {"rel": 1e-2, "differ": 0.0}
