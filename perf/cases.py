"""What the performance of this package is measured on: the work a user has it do, through its public entry points.

A case is a plain dict; ``prepare`` builds what a program holds before the call (tokens, router and expert weights),
``run`` is one pass.  Four kinds of pass:

* ``forward`` -- ``topk_moe_forward`` without gradients: decoding steps of a few tokens up to prefill batches;
* ``train``   -- ``topk_moe_forward`` and its backward pass: gradients of the tokens and of every weight;
* ``grouped`` -- the layer composed by hand from the functional calls: ``get_token_indices``, the gathering and the
  scattering ``m_grouped_gemm``, ``scale_and_reduce``;
* ``permute`` -- ``expert_input_permute`` / ``expert_output_permute`` around experts of the caller's own.

Tokens are N(0, 1), weights N(0, 0.02), as in the benchmark.  Feature 0 of every token is 1, so row 0 of the router
weight acts as a per-expert bias: it sets how unevenly the experts are loaded (``skew``).
"""
import math
import os
import sys

import torch

for _p in (os.path.join(os.getcwd(), "moe-explore_b200"), os.getcwd()):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from moe_explore.expert_permute import expert_input_permute, expert_output_permute, get_token_indices  # noqa: E402
from moe_explore.functional.scale_and_reduce import scale_and_reduce  # noqa: E402
from moe_explore.functional.topk_moe import topk_moe_forward  # noqa: E402
from moe_explore.params import (ErnieRouterParams, MLPParams, MOEParams, SharedExpertParams,  # noqa: E402
                                TopkRouterParams)
from moe_explore.router import router  # noqa: E402
from moe_explore.triton_kernels.m_grouped_gemm import MGroupedGEMMParams, m_grouped_gemm  # noqa: E402

# hidden size d, experts E, slots per token k, expert width I: the shapes the benchmark and the baseline notes use
SHAPES = {
    "small": dict(d=256, E=8, k=2, I=512),
    "olmoe": dict(d=2048, E=64, k=8, I=1024),
    "qwen15_moe": dict(d=2048, E=60, k=4, I=1408),
    "qwen3_moe": dict(d=2048, E=128, k=8, I=768),
    "mixtral": dict(d=4096, E=8, k=2, I=14336),
    # one of four expert-parallel ranks of the DeepSeek-V3 shape: 64 of its 256 experts
    "deepseek_v3_rank": dict(d=7168, E=64, k=8, I=2048),
}
# the largest listed case: FLOPs of a pass, and the expert weights a case may hold
MOST_FLOPS = 18.0 * 65536 * 7168 * 2048
MOST_WEIGHTS = 3 * 64 * 7168 * 2048


def _case(kind, tokens, shape, **more):
    case = dict(kind=kind, T=tokens, act="swiglu", dtype="bf16", skew="none", router="topk", softmax_first=False,
                normalize=False, fused_fold=False, shared=0)
    case.update(SHAPES[shape] if isinstance(shape, str) else shape)
    case.update(more)
    return case


def listed():
    cases = [
        # one sequence generating text: the smallest call there is, nothing but latency and launches
        _case("forward", 1, "qwen15_moe", name="decode_1", softmax_first=True),
        # a small serving batch with the options made for inference: one-kernel router tail, fold in the GEMM's epilogue
        _case("forward", 33, "olmoe", name="decode_33_fused", router="fused", softmax_first=True, fused_fold=True,
              skew="mild"),
        # a larger serving batch on few, wide experts: every weight is read for 16 rows of tokens
        _case("forward", 64, "mixtral", name="decode_64_wide"),
        # a prompt of odd length on many narrow experts
        _case("forward", 3001, "qwen3_moe", name="prefill_3001", softmax_first=True, normalize=True, skew="mild"),
        # training at the sizes of a routing-stress sweep: weights and their gradients dominate
        _case("train", 128, "olmoe", name="train_128"),
        # the same with an odd token count and a few popular experts
        _case("train", 1001, "olmoe", name="train_1001_skewed", skew="zipf"),
        # ordinary training of a fine-grained layer with moderate imbalance
        _case("train", 16384, "qwen15_moe", name="train_16384_fine", skew="mild"),
        # training of few, wide experts
        _case("train", 8192, "mixtral", name="train_8192_wide"),
        # one rank's experts of a very large layer, skewed, beside a shared expert: the largest pass
        _case("train", 8192, "deepseek_v3_rank", name="train_8192_shared", skew="zipf", shared=1),
        # a half-precision layer of ungated experts at widths that are no multiple of any tile
        _case("train", 1777, dict(d=776, E=12, k=3, I=1544), name="train_1777_gelu_fp16", act="gelu", dtype="fp16"),
        # a layer composed from the functional calls
        _case("grouped", 4111, "olmoe", name="grouped_4111", softmax_first=True),
        # row movement alone, around experts of the caller's own
        _case("permute", 8192, "olmoe", name="permute_8192", softmax_first=True, skew="mild"),
    ]
    return cases


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(("forward", "forward", "train", "train", "grouped", "permute"))
        if rng.random() < 0.6:
            shape = SHAPES[rng.choice(sorted(SHAPES))]
        else:
            experts = _log_int(rng, 4, 160)
            shape = dict(d=8 * _log_int(rng, 32, 640), E=experts, k=min(experts, rng.randint(1, 8)),
                         I=8 * _log_int(rng, 32, 512))
        tokens = _log_int(rng, {"forward": 1, "train": 32, "grouped": 16, "permute": 16}[kind], 20000)
        router_kind = rng.choice(("topk", "topk", "fused", "ernie")) if kind == "forward" else "topk"
        case = _case(kind, tokens, shape, dtype=rng.choice(("bf16", "bf16", "bf16", "fp16")),
                     act=rng.choice(("swiglu", "swiglu", "swiglu", "geglu", "gelu", "silu")),
                     skew=rng.choice(("none", "mild", "zipf")), router=router_kind,
                     softmax_first=router_kind != "ernie" and rng.random() < 0.5, normalize=rng.random() < 0.3,
                     fused_fold=kind == "forward" and rng.random() < 0.3,
                     shared=1 if kind in ("forward", "train") and rng.random() < 0.15 else 0)
        flops = work(case)["flops"]
        if flops <= MOST_FLOPS and case["E"] * case["d"] * case["I"] * 3 <= MOST_WEIGHTS:
            return case


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float16


def _is_glu(case):
    return "glu" in case["act"]


def _router_bias(case, gen):
    """Row 0 of the router weight: what the constant feature adds to every token's logits."""
    E = case["E"]
    if case["skew"] == "mild":
        return 0.5 * torch.randn(E, generator=gen, device="cuda")
    if case["skew"] == "zipf":
        rank = torch.randperm(E, generator=gen, device="cuda").float() + 1.0
        return -1.1 * torch.log(rank)
    return torch.zeros(E, device="cuda")


def prepare(case, seed):
    torch.cuda.init()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _dtype(case)
    T, d, E, k, width = case["T"], case["d"], case["E"], case["k"], case["I"]
    train = case["kind"] == "train"

    def normal(*shape, std=1.0):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype).mul_(std)

    x = normal(T, d)
    x[:, 0] = 1.0
    router_weight = torch.randn(d, E, generator=gen, device="cuda") * 0.02
    router_weight[0] = _router_bias(case, gen)
    if case["router"] == "ernie":
        bias = 0.001 * torch.randn(E, generator=gen, device="cuda")
        router_params = ErnieRouterParams(router_weight, bias, k)
    else:
        router_weight = router_weight.to(dtype)
        router_params = TopkRouterParams(router_weight, k, case["softmax_first"], case["normalize"])
    state = dict(case=case, x=x, router_weight=router_weight, router_params=router_params)
    if case["kind"] == "permute":
        with torch.no_grad():
            state["scores"], state["indices"] = router(x, router_params)
        return state
    up = 2 * width if _is_glu(case) else width
    w1, w2 = normal(E, d, up, std=0.02), normal(E, width, d, std=0.02)
    shared = None
    leaves = [x, router_weight, w1, w2]
    if case["shared"]:
        s1, s2 = normal(case["shared"], d, up, std=0.02), normal(case["shared"], width, d, std=0.02)
        shared = SharedExpertParams(s1, s2, case["act"])
        leaves += [s1, s2]
    if train:
        for leaf in leaves:
            leaf.requires_grad_()
        state["grad_out"] = normal(T, d)
    state.update(leaves=leaves, w1=w1, w2=w2,
                 params=MOEParams(router_params, MLPParams(w1, w2, case["act"]), E, k, shared))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        out = topk_moe_forward(state["x"], state["params"])
        return [out] + list(torch.autograd.grad(out, state["leaves"], state["grad_out"]))
    with torch.no_grad():
        if case["kind"] == "forward":
            return topk_moe_forward(state["x"], state["params"], fused_router=case["router"] == "fused",
                                    fused_combine=case["fused_fold"])
        if case["kind"] == "grouped":
            return _grouped(state, case)
        grouped = expert_input_permute(state["x"], state["indices"], case["E"], case["k"])
        out = expert_output_permute(grouped, state["scores"], case["k"], state["x"].shape)
        return [grouped.tokens, grouped.group_indices, grouped.indices, out]


def _grouped(state, case):
    T, k = case["T"], case["k"]
    scores, indices = router(state["x"], state["router_params"])
    found = get_token_indices(indices, k, case["E"], zero_prefix=True)
    hidden = m_grouped_gemm(state["x"], MGroupedGEMMParams(state["w1"], found.group_indices, found.indices, True, False,
                                                           T, k, activation=case["act"]))
    rows = m_grouped_gemm(hidden, MGroupedGEMMParams(state["w2"], found.group_indices, found.indices, False, True, T, k))
    return scale_and_reduce(rows, scores, T, k, case["d"])


def work(case):
    """Bytes: tokens, every touched weight and the results once each way (16-bit elements).  FLOPs: the contractions."""
    T, d, E, k, width = case["T"], case["d"], case["E"], case["k"], case["I"]
    rows = T * k
    if case["kind"] == "permute":
        # tokens, the sorted rows written and read again, the result; indices in and out
        return dict(bytes=2.0 * d * (2 * T + 2 * rows) + 8.0 * 2 * rows + 2.0 * rows + 4.0 * (E + 1), flops=2.0 * rows * d)
    matrices = 3 if _is_glu(case) else 2
    per_expert = matrices * d * width
    weights = per_expert * min(E, rows) + per_expert * case["shared"]
    flops = 2.0 * per_expert * (rows + T * case["shared"]) + 2.0 * T * d * E
    router_bytes = d * E * (4.0 if case["router"] == "ernie" else 2.0)
    if case["kind"] == "train":
        # tokens and dOut in, out and dX out; weights in, their gradients out
        grads = per_expert * (E + case["shared"])
        return dict(bytes=2.0 * (4 * T * d + weights + grads) + 2 * router_bytes, flops=3.0 * flops)
    return dict(bytes=2.0 * (2 * T * d + weights) + router_bytes, flops=flops)


def tolerance(case):
    """Three to four times the 2-norm deviation from the same pass in 64-bit (the widest layers: 32-bit) arithmetic:
    intermediate rows are rounded to the 16-bit type (measured 3.2e-3 to 5.6e-3 in bf16, 4.3e-4 to 8.5e-4 in fp16;
    the fold of the permutes alone 1.7e-3 and 2e-4); folding in the epilogue rounds once per slot."""
    if case["kind"] == "permute":
        return {"rel": 0.008 if case["dtype"] == "bf16" else 0.001}
    if case["dtype"] == "fp16":
        return {"rel": 0.004 if case["fused_fold"] else 0.003}
    return {"rel": 0.024 if case["fused_fold"] else 0.016}
