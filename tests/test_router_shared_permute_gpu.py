"""The steps either side of the expert GEMMs: the opt-in fused router kernel, the shared-expert branch and the
stand-alone permute API, each against torch / the oracle on the GPU."""
import numpy as np
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu

TOL = 2e-2


def relerr(a, b):
    return float((a.float() - b.float()).abs().max() / b.float().abs().max().clamp_min(1e-30))


@pytest.mark.parametrize("softmax_before,normalize", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("T,E,k,dtype", [(1000, 8, 2, torch.bfloat16), (513, 60, 4, torch.bfloat16), (300, 64, 8, torch.float16),
                                          (257, 256, 8, torch.float32), (64, 1024, 8, torch.float32), (5, 8, 8, torch.float32)])
def test_fused_router_kernel_on_tie_free_logits(T, E, k, dtype, softmax_before, normalize, native):
    """Logits without ties (a random permutation of distinct values per row): the kernel selects exactly torch.topk's
    experts -- in descending order of value, which is torch.topk(sorted=True)'s order -- and its scores match the
    reference's torch ops (router.py:17-35) to a rounding of the output type; the histogram equals bincount."""
    g = torch.Generator(device="cuda").manual_seed(T + E)
    # distinct, exactly representable values: multiples of 1/8 in [-E/16, E/16), shuffled per row
    base = (torch.arange(E, device="cuda", dtype=torch.float32) - E // 2) / 8
    logits = torch.stack([base[torch.randperm(E, generator=g, device="cuda")] for _ in range(T)]).to(dtype)
    scores, idx, counts = native.router_topk(logits, k, softmax_before, normalize, want_counts=True)
    ref_in = torch.softmax(logits, -1, dtype=torch.float32) if softmax_before else logits
    ref_s, ref_i = torch.topk(ref_in, k, dim=-1, sorted=True)
    if not softmax_before:
        ref_s = torch.softmax(ref_s, -1, dtype=torch.float32)
    if normalize:
        ref_s = ref_s / ref_s.sum(-1, keepdim=True)
    assert idx.dtype == torch.int64 and torch.equal(idx, ref_i)
    assert scores.dtype == dtype
    assert relerr(scores, ref_s.to(dtype)) <= (1e-5 if dtype is torch.float32 else 1e-2)
    assert torch.equal(counts.long(), torch.bincount(ref_i.reshape(-1), minlength=E))


def test_fused_router_declared_tie_rule(native):
    """Equal logits: the lowest expert index is taken first (torch.topk's choice here is unspecified, which is why the
    fused router is opt-in); NaN is never selected."""
    logits = torch.zeros(4, 16, device="cuda")
    logits[1, 9] = 1.0
    logits[2, :] = float("nan")
    logits[2, 5] = -3.0
    logits[3, 2] = float("nan")
    _, idx, _ = native.router_topk(logits, 3, False, False)
    assert idx[0].tolist() == [0, 1, 2]
    assert idx[1].tolist() == [9, 0, 1]
    assert idx[2].tolist()[0] == 5
    assert idx[3].tolist() == [0, 1, 3]


def test_layer_with_the_fused_router_matches_the_default_router(native):
    """Whole layer, forward and backward, with ``fused_router=True`` against the default (torch-op) router on logits
    that are tie-free after the bf16 GEMM's rounding is accounted for: the selected sets are equal, so outputs and
    gradients agree to the tolerance (the slot order inside a token differs, which only permutes summands)."""
    from moe_explore.functional.topk_moe import topk_moe_forward
    from moe_explore.params import MLPParams, MOEParams, TopkRouterParams

    T, d, E, k, I = 700, 256, 16, 4, 128
    g = torch.Generator(device="cuda").manual_seed(8)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).bfloat16()
    x, wr, w1, w2, grad = mk(T, d), mk(d, E, std=0.3), mk(E, d, 2 * I, std=0.05), mk(E, I, d, std=0.05), mk(T, d)
    logits = x @ wr
    top5 = torch.topk(logits.float(), k + 1, dim=-1).values
    keep = (top5[:, :-1] - top5[:, 1:]).min(-1).values > 0      # rows whose top-(k+1) logits are all distinct
    x, grad = x[keep].contiguous(), grad[keep].contiguous()
    results = []
    for fused in (False, True):
        leaves = [t.detach().clone().requires_grad_() for t in (x, wr, w1, w2)]
        params = MOEParams(TopkRouterParams(leaves[1], k, False, False), MLPParams(leaves[2], leaves[3], "swiglu"), E, k)
        out = topk_moe_forward(leaves[0], params, fused_router=fused)
        out.backward(grad)
        results.append([out.detach()] + [t.grad for t in leaves])
    for name, a, b in zip(("out", "dx", "d_router", "dw1", "dw2"), results[1], results[0]):
        assert relerr(a, b) <= TOL, name


@pytest.mark.parametrize("num_shared,act", [(1, "swiglu"), (2, "swiglu"), (3, "silu")])
def test_shared_expert_branch(num_shared, act, native):
    """topk_moe_forward with ``shared_expert_params`` (functional/topk_moe.py:56-62): the routed output plus the sum
    over the shared experts of act(x @ up) @ down, forward and backward, against fp32 torch on the same inputs."""
    from moe_explore.functional.topk_moe import topk_moe_forward
    from moe_explore.params import MLPParams, MOEParams, SharedExpertParams, TopkRouterParams

    T, d, E, k, I, Is = 400, 256, 8, 2, 128, 192
    g = torch.Generator(device="cuda").manual_seed(num_shared)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).bfloat16()
    x, wr, w1, w2, grad = mk(T, d), mk(d, E, std=0.1), mk(E, d, 2 * I, std=0.05), mk(E, I, d, std=0.05), mk(T, d)
    up = mk(num_shared, d, 2 * Is if "glu" in act else Is, std=0.05)
    down = mk(num_shared, Is, d, std=0.05)
    leaves = [t.detach().clone().requires_grad_() for t in (x, w1, w2, up, down)]
    params = MOEParams(TopkRouterParams(wr, k, False, False), MLPParams(leaves[1], leaves[2], "swiglu"), E, k,
                       SharedExpertParams(leaves[3], leaves[4], act))
    out = topk_moe_forward(leaves[0], params)
    out.backward(grad)
    # oracle: routed part by the oracle's expert loop (scores re-derived in fp32 from the same selection, so that the
    # input gradient includes the path through the router), shared part as the reference writes it
    from moe_explore.router import router

    with torch.no_grad():
        _, idx = router(x, params.router_params)
    f = [t.detach().float().requires_grad_() for t in (x, w1, w2, up, down)]
    scores = torch.softmax(torch.gather(f[0] @ wr.float(), -1, idx), -1)
    ref = O.expert_compute(f[0], scores, idx, f[1], f[2], "swiglu")
    h = O.activation(f[0] @ f[3], act) @ f[4]
    ref = ref + h.sum(0)
    ref.backward(grad.float())
    assert relerr(out, ref) <= TOL
    for name, a, b in zip(("dx", "dw1", "dw2", "d_up", "d_down"), [t.grad for t in leaves], [t.grad for t in f]):
        assert relerr(a, b) <= TOL, name


def test_expert_input_and_output_permute(native):
    """expert_input_permute / expert_output_permute (expert_permute.py:43-68): rows gathered into expert order are
    exact copies, the group prefix is the reference's, and permuting back with the router weights folds the k slots."""
    from moe_explore.expert_permute import expert_input_permute, expert_output_permute

    T, d, E, k = 777, 264, 16, 4
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(T, d, generator=g, device="cuda").bfloat16()
    top, idx = torch.topk(torch.randn(T, E, generator=g, device="cuda"), k, dim=-1, sorted=False)
    scores = torch.softmax(top, -1).bfloat16()
    grouped = expert_input_permute(x, idx, E, k)
    ref = O.get_token_indices(idx.cpu(), k, E, zero_prefix=True)
    assert torch.equal(grouped.group_indices.cpu(), ref.group_indices)
    assert torch.equal(grouped.indices.cpu(), ref.indices)
    assert torch.equal(grouped.tokens, x[(ref.indices // k).cuda()])
    back = expert_output_permute(grouped, scores, k, x.shape)
    # every token's k copies of its own row, weighted: x[t] * sum_s scores[t, s] (fp32 fold, one rounding)
    expect = (x.float() * scores.float().sum(-1, keepdim=True))
    assert back.shape == x.shape and relerr(back, expect) <= 1e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("softmax_before,normalize", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("T,E,k", [(1, 8, 1), (7, 8, 8), (3, 31, 5), (300, 33, 2), (513, 60, 4), (1000, 64, 8), (65, 100, 6),
                                   (2048, 128, 7), (70, 257, 9), (33, 1024, 32), (5, 600, 31), (9, 20, 13)])
def test_router_tail_leaves_the_bits_of_the_torch_ops(T, E, k, softmax_before, normalize, dtype, native):
    """Scores and indices against the launches the kernel stands for, among ties (every third row is a few distinct values),
    signed zeros, infinities and NaN."""
    from moe_explore.params import TopkRouterParams
    from moe_explore.router import topk_of_logits

    g = torch.Generator(device="cuda").manual_seed(T + E)
    logits = torch.randn(T, E, generator=g, device="cuda") * 2
    logits[::3] = (logits[::3] * 0.7).round()
    if T > 6:
        logits[1, ::2], logits[1, 1::2] = 0.0, -0.0
        logits[2, E // 2] = float("nan")
        logits[3, :2] = float("inf")
        logits[4, 1:] = float("-inf")
        logits[5] = float("-inf")
    logits = logits.to(dtype)
    p = TopkRouterParams(None, k, softmax_before, normalize)
    seen = []
    real, native.router_tail = native.router_tail, lambda *a: seen.append(1) or real(*a)
    try:
        scores, idx = topk_of_logits(logits, p, dtype)
    finally:
        native.router_tail = real
    ref_s, ref_i = topk_of_logits(logits.clone().requires_grad_(), p, dtype)     # a gradient wanted: the single ops
    assert len(seen) == 1 and ref_s.requires_grad
    assert torch.equal(idx, ref_i) and scores.dtype is dtype
    assert torch.equal(scores.nan_to_num(nan=-7.0), ref_s.detach().nan_to_num(nan=-7.0))


def test_router_tail_leaves_transforms_to_the_single_ops(native):
    from moe_explore.params import TopkRouterParams
    from moe_explore.router import topk_of_logits
    import torch.autograd.forward_ad as fwd

    p = TopkRouterParams(None, 2, True, True)
    logits = torch.randn(4, 6, 8, device="cuda")
    ref = torch.stack([topk_of_logits(row, p, torch.float32)[0] for row in logits])
    assert torch.equal(torch.func.vmap(lambda row: topk_of_logits(row, p, torch.float32)[0])(logits), ref)
    with fwd.dual_level():
        out, _ = topk_of_logits(fwd.make_dual(logits[0], torch.ones_like(logits[0])), p, torch.float32)
        assert fwd.unpack_dual(out).tangent is not None
    with torch.no_grad():
        out, _ = topk_of_logits(logits[0].t().contiguous().t(), p, torch.float32)      # other strides: the single ops
        assert torch.equal(out, ref[0])


def test_transforms_over_the_bias_see_the_single_ops(native):
    from moe_explore.params import ErnieRouterParams
    from moe_explore.router import ernie_router

    x, w, biases = (torch.randn(*s, device="cuda") for s in ((5, 16), (16, 8), (3, 8)))
    each = [ernie_router(x, ErnieRouterParams(w, b, 2)) for b in biases]
    scores, indices = torch.func.vmap(lambda b: ernie_router(x, ErnieRouterParams(w, b, 2)))(biases)
    assert torch.equal(scores, torch.stack([s for s, _ in each])) and torch.equal(indices, torch.stack([i for _, i in each]))
    # the bias only selects: its gradient is zero
    zero = torch.func.grad(lambda b: ernie_router(x, ErnieRouterParams(w, b, 2))[0].sum())(biases[0])
    assert torch.equal(zero, torch.zeros_like(zero))


@pytest.mark.parametrize("router_topk", [torch.tensor(2), np.int64(2)], ids=["tensor", "numpy"])
def test_a_router_may_count_its_slots_in_another_type(router_topk, native):
    from moe_explore.functional.topk_moe import topk_moe_forward
    from moe_explore.params import MLPParams, MOEParams, TopkRouterParams

    E, d = 4, 64
    x, wr, w1, w2 = ((torch.randn(*s, device="cuda") * 0.3).bfloat16() for s in ((9, d), (d, E), (E, d, 2 * d), (E, d, d)))
    out = [topk_moe_forward(x, MOEParams(TopkRouterParams(wr, k, True, False), MLPParams(w1, w2, "swiglu"), E, 2)) for k in (2, router_topk)]
    assert torch.equal(*out)


def test_the_router_compiles_into_one_graph(native):
    from moe_explore.params import ErnieRouterParams, TopkRouterParams
    from moe_explore.router import router

    x, w, bias = (torch.randn(*s, device="cuda") for s in ((5, 16), (16, 8), (8,)))
    for p in (TopkRouterParams(w, 2, True, True), TopkRouterParams(w, 2, False, False), ErnieRouterParams(w, bias, 2)):
        for got, want in zip(torch.compile(lambda x: router(x, p), backend="eager", fullgraph=True)(x), router(x, p)):
            assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,E,k", [(1, 8, 1), (7, 8, 8), (300, 33, 2), (1000, 64, 8), (65, 257, 9), (3, 1024, 32)])
def test_ernie_tail_leaves_the_bits_of_the_torch_ops(T, E, k, dtype, native):
    from moe_explore.params import ErnieRouterParams
    from moe_explore.router import ernie_router

    g = torch.Generator(device="cuda").manual_seed(T + E)
    x = torch.randn(T, 64, generator=g, device="cuda").to(dtype)
    if T > 6:
        x[1] = 0          # equal probabilities everywhere
        x[2] = float("nan")
    w = torch.randn(64, E, generator=g, device="cuda") * 0.2
    for bias in (0.01 * torch.randn(E, generator=g, device="cuda"), torch.zeros(E, device="cuda")):
        p = ErnieRouterParams(w, bias, k)
        scores, idx = ernie_router(x, p)
        ref_s, ref_i = ernie_router(x.clone().requires_grad_(), p)     # a gradient wanted: the single ops
        assert ref_s.requires_grad and not scores.requires_grad and scores.dtype is dtype
        assert torch.equal(idx, ref_i)
        assert torch.equal(scores.nan_to_num(nan=-7.0), ref_s.detach().nan_to_num(nan=-7.0))


@pytest.mark.parametrize("kind", ["topk", "fused", "ernie"])
def test_routers_inside_a_forward_pass(kind, native):
    """The layer without gradients against its router and its experts one after the other."""
    from moe_explore.expert_compute import routed_expert_compute
    from moe_explore.functional.topk_moe import topk_moe_forward
    from moe_explore.params import ErnieRouterParams, MLPParams, MOEParams, TopkRouterParams
    from moe_explore.router import fused_topk_router, router

    T, d, inter, E, k = 45, 136, 72, 9, 3
    g = torch.Generator(device="cuda").manual_seed(5)
    mk = lambda *s, std=1.0: torch.randn(*s, generator=g, device="cuda") * std
    x, w1, w2 = mk(T, d).bfloat16(), mk(E, d, 2 * inter, std=0.1).bfloat16(), mk(E, inter, d, std=0.1).bfloat16()
    wr = mk(d, E, std=0.1)
    rp = ErnieRouterParams(wr, mk(E, std=0.01), k) if kind == "ernie" else TopkRouterParams(wr.bfloat16(), k, True, True)
    with torch.no_grad():
        out = topk_moe_forward(x, MOEParams(rp, MLPParams(w1, w2, "swiglu"), E, k), fused_router=kind == "fused")
        scores, idx = fused_topk_router(x, rp) if kind == "fused" else router(x, rp)
        assert torch.equal(out, routed_expert_compute(x, scores, w1, w2, idx, E, k, "swiglu"))


@pytest.mark.parametrize("device", ["cuda", "cpu"])
def test_a_default_device_leaves_a_forward_pass_as_it_is(device, native):
    from moe_explore.functional.topk_moe import topk_moe_forward
    from moe_explore.params import MLPParams, MOEParams, TopkRouterParams

    E, d = 4, 64
    x, wr, w1, w2 = ((torch.randn(*s, device="cuda") * 0.3).bfloat16() for s in ((9, d), (d, E), (E, d, 2 * d), (E, d, d)))
    params = MOEParams(TopkRouterParams(wr, 2, True, True), MLPParams(w1, w2, "swiglu"), E, 2)
    seen = []
    real, native.run_pass = native.run_pass, lambda name, p, steps, rows: (seen.append([s[0] for s in steps]), real(name, p, steps, rows))
    try:
        with torch.no_grad():
            out = topk_moe_forward(x, params)
            with torch.device(device):
                assert torch.equal(topk_moe_forward(x, params), out)
    finally:
        native.run_pass = real
    assert seen[0] == seen[1] and native.FWD_TAIL in seen[1]
