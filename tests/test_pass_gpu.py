"""A pass over the experts where whole 64-row blocks of the padded layout hold no routed row: those blocks are neither written nor
read, so whatever the allocator hands out there (here: NaN) must not reach a result."""
import pytest
import torch

from moe_explore.expert_compute import expert_compute, routed_expert_compute
from moe_explore.routing_plan import build_routing_plan, device_status
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu


def _poison(mb=512):
    blocks = [torch.full((n << 18,), float("nan"), device="cuda") for n in (1, 1, 2, 4, 8, 16, 32, mb // 4)]
    del blocks


def _relerr(a, b):
    return float((a.float() - b.float()).abs().max() / b.float().abs().max().clamp_min(1e-30))


@pytest.mark.parametrize("act", ["swiglu", "gelu"])
@pytest.mark.parametrize("rows", [
    (1, 63, 64, 65, 127, 128, 129, 0, 2),       # one-CTA kernels: at most one row tile per expert on average
    (33, 0, 0, 1),                              # empty experts, weight gradients over one 64-row step
    (193, 255, 256, 257, 320, 0, 449, 129),     # CTA pairs with a half-empty second tile
])
def test_blocks_without_rows_do_not_leak(rows, act, native):
    d, inter, E = 136, 200, len(rows)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))
    g = torch.Generator().manual_seed(len(ids))
    ids = ids[torch.randperm(len(ids), generator=g)].view(-1, 1).cuda()
    T = ids.size(0)
    gen = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=gen, device="cuda") * std).bfloat16()
    up = 2 * inter if act == "swiglu" else inter
    leaves = [mk(T, d), torch.rand(T, 1, generator=gen, device="cuda").bfloat16(), mk(E, d, up, std=0.1), mk(E, inter, d, std=0.1)]
    grad = mk(T, d)

    def run(how):
        p = [t.clone().requires_grad_() for t in leaves]
        _poison()
        out = how(p)
        _poison()
        return [out.detach()] + list(torch.autograd.grad(out, p, grad))

    routed = run(lambda p: routed_expert_compute(*p, ids, E, 1, act))
    planned = run(lambda p: expert_compute(*p, build_routing_plan(ids, E, 1), act))
    gathered = run(lambda p: routed_expert_compute(*p, ids, E, 1, act, gather_in_gemm=True))
    f = [t.float().requires_grad_() for t in leaves]
    ref = O.expert_compute(f[0], f[1], ids, f[2], f[3], act)
    expect = [ref.detach()] + list(torch.autograd.grad(ref, f, grad.float()))
    for a, b, c, e in zip(routed, planned, gathered, expect):
        assert torch.equal(a, b) and torch.equal(a, c)
        assert _relerr(a, e) <= 2e-2     # bf16 storage of every intermediate row, as in the layer tests
    for e, n in enumerate(rows):
        if n == 0:
            assert not routed[3][e].any() and not routed[4][e].any()
    with torch.no_grad():
        _poison()
        assert torch.equal(routed_expert_compute(*leaves, ids, E, 1, act), routed[0])
        _poison()
        assert _relerr(routed_expert_compute(*leaves, ids, E, 1, act, fused_combine=True), expect[0]) <= 2e-2
    assert native.read_status(build_routing_plan(ids, E, 1).status) == 0


@pytest.mark.parametrize("act", [None, "silu", "swiglu"])
@pytest.mark.parametrize("gather,scatter", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("rows", [(1, 63, 64, 65, 127, 128, 129, 0, 3), (0, 520, 1, 255, 0, 384), (2049,)])
def test_functional_gemm_against_its_steps(rows, gather, scatter, act, native):
    """Rows read without padding, rows gathered, rows stored through the map (gated ones too): bit for bit what copying into the
    padded layout, contracting there and copying back gives."""
    from moe_explore.routing_plan import plan_from_groups
    from moe_explore.triton_kernels.m_grouped_gemm import MGroupedGEMMParams, m_grouped_gemm

    E, K, N, topk, R = len(rows), 136, 208, 1 if gather and scatter else 3, sum(rows)
    if R % topk:
        topk = 1
    g = torch.Generator(device="cuda").manual_seed(R)
    groups = torch.tensor([0] + list(rows), dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    perm = torch.randperm(R, generator=g, device="cuda")
    w = (torch.randn(E, K, N, generator=g, device="cuda") * 0.1).bfloat16()
    x = torch.randn(R // topk if gather else R, K, generator=g, device="cuda").bfloat16()
    tokens = R // topk if (gather or scatter) else R
    out = m_grouped_gemm(x, MGroupedGEMMParams(w, groups, perm, gather, scatter, tokens, topk, activation=act))

    plan = plan_from_groups(groups, R)
    pos = plan.row_src.long()
    src = torch.where(pos >= 0, perm[pos.clamp_min(0)] // topk if gather else pos, -1).int()
    a = torch.empty(plan.padded_rows, K, dtype=x.dtype, device="cuda")
    native.gather_rows(x, src, plan.num_mtiles, a, 1)
    cols = N // 2 if act == "swiglu" else N
    y = torch.empty(plan.padded_rows, cols, dtype=x.dtype, device="cuda")
    native.mgrouped_gemm(a, w, y, None, plan.mtile_expert, plan.tile_pairs, plan.num_mtiles, False, act, plan.status)
    ref = torch.empty(R, cols, dtype=x.dtype, device="cuda")
    native.unpad_rows(y, plan.dst_row, ref)
    if scatter:
        ref = torch.empty_like(ref).index_copy_(0, perm, ref)
    assert torch.equal(out, ref)


@pytest.mark.parametrize("normalize", [False, True])
@pytest.mark.parametrize("E,k,d,dtype", [(8, 1, 64, torch.bfloat16), (60, 4, 264, torch.float16), (64, 8, 520, torch.bfloat16),
                                         (129, 9, 72, torch.bfloat16), (300, 40, 128, torch.bfloat16)])
def test_router_inside_the_pass(E, k, d, dtype, normalize, native):
    """Router and experts in one step against the router's torch ops in front of the experts: the forward bit for bit, the
    gradients against 32-bit autograd no further off than the composed form (whose input gradient is rounded three times)."""
    from moe_explore.expert_compute import routed_layer, router_joins_the_pass
    from moe_explore.params import TopkRouterParams
    from moe_explore.router import topk_router

    T, inter = 203, 64
    g = torch.Generator(device="cuda").manual_seed(E + k)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(dtype)
    leaves = [mk(T, d), mk(d, E, std=0.3), mk(E, d, 2 * inter, std=0.1), mk(E, inter, d, std=0.1)]
    addend, grad = mk(T, d), mk(T, d)

    def run(fused):
        x, wr, w1, w2 = p = [t.clone().requires_grad_() for t in leaves]
        a = addend.clone().requires_grad_()
        rp = TopkRouterParams(wr, k, False, normalize)
        if fused:
            assert router_joins_the_pass(x, rp, E, k) == (k <= 8) and not router_joins_the_pass(x.detach(), TopkRouterParams(wr.detach(), k, False, normalize), E, k)
            out = routed_layer(x, rp, w1, w2, E, "swiglu", addend=a)
        else:
            scores, idx = topk_router(x, rp)
            out = routed_expert_compute(x, scores, w1, w2, idx, E, k, "swiglu", addend=a)
        return [out.detach()] + list(torch.autograd.grad(out, p + [a], grad))

    fused, composed = run(True), run(False)
    assert torch.equal(fused[0], composed[0]) and torch.equal(fused[5], composed[5])
    f = [t.float().requires_grad_() for t in leaves]
    with torch.no_grad():
        _, idx = topk_router(leaves[0], TopkRouterParams(leaves[1], k, False, normalize))
    scores = torch.softmax(torch.gather(f[0] @ f[1], -1, idx), -1)
    ref = O.expert_compute(f[0], scores, idx, f[2], f[3], "swiglu") + addend.float()
    expect = [ref.detach()] + list(torch.autograd.grad(ref, f, grad.float()))
    for a, c, e in zip(fused, composed, expect):
        err = lambda t: float((t.float() - e).norm() / e.norm().clamp_min(1e-20))
        # 1.25: the roundings of the two forms differ, in 2-norms over thousands of elements by far less
        assert err(a) <= 1.25 * err(c) + 1e-5


@pytest.mark.parametrize("act", [None, "silu", "swiglu"])
@pytest.mark.parametrize("T", [1, 63, 64, 65, 129, 700])
def test_one_expert_for_every_token(T, act, native):
    """The in-place form of one always-selected expert against the same expert as a top-1 layer with unit weights: every
    element is the same sum of the same products, so bit for bit (the fold of one row with weight one is exact)."""
    from moe_explore.expert_compute import dense_expert

    d, inter = 136, 200
    g = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).bfloat16()
    leaves = [mk(T, d), mk(1, d, 2 * inter if act == "swiglu" else inter, std=0.1), mk(1, inter, d, std=0.1)]
    grad = mk(T, d)
    ids = torch.zeros(T, 1, dtype=torch.int64, device="cuda")
    ones = torch.ones(T, 1, dtype=torch.bfloat16, device="cuda")

    def run(how):
        p = [t.clone().requires_grad_() for t in leaves]
        _poison()
        out = how(*p)
        _poison()
        return [out.detach()] + list(torch.autograd.grad(out, p, grad))

    dense = run(lambda x, w1, w2: dense_expert(x, w1, w2, act))
    layer = run(lambda x, w1, w2: routed_expert_compute(x, ones, w1, w2, ids, 1, 1, act))
    for a, b in zip(dense, layer):
        assert torch.equal(a, b)
    with torch.no_grad():
        assert torch.equal(dense_expert(*leaves, act), dense[0])


def _poison_maps():
    """Freed blocks full of indices that are out of every range, for the index arrays of the next calls."""
    blocks = [torch.full((n << 10,), 0x7FFFFFFF, dtype=torch.int32, device="cuda") for n in (1, 1, 1, 2, 4, 16, 64, 256)]
    del blocks


@pytest.mark.parametrize("T,k,E", [(1, 2, 8), (300, 2, 8), (2048, 2, 4)])   # one-CTA kernels; the last one: CTA pairs
def test_every_row_dropped(T, k, E, native):
    """All expert ids out of range: no row tile is in use and no map entry may be used.  Zeros everywhere, status 100."""
    d, inter = 136, 200
    g = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    leaves = [mk(T, d), mk(T, k), mk(E, d, 2 * inter), mk(E, inter, d)]
    ids = torch.full((T, k), E + 5, dtype=torch.int64, device="cuda")
    ids[0, 0] = -1

    def check(tensors):
        torch.cuda.synchronize()
        assert all(not t.any() for t in tensors)
        assert native.read_status(device_status(), reset=True) == 100

    native.read_status(device_status(), reset=True)
    for gather in (False, True):
        p = [t.clone().requires_grad_() for t in leaves]
        _poison_maps()
        out = routed_expert_compute(*p, ids, E, k, "swiglu", gather_in_gemm=gather)
        check([out.detach()] + list(torch.autograd.grad(out, p, mk(T, d))))
        with torch.no_grad():
            for fused in (False, True):
                _poison_maps()
                check([routed_expert_compute(*leaves, ids, E, k, "swiglu", gather_in_gemm=gather, fused_combine=fused)])
    _poison_maps()
    check([expert_compute(*leaves, build_routing_plan(ids, E, k), "swiglu")])


@pytest.mark.parametrize("gather,scatter", [(False, False), (True, True)])
def test_refused_group_with_all_the_rows(gather, scatter, native):
    """A prefix that ends past the rows: the only group with rows is refused (status 5) and nothing is contracted."""
    from moe_explore.triton_kernels.m_grouped_gemm import MGroupedGEMMParams, m_grouped_gemm

    R, K, N = 70, 136, 208
    x = torch.randn(R, K, device="cuda").bfloat16()
    for groups in ([0, R + 1], [0, 0, R + 200]):
        w = torch.randn(len(groups) - 1, K, N, device="cuda").bfloat16()
        _poison_maps()
        out = m_grouped_gemm(x, MGroupedGEMMParams(w, torch.tensor(groups, dtype=torch.int32, device="cuda"),
                                                   torch.arange(R, device="cuda"), gather, scatter, R, 1))
        torch.cuda.synchronize()
        assert out.shape == (R, N) and native.read_status(device_status(), reset=True) == 5


@pytest.mark.parametrize("one_block", [True, False])
def test_scratch_in_one_block_or_several(one_block, monkeypatch, native):
    """The same bits however the buffers of a pass are allocated and wherever the saved ones come back to."""
    from moe_explore import expert_compute as ec
    from moe_explore.functional.topk_moe import topk_moe_forward
    from moe_explore.params import MLPParams, MOEParams, TopkRouterParams

    T, d, inter, E, k = 77, 136, 200, 6, 2
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).bfloat16()
    leaves = [mk(T, d), mk(d, E, std=0.1), mk(E, d, 2 * inter, std=0.1), mk(E, inter, d, std=0.1)]
    grad = mk(T, d)

    def run(softmax_before):
        x, wr, w1, w2 = p = [t.clone().requires_grad_() for t in leaves]
        params = MOEParams(TopkRouterParams(wr, k, softmax_before, True), MLPParams(w1, w2, "swiglu"), E, k)
        moved = torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), lambda t: t.clone())
        with moved:
            _poison()
            out = topk_moe_forward(x, params)
            _poison()
            grads = torch.autograd.grad(out, p, grad)
        with torch.no_grad():
            again = topk_moe_forward(x, params)                  # router and experts without a gradient: one call
            _poison()
            assert torch.equal(again, out)
            composed = topk_moe_forward(x, params, fused_combine=False, gather_in_gemm=True)
            assert torch.equal(composed, out)
        return [out.detach(), *grads]

    ref = [run(b) for b in (False, True)]
    if not one_block:
        monkeypatch.setattr(ec, "SCRATCH_IN_ONE", 0)
        for b in (False, True):
            assert all(torch.equal(x, y) for x, y in zip(run(b), ref[b]))
