"""The contractions of a pass on transposed tiles against the same steps through the entry points that take 128-row tiles."""
import pytest
import torch

from moe_explore.expert_compute import dense_expert, routed_expert_compute
from moe_explore.routing_plan import build_routing_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", [None, "silu", "gelu", "swiglu", "geglu"])
@pytest.mark.parametrize("d,inter", [(264, 200), (128, 320), (72, 8)])    # columns past a tile, a CTA, a warp; K past a step
@pytest.mark.parametrize("rows", [
    (1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 0, 300),       # row units of one tile
    (193, 255, 256, 257, 320, 0, 449, 129),                   # the same, too few of them for larger ones
    (193, 255, 256, 257, 320, 0, 449, 129) * 5,               # of two, with one, with a rest
])
def test_a_pass_equals_its_steps(rows, d, inter, act, dtype, native):
    """Every element is the same sum of the same products in the same order: bit for bit."""
    E = len(rows)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(d))].view(-1, 1).cuda()
    T = ids.size(0)
    gen = torch.Generator(device="cuda").manual_seed(inter)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=gen, device="cuda") * std).to(dtype)
    n1 = 2 * inter if act in ("swiglu", "geglu") else inter
    x, scores = mk(T, d), torch.rand(T, 1, generator=gen, device="cuda").to(dtype)
    w1, w2, grad = mk(E, d, n1, std=0.1), mk(E, inter, d, std=0.1), mk(T, d)
    leaves = [t.requires_grad_() for t in (x, scores, w1, w2)]
    out = routed_expert_compute(*leaves, ids, E, 1, act)
    got = [out.detach()] + list(torch.autograd.grad(out, leaves, grad))
    with torch.no_grad():
        assert torch.equal(routed_expert_compute(*leaves, ids, E, 1, act), got[0])
        fused = routed_expert_compute(*leaves, ids, E, 1, act, fused_combine=True)
        assert torch.equal(fused, got[0])     # one slot: one addition to zero

        plan = build_routing_plan(ids, E, 1)
        maps = (plan.mtile_expert, plan.tile_pairs, plan.num_mtiles)
        new = lambda n: torch.empty(plan.padded_rows, n, dtype=dtype, device="cuda")
        xs, pre, hidden, ys, gs, d_pre, dxs = new(d), new(n1) if act else None, new(inter), new(d), new(d), new(n1), new(d)
        native.gather_rows(x, plan.row_src, plan.num_mtiles, xs, 1)
        native.mgrouped_gemm(xs, w1, hidden, pre, *maps, False, act, plan.status)
        native.mgrouped_gemm(hidden, w2, ys, None, *maps, False, None, plan.status)
        d_scores = torch.empty_like(scores)
        native.combine_bwd_tokens(grad, scores, ys, plan.dst_row, plan.row_src, plan.num_mtiles, gs, d_scores, 1)
        if act is None:
            native.mgrouped_gemm(gs, w2, d_pre, None, *maps, True, None, plan.status)
        else:
            native.mgrouped_gemm_dglu(gs, w2, pre, d_pre, *maps, act, plan.status)
        native.mgrouped_gemm(d_pre, w1, dxs, None, *maps, True, None, plan.status)
        ref, dx, dw1, dw2 = torch.empty_like(x), torch.empty_like(x), torch.empty_like(w1), torch.empty_like(w2)
        native.combine_topk(ys, scores, plan.dst_row, ref, 1)
        native.combine_topk(dxs, None, plan.dst_row, dx, 1)
        native.kgrouped_gemm(xs, d_pre, dw1, plan.pad_offsets, plan.status)
        native.kgrouped_gemm(hidden, gs, dw2, plan.pad_offsets, plan.status)
    for a, b in zip(got, (ref, dx, d_scores, dw1, dw2)):
        assert torch.equal(a, b)
    assert native.read_status(plan.status) == 0


@pytest.mark.parametrize("tokens", [5, 700])     # one row unit per expert; more units than CTA pairs
def test_operands_written_right_before_a_pass_are_the_ones_it_reads(tokens):
    """The contractions ask for weights and row maps before the kernel before them has ended, but not before the pass begins."""
    E, k, d, inter = 32, 4, 768, 512
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)
    sets = [(mk(tokens, d), torch.rand(tokens, k, generator=gen, device="cuda").bfloat16(), mk(E, d, 2 * inter), mk(E, inter, d),
             torch.rand(tokens, E, generator=gen, device="cuda").topk(k).indices, mk(tokens, d)) for _ in range(2)]

    def run(x, scores, w1, w2, ids, grad):
        leaves = [t.detach().requires_grad_() for t in (x, scores, w1, w2)]
        out = routed_expert_compute(*leaves, ids, E, k, "swiglu")
        return [out.detach()] + list(torch.autograd.grad(out, leaves, grad))

    expected = [run(*s) for s in sets]
    now = [t.clone() for t in sets[0]]
    for i in range(20):
        for t, new in zip(now, sets[i % 2]):
            t.copy_(new)
        for a, b in zip(run(*now), expected[i % 2]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("tokens", [5, 700])
def test_maps_are_the_ones_of_this_pass_and_not_of_the_one_before(tokens):
    """Two routings in turn, out of a graph: each pass writes its row maps where the pass before had its own, and its contractions read
    them before they wait for the kernel in front."""
    E, k, d, inter = 32, 4, 256, 128
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(torch.bfloat16)
    x, scores, w1, w2 = mk(tokens, d), torch.rand(tokens, k, generator=gen, device="cuda").bfloat16(), mk(E, d, 2 * inter), mk(E, inter, d)
    routings = [torch.rand(tokens, E, generator=gen, device="cuda").topk(k).indices for _ in range(2)]
    with torch.no_grad():
        expected = [routed_expert_compute(x, scores, w1, w2, ids, E, k, "swiglu") for ids in routings]
        wrong = torch.zeros((), dtype=torch.int64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for i in range(20):
                wrong += torch.ne(routed_expert_compute(x, scores, w1, w2, routings[i % 2], E, k, "swiglu"), expected[i % 2]).any()
        for _ in range(1000):
            graph.replay()
    assert not torch.equal(*expected) and int(wrong) == 0


@pytest.mark.parametrize("act", [None, "silu", "swiglu"])
@pytest.mark.parametrize("T,d,inter", [(2, 1800, 1800), (128, 9480, 264), (129, 9480, 264), (520, 4616, 520),
                                       (1400, 1800, 1800)])     # one-tile and two-tile row units, with one and with several units
def test_one_dense_expert_equals_its_steps(T, d, inter, act, native):
    gen = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=gen, device="cuda") * std).bfloat16()
    n1 = 2 * inter if act == "swiglu" else inter
    x, w1, w2 = leaves = [t.requires_grad_() for t in (mk(T, d), mk(1, d, n1, std=0.05), mk(1, inter, d, std=0.05))]
    grad = mk(T, d)
    out = dense_expert(*leaves, act)
    got = [out.detach()] + list(torch.autograd.grad(out, leaves, grad))
    with torch.no_grad():
        assert torch.equal(dense_expert(*leaves, act), got[0])
        plan = build_routing_plan(torch.zeros(T, 1, dtype=torch.int64, device="cuda"), 1, 1)
        maps = (plan.mtile_expert, plan.tile_pairs, plan.num_mtiles)
        new = lambda n: torch.empty(plan.padded_rows, n, dtype=x.dtype, device="cuda")
        xs, pre, hidden, ys, gs, d_pre, dxs = new(d), new(n1) if act else None, new(inter), new(d), new(d), new(n1), new(d)
        native.gather_rows(x, plan.row_src, plan.num_mtiles, xs, 1)
        native.gather_rows(grad, plan.row_src, plan.num_mtiles, gs, 1)
        native.mgrouped_gemm(xs, w1, hidden, pre, *maps, False, act, plan.status)
        native.mgrouped_gemm(hidden, w2, ys, None, *maps, False, None, plan.status)
        if act is None:
            native.mgrouped_gemm(gs, w2, d_pre, None, *maps, True, None, plan.status)
        else:
            native.mgrouped_gemm_dglu(gs, w2, pre, d_pre, *maps, act, plan.status)
        native.mgrouped_gemm(d_pre, w1, dxs, None, *maps, True, None, plan.status)
        dw1, dw2 = torch.empty_like(w1), torch.empty_like(w2)
        native.kgrouped_gemm(xs, d_pre, dw1, plan.pad_offsets, plan.status)
        native.kgrouped_gemm(hidden, gs, dw2, plan.pad_offsets, plan.status)
    for a, b in zip(got, (ys[:T], dxs[:T], dw1, dw2)):
        assert torch.equal(a, b)
    assert native.read_status(plan.status) == 0
