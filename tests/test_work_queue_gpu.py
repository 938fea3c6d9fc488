"""Passes whose contractions claim their work items against the same passes with the items dealt out: bit for bit, and again when
a contraction is launched once more without the kernel that zeroes the words the items are claimed from."""
import pytest
import torch

from moe_explore import _native
from moe_explore.expert_compute import routed_expert_compute
from moe_explore.triton_kernels.m_grouped_gemm import MGroupedGEMMParams, m_grouped_gemm

pytestmark = pytest.mark.gpu

ONCE = {"moe_expert_forward": _native.FWD_ROUTE | _native.FWD_DISPATCH, "moe_expert_backward": _native.BWD_FOLD,
        "moe_rows_gemm": _native.ROWS_LAYOUT}


@pytest.fixture
def launch(monkeypatch):
    real, how = _native.run_pass, {}

    def run_pass(name, p, steps, rows):
        if how["mode"] == "dealt out":
            p.counters = None
        real(name, p, steps, rows)
        if how["mode"] == "twice":
            real(name, p, [s for s in steps if not s[0] & ONCE[name]], rows)
    monkeypatch.setattr(_native, "run_pass", run_pass)
    return lambda mode: how.update(mode=mode)


@pytest.mark.parametrize("act,dtype", [("swiglu", torch.bfloat16), ("gelu", torch.float16)])
@pytest.mark.parametrize("T,E,spread", [(2000, 96, 1.0), (700, 128, 3.0), (9000, 96, 0.0)])   # some experts without a row at 3.0
def test_claimed_and_dealt_out_items(T, E, spread, act, dtype, launch, native):
    d, inter, k = 520, 1032, 4
    g = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(dtype)
    ids = torch.topk(torch.randn(T, E, generator=g, device="cuda") + spread * torch.randn(E, generator=g, device="cuda"), k).indices
    leaves = [mk(T, d), torch.rand(T, k, generator=g, device="cuda").to(dtype), mk(E, d, 2 * inter if act == "swiglu" else inter, std=0.1),
              mk(E, inter, d, std=0.1)]
    grad = mk(T, d)

    def run(mode):
        launch(mode)
        p = [t.clone().requires_grad_() for t in leaves]
        out = routed_expert_compute(*p, ids, E, k, act)
        got = [out.detach(), *torch.autograd.grad(out, p, grad)]
        with torch.no_grad():
            got.append(routed_expert_compute(*p, ids, E, k, act))
        groups = torch.bincount(ids.flatten(), minlength=E).cumsum(0).int()
        groups = torch.cat([groups.new_zeros(1), groups])
        got.append(m_grouped_gemm(mk(T * k, d) * 0 + 1, MGroupedGEMMParams(leaves[2], groups, None, False, False, T * k, 1)))
        return got

    ref = run("dealt out")
    for mode in ("claimed", "claimed", "twice"):
        assert all(torch.equal(a, b) for a, b in zip(run(mode), ref)), mode


def test_nothing_to_claim(launch, native):
    """Every id out of range: no row tile is in use, the words stay as they are."""
    from moe_explore.routing_plan import device_status

    T, E, d, inter = 3000, 96, 136, 1032
    x, w1, w2 = (torch.randn(*s, device="cuda").bfloat16() for s in ((T, d), (E, d, 2 * inter), (E, inter, d)))
    scores, ids = torch.ones(T, 2, device="cuda").bfloat16(), torch.full((T, 2), E, device="cuda")
    launch("twice")
    p = [t.requires_grad_() for t in (x, scores, w1, w2)]
    out = routed_expert_compute(*p, ids, E, 2, "swiglu")
    assert all(not t.any() for t in (out, *torch.autograd.grad(out, p, torch.ones_like(out))))
    assert native.read_status(device_status(), reset=True) == 100


def _every_launch_leaves_the_same(out, launch, launches):
    """``launch`` writes ``out``, again and again out of a graph, every time over NaN: a work item that was another one leaves them."""
    def once():
        out.fill_(float("nan"))
        launch()
    once()
    first = out.clone().view(torch.int64)
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(100):
            once()
            wrong += torch.ne(out.view(torch.int64), first).any()
    for _ in range(launches // 100):
        graph.replay()
    assert not out[0].isnan().any() and int(wrong) == 0


def _pass_of_many_items(E, rows, d, inter, native, **buffers):
    """``rows`` tokens per expert, one slot each, dispatched; with a word to claim items from."""
    from moe_explore.routing_plan import build_routing_plan

    T = E * rows
    ids = torch.arange(T, device="cuda").remainder(E).view(T, 1)
    plan = build_routing_plan(ids, E, 1)
    x = torch.randn(T, d, generator=torch.Generator(device="cuda").manual_seed(E), device="cuda").bfloat16()
    xs = torch.empty(plan.padded_rows, d, dtype=x.dtype, device="cuda")
    counters = torch.empty(4, dtype=torch.int32, device="cuda")
    p = _native.ExpertPass(num_tokens=T, padded_rows=plan.padded_rows, d=d, inter=inter, num_experts=E, topk=1, keep=1,
                           act=_native.ACT_CODES[None], x=x.data_ptr(), xs=xs.data_ptr(), counters=counters.data_ptr(),
                           **{n: getattr(plan, n).data_ptr() for n in ("group_indices", "pad_offsets", "row_src", "dst_row",
                                                                       "mtile_expert", "tile_pairs", "num_mtiles", "status")})
    _native.run_pass("moe_expert_forward", p, [(_native.FWD_DISPATCH, "rows:gather", 1)], T)
    return p, plan, (x, xs, counters)


def test_a_hundred_thousand_launches_of_claimed_rows(native):
    E, d, inter = 128, 64, 1544
    p, plan, held = _pass_of_many_items(E, 16, d, inter, native)
    w1 = torch.randn(E, d, inter, device="cuda").bfloat16()
    hidden = torch.empty(plan.padded_rows, inter, dtype=w1.dtype, device="cuda")
    p.w1, p.hidden = w1.data_ptr(), hidden.data_ptr()
    _every_launch_leaves_the_same(
        hidden, lambda: _native.run_pass("moe_expert_forward", p, [(_native.FWD_UP, "mgrouped_gemm:plain", 1)], E * 16), 100_000)
    assert native.read_status(plan.status) == 0


def test_a_hundred_thousand_launches_of_claimed_weight_gradients(native):
    E, d, inter = 192, 264, 264     # four items per expert, most of them a sliver of a tile
    p, plan, held = _pass_of_many_items(E, 16, d, inter, native)
    d_pre = torch.randn(plan.padded_rows, inter, device="cuda").bfloat16() * (plan.row_src >= 0)[:, None]
    d_w1 = torch.empty(E, d, inter, dtype=d_pre.dtype, device="cuda")
    p.d_pre, p.d_w1 = d_pre.data_ptr(), d_w1.data_ptr()
    _every_launch_leaves_the_same(
        d_w1, lambda: _native.run_pass("moe_expert_backward", p, [(_native.BWD_DW1, "kgrouped_gemm:dw1", 1)], E * 16), 100_000)
    assert native.read_status(plan.status) == 0
