"""Row kernels at the edges of their thread splits: row widths around 32 / 64 / 128 sixteen-byte pieces, slot counts around the
powers of two their loads are grouped by, one to a few hundred tokens, dropped slots."""
import pytest
import torch

from moe_explore.expert_permute import expert_input_permute, expert_output_permute
from moe_explore.routing_plan import build_routing_plan

pytestmark = pytest.mark.gpu

WIDTHS = [8, 256, 264, 512, 520, 1024, 1032, 2056, 7168]


def _case(T, k, cols, E=7, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(T * 1000 + k * 100 + cols)
    idx = torch.stack([torch.randperm(max(E, k), generator=g, device="cuda")[:k] for _ in range(T)])
    if T > 2:
        idx[T // 2, 0] = 10_000   # out of range: dropped by the routing metadata
    plan = build_routing_plan(idx, max(E, k), k)
    plan.status.zero_()
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)
    return plan, mk(T, cols), mk(T, k), mk(plan.padded_rows, cols)


@pytest.mark.parametrize("cols", WIDTHS)
@pytest.mark.parametrize("T,k", [(1, 1), (3, 2), (33, 3), (130, 4), (7, 5), (129, 8), (5, 9)])
def test_rows_against_torch(T, k, cols, native):
    plan, x, scores, ys = _case(T, k, cols)
    dst = plan.dst_row.long()
    live = dst >= 0
    rows = int(plan.num_mtiles[0]) * 128
    # dispatch: copies, so exact; padding rows zero, or untouched
    expect = torch.zeros(plan.padded_rows, cols, dtype=x.dtype, device="cuda")
    expect[dst[live]] = x.repeat_interleave(k, 0)[live]
    xs = torch.full_like(expect, 7.0)
    native.dispatch_rows(x, plan.dst_row, plan.row_src, plan.num_mtiles, xs, k)
    assert torch.equal(xs[:rows], expect[:rows]) and bool((xs[rows:] == 7).all())
    only = torch.full_like(expect, 7.0)
    native.dispatch_rows_only(x, plan.dst_row, only, k)
    pads = plan.row_src[:rows] < 0
    assert torch.equal(only[:rows][~pads], expect[:rows][~pads]) and bool((only[:rows][pads] == 7).all())
    # gathers
    again = torch.full_like(expect, 7.0)
    native.gather_rows(x, plan.row_src, plan.num_mtiles, again, k)
    assert torch.equal(again[:rows], expect[:rows]) and bool((again[rows:] == 7).all())
    out = torch.empty(T * k, cols, dtype=x.dtype, device="cuda")
    native.unpad_rows(ys, plan.dst_row, out)
    assert torch.equal(out, torch.where(live[:, None], ys[dst.clamp_min(0)], torch.zeros_like(out)))
    native.index_rows(x, plan.perm, out, div=k)
    assert torch.equal(out, torch.where(plan.perm[:, None] >= 0, x[plan.perm.clamp_min(0) // k], torch.zeros_like(out)))
    # folds: fp32 sums of exact products, one rounding (half a unit in the last place of 8 bits; sums differ in order by
    # k * 2^-24 of the sum of magnitudes)
    picked = torch.where(live[:, None], ys[dst.clamp_min(0)], torch.zeros_like(out)).float().view(T, k, cols)
    for s in (scores, None):
        terms = picked if s is None else picked * s.float()[..., None]
        fold = torch.empty(T, cols, dtype=x.dtype, device="cuda")
        native.combine_topk(ys, s, plan.dst_row, fold, k)
        bound = terms.sum(1).abs() * 2.0 ** -8 + k * 2.0 ** -23 * terms.abs().sum(1)
        assert bool(((fold.float() - terms.sum(1)).abs() <= bound).all())
    # backward fold: the token-order kernel is the padded-order kernel bit for bit, and zero where a slot was dropped
    gs, gs2 = torch.full_like(ys, 7.0), torch.full_like(ys, 7.0)
    ds, ds2 = torch.full_like(scores, 7.0), torch.zeros_like(scores)
    native.combine_bwd_tokens(x, scores, ys, plan.dst_row, plan.row_src, plan.num_mtiles, gs, ds, k)
    native.combine_bwd(x, scores, ys, plan.row_src, plan.num_mtiles, gs2, ds2, k)
    assert torch.equal(gs, gs2) and torch.equal(ds, ds2)


@pytest.mark.parametrize("T,k,cols", [(1, 1, 8), (65, 3, 520), (700, 8, 2048)])
def test_permute_round_trip_with_and_without_a_score_gradient(T, k, cols, native):
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, cols, generator=g, device="cuda").bfloat16()
    idx = torch.stack([torch.randperm(16, generator=g, device="cuda")[:k] for _ in range(T)])
    scores = torch.rand(T, k, generator=g, device="cuda").bfloat16()
    grouped = expert_input_permute(x, idx, 16, k)
    order = torch.sort(idx.reshape(-1), stable=True).indices
    assert torch.equal(grouped.indices, order) and torch.equal(grouped.tokens, x[order // k])
    out = expert_output_permute(grouped, scores, k, x.shape)
    leaf = scores.clone().requires_grad_()
    out_grad = expert_output_permute(grouped, leaf, k, x.shape)   # through the un-permuted copy
    assert torch.equal(out, out_grad) and not out.requires_grad
    out_grad.backward(x)
    ref = (x.float()[:, None, :] * x.float()[:, None, :].expand(T, k, cols)).sum(-1)
    # fp32 sum of `cols` products, rounded once to bf16
    assert bool(((leaf.grad.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + cols * 2.0 ** -23 * ref.abs()).all())


@pytest.mark.parametrize("cols", [8, 520, 2056])
def test_every_negative_index_is_a_zero_row(cols, native):
    """-1, -2 and any other negative index, in 32 and 64 bits (where the low half may be positive): a row of zeros."""
    from moe_explore.expert_permute import row_gather

    g = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn(40, cols, generator=g, device="cuda").bfloat16()
    idx = torch.randint(0, 40, (300,), generator=g, device="cuda")
    idx[::7] = torch.tensor([-1, -2, -3, -2 ** 31], device="cuda").repeat(11)[:43]
    expect = lambda i, div: torch.where(i[:, None] >= 0, x[i.clamp_min(0) // div], torch.zeros((), dtype=x.dtype, device="cuda"))
    assert torch.equal(row_gather(x, idx), expect(idx, 1))
    rows = torch.full((384, cols), 7.0, device="cuda").bfloat16()
    native.gather_rows(x, torch.cat([idx, idx[:84]]).int(), torch.tensor([3, 2, 3, 0], dtype=torch.int32, device="cuda"), rows, 3)
    assert torch.equal(rows, expect(torch.cat([idx, idx[:84]]), 3))
    idx[5:9] = torch.tensor([-2 ** 32 + 1, -2 ** 32, -2 ** 62, -2 ** 33 + 7], device="cuda")
    for div in (1, 3):
        out = torch.full((300, cols), 7.0, device="cuda").bfloat16()
        native.index_rows(x, idx, out, div=div)
        assert torch.equal(out, expect(idx, div))


@pytest.mark.parametrize("act", [None, "swiglu"])
@pytest.mark.parametrize("gather,scatter", [(True, False), (True, True), (False, True)])
def test_functional_gemm_with_negative_positions(gather, scatter, act, native):
    """Negative entries of permute_indices: a zero input row with gather, no output row with scatter."""
    from moe_explore.triton_kernels.m_grouped_gemm import MGroupedGEMMParams, m_grouped_gemm

    rows = (70, 0, 129, 1, 300)
    R, K, N = sum(rows), 136, 208
    g = torch.Generator(device="cuda").manual_seed(R)
    groups = torch.tensor([0] + list(rows), dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    w = (torch.randn(len(rows), K, N, generator=g, device="cuda") * 0.1).bfloat16()
    x = torch.randn(R, K, generator=g, device="cuda").bfloat16()
    perm = torch.randperm(R, generator=g, device="cuda")
    bad = torch.arange(0, R, 9, device="cuda")
    holes = perm.clone()
    holes[bad] = torch.tensor([-1, -2, -7, -2 ** 32 + 3], device="cuda").repeat(R)[:bad.numel()]

    def run(p):
        del_me = [torch.full((n << 18,), float("nan"), device="cuda") for n in (1, 1, 2, 4)]
        del del_me
        return m_grouped_gemm(x, MGroupedGEMMParams(w, groups, p, gather, scatter, R, 1, activation=act))

    full, out = run(perm), run(holes)
    if scatter:
        stored = perm[(holes >= 0).nonzero().flatten()]
        assert torch.equal(out[stored], full[stored])
    else:
        full[bad] = 0
        assert torch.equal(out, full)


@pytest.mark.parametrize("T,k,cols", [(2, 1, 8), (65, 3, 520), (700, 8, 2048)])
def test_permute_round_trip_with_dropped_slots(T, k, cols, native):
    """Ids outside [0, E) leave -1 at the tail of the permutation: such slots add nothing, all others are exact, with and
    without a gradient of the scores."""
    from moe_explore.expert_permute import row_scatter

    E = 16
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, cols, generator=g, device="cuda").bfloat16()
    idx = torch.stack([torch.randperm(E, generator=g, device="cuda")[:k] for _ in range(T)])
    idx[0, 0], idx[T // 2, k - 1], idx[T - 1, k // 2] = E, -3, 10 ** 9
    dropped = (idx < 0) | (idx >= E)
    scores = torch.rand(T, k, generator=g, device="cuda").bfloat16()
    poison = [torch.full((n << 10,), 0x7FFFFFFF, dtype=torch.int32, device="cuda") for n in (1, 1, 2, 4, 8, 16, 64)]
    del poison
    grouped = expert_input_permute(x, idx, E, k)
    flat = scores.masked_fill(dropped, 0)
    # fp32 sum of k exact products, rounded once
    terms = x.float()[:, None, :] * flat.float()[..., None]
    bound = terms.sum(1).abs() * 2.0 ** -8 + k * 2.0 ** -23 * terms.abs().sum(1)
    leaf = scores.clone().requires_grad_()
    out, out_grad = (expert_output_permute(grouped, s, k, x.shape) for s in (scores, leaf))
    assert bool(((out.float() - terms.sum(1)).abs() <= bound).all()) and torch.equal(out, out_grad)
    out_grad.backward(x)
    assert not leaf.grad[dropped].any() and bool(leaf.grad[~dropped].any()) == bool((~dropped).any())
    rows = row_scatter(grouped.tokens, grouped.indices)
    assert torch.equal(rows, x.repeat_interleave(k, 0).masked_fill(dropped.reshape(-1, 1), 0))
    assert native.read_status(build_routing_plan(idx, E, k).status, reset=True) == 100


@pytest.mark.parametrize("rows", [1, 255, 256, 257, 70000])
def test_inverse_rows(rows, native):
    from moe_explore.routing_plan import device_status

    g = torch.Generator(device="cuda").manual_seed(rows)
    index = torch.randperm(rows, generator=g, device="cuda")
    index[::5] = -1 - index[::5]
    out = torch.full((rows,), 7, dtype=torch.int32, device="cuda")
    native.read_status(device_status(), reset=True)
    native.inverse_rows(index, out, device_status())
    expect = torch.full_like(out, -1)
    live = index >= 0
    expect[index[live]] = torch.arange(rows, dtype=torch.int32, device="cuda")[live]
    assert torch.equal(out, expect) and native.read_status(device_status()) == 0
    index[0] = rows   # (was negative) one past the end: named in the status word, written nowhere
    native.inverse_rows(index, out, device_status())
    assert torch.equal(out, expect) and native.read_status(device_status(), reset=True) == 5


@pytest.mark.parametrize("cols", [8, 256, 264, 1000, 2048])
@pytest.mark.parametrize("rows", [(1, 63, 64, 65, 0, 127), (700, 1000) * 80])     # fewer 64-row blocks than warps, and more
def test_padding_rows_and_only_they_are_zeroed(rows, cols, native):
    from moe_explore.routing_plan import plan_from_groups

    groups = torch.tensor((0,) + rows, dtype=torch.int32).cumsum(0).int().cuda()
    plan = plan_from_groups(groups, sum(rows))
    used = int(plan.num_mtiles[0]) * 128
    buf = torch.ones(used + 128, cols, dtype=torch.bfloat16, device="cuda")
    native.zero_padding_rows(plan.row_src, plan.num_mtiles, buf)
    expect = (plan.row_src[:used] >= 0).to(buf.dtype)[:, None].expand(used, cols)
    assert torch.equal(buf[:used], expect) and bool((buf[used:] == 1).all())
