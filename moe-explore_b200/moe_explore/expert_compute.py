"""The differentiable expert-compute step of the MoE layer on the native kernels.

forward : gate/up grouped GEMM with a fused GLU epilogue, its token rows either gathered by the GEMM's own
          operand loads (``gather_in_gemm``) or copied into the padded expert-sorted layout first -> down grouped
          GEMM -> weighted fold of the top-k slots (a separate deterministic kernel, or -- ``fused_combine``,
          forward-only -- scaled and added into the output by the down GEMM's epilogue).
backward: score-scaled gather of dOut (+ router-weight gradient as a row dot product) ->
          grouped GEMM against W2^T with the activation's derivative fused (GLU or plain) -> grouped GEMM against W1^T
          and an unweighted fold for dX -> two K-grouped GEMMs for the expert weight gradients.

The reference's forward is topk_moe_forward (src/moe_explore/functional/topk_moe.py:16-54);
it has no backward.  The gradients follow from out[t] = sum_s score[t,s] * (act(x_t W1[e]) W2[e]).
"""
from __future__ import annotations

import functools

import torch

from moe_explore import _native
from moe_explore.functional.activation import is_glu
from moe_explore.params import ErnieRouterParams, TopkRouterParams
from moe_explore.router import ernie_router, fused_topk_of_logits, nothing_watches, tail_in_one_kernel, topk_of_logits
from moe_explore.routing_plan import RoutingPlan, device_status, packed_layout


def _plan_pointers(plan: RoutingPlan):
    return tuple(t.data_ptr() for t in (plan.group_indices, plan.pad_offsets, plan.row_src, plan.dst_row, plan.mtile_expert,
                                        plan.tile_pairs, plan.num_mtiles, plan.status))


def _packed_pointers(base: int, offsets, status: torch.Tensor):
    return tuple(base + o for o in offsets) + (status.data_ptr(),)


class _Pass:
    """What the backward pass needs to know about its forward pass besides the saved tensors."""
    __slots__ = ("sizes", "routing", "act", "gathered", "scratch", "tail")


# Up to here the buffers of a pass are cut from one allocation, above each is one of its own.  An allocation costs the host 1.7 us
# and a pass had seven to twelve: with the router's tail in the same library call, one token takes 88 -> 58 us (the host is what
# it waits for), and the host issues a training pass of 64 MB (1777 tokens x 3 slots, 12 experts of 776 x 1544) in 250 us instead of
# 300.  Larger passes wait for the GPU, and one large block is harder to place than several.
SCRATCH_IN_ONE = 256 << 20


@functools.lru_cache(maxsize=256)
def _cuts(sizes):
    offsets, total = [], 0
    for n in sizes:
        offsets.append(total)
        total += (n + 255) // 256 * 256
    return tuple(offsets), total


def _buffers(sizes, device):
    """(tensors, addresses) of buffers of these many bytes (0: none, address None)."""
    offsets, total = _cuts(sizes)
    if total <= SCRATCH_IN_ONE:
        block = torch.empty(total, dtype=torch.uint8, device=device)
        tensors = (block,)
    else:
        tensors = tuple(torch.empty(n, dtype=torch.uint8, device=device) for n in sizes if n)
    return tensors, _addresses(sizes, tensors)


def _addresses(sizes, tensors):
    offsets, total = _cuts(sizes)
    if total <= SCRATCH_IN_ONE:
        base = tensors[0].data_ptr()
        return [base + o if n else None for o, n in zip(offsets, sizes)]
    rest = iter(tensors)
    return [next(rest).data_ptr() if n else None for n in sizes]


def _forward(x, scores, weight1, weight2, routing, act, gather_in_gemm: bool, fused_combine: bool, needs_grad: bool, addend=None,
             tail=None):
    """-> (out, _Pass, tensors to save).  ``tail`` = (logits, softmax before top-k, normalize, bias or None, fused router's tie rule):
    scores and expert indices are the router's tail of these logits, taken as part of the pass (``scores`` and the indices of
    ``routing`` are then None)."""
    _native.require_cuda(x, weight1, weight2)
    assert x.dim() == 2 and weight1.dim() == 3 and weight2.dim() == 3
    T, d = x.shape
    E, d1, n1 = weight1.shape
    inter = weight2.size(1)
    assert d1 == d and weight2.size(0) == E and weight2.size(2) == d, "weight shapes do not match the input"
    assert n1 == (2 * inter if is_glu(act) else inter), "weight1 width does not match weight2 and the activation"
    planned = isinstance(routing, RoutingPlan)
    flat = None
    if planned:
        topk = routing.topk
        assert routing.num_rows == T * topk and routing.num_experts == E
    else:
        indices, num_experts, topk = routing
        assert num_experts == E
        if tail is None:
            flat = indices.reshape(-1).contiguous()
            assert flat.numel() == T * topk
        else:
            assert tail[0].shape == (T, E) and tail[0].is_contiguous()
    x = x.contiguous()
    if tail is None:
        _native.require_cuda(scores)
        scores = scores.to(x.dtype).contiguous()
    weight1 = weight1.contiguous()
    weight2 = weight2.contiguous()
    code = _native.dtype_code(x.dtype)
    act_code = _native.ACT_CODES[act]
    rows = T * topk
    fold = not fused_combine or needs_grad   # the backward pass needs the per-slot rows for the router-weight gradient

    steps = []
    workspace = None
    if planned:
        rp, num_words = routing.padded_rows, 0
    else:
        rp, offsets, num_words = packed_layout(rows, E)
        launches = _native.routing_launches(rows, E)
        if launches > 1:
            workspace = torch.empty(max(_native.routing_workspace_bytes(rows, E), 16), dtype=torch.uint8, device=x.device)
        if tail is not None:
            steps.append((_native.FWD_TAIL, "router:topk", 1))
        steps.append((_native.FWD_ROUTE, "routing", launches))
    # index arrays, scores and indices of the tail, expert-sorted input, un-activated product (needed by the backward pass; not
    # kept for inference or without an activation), activated product, per-slot rows, words the contractions claim work items from
    scratch = (4 * num_words, 2 * rows if tail else 0, 8 * rows if tail else 0, 0 if gather_in_gemm else 2 * rp * d,
               2 * rp * n1 if act is not None and needs_grad else 0, 2 * rp * inter, 2 * rp * d if fold else 0,
               4 * _native.WORK_COUNTERS)
    buffers, (words, tail_scores, tail_ids, xs, pre_act, hidden, ys, counters) = _buffers(scratch, x.device)
    if planned:
        plan_ptrs = _plan_pointers(routing)
    else:
        plan_ptrs = _packed_pointers(words, offsets, device_status(x.get_device()))
    out = torch.empty(T, d, dtype=x.dtype, device=x.device)
    kind = "glu" if is_glu(act) else "plain"
    if not gather_in_gemm:
        steps.append((_native.FWD_DISPATCH, "rows:gather", 1))
    steps.append((_native.FWD_UP, "mgrouped_gemm:" + kind + ("+gather" if gather_in_gemm else ""), 1))
    if fold:
        steps.append((_native.FWD_DOWN, "mgrouped_gemm:plain", 1))
        steps.append((_native.FWD_FOLD, "rows:combine", 1))
    else:
        steps.append((_native.FWD_DOWN, "mgrouped_gemm:combine", 1))
    if addend is not None:
        assert fold and addend.shape == out.shape and addend.dtype is out.dtype and addend.is_cuda
        addend = addend.contiguous()
    ptr = _native._ptr
    ids = tail_ids if tail is not None else ptr(flat)
    p = _native.ExpertPass(
        T, rp, d, inter, E, topk, act_code, code, gather_in_gemm, not fold, needs_grad, 0, ids, x.data_ptr(),
        tail_scores if tail is not None else scores.data_ptr(), weight1.data_ptr(), weight2.data_ptr(), *plan_ptrs, ptr(workspace),
        0 if workspace is None else workspace.numel(), xs, pre_act, hidden, ys, out.data_ptr())
    p.addend, p.counters = ptr(addend), counters
    if tail is not None:
        p.logits, p.softmax_before_topk, p.normalize, p.router_bias = tail[0].data_ptr(), bool(tail[1]), int(tail[2]), ptr(tail[3])
        p.logits_dtype, p.own_tie_rule = _native.float_code(tail[0].dtype), tail[4]
    _native.run_pass("moe_expert_forward", p, steps, rows)
    if not needs_grad:
        return out, None, ()
    info = _Pass()
    info.sizes = (T, d, inter, E, topk, rp, n1)
    info.routing = routing if planned else None
    info.act = act
    info.gathered = bool(gather_in_gemm)
    info.scratch = scratch
    info.tail = tail is not None
    return out, info, (x if gather_in_gemm else None, scores, weight1, weight2, *buffers)


def _backward(info: _Pass, saved, grad_out, router=None):
    """-> (dx, d_scores, d_w1, d_w2[, dlogits]); ``router`` = (logits, router weight, expert indices or None where the pass took
    the router's tail) makes the router's tail and its share of dx part of the pass."""
    x, scores, weight1, weight2, *buffers = saved
    T, d, inter, E, topk, rp, n1 = info.sizes
    act = info.act
    rows = T * topk
    grad_out = grad_out.contiguous()
    words, tail_scores, tail_ids, xs, pre_act, hidden, ys, _ = _addresses(info.scratch, buffers)
    new = lambda *shape: torch.empty(shape, dtype=grad_out.dtype, device=grad_out.device)

    # score-scaled dOut rows, gradient of the un-activated product, per-slot rows of dX; with a router the gradient of the selected
    # logits in fp32 and the transposed router weight
    scratch = (2 * rp * d, 2 * rp * n1, 2 * rp * d, 4 * _native.WORK_COUNTERS) + \
        ((4 * rows, 2 * E * d) if router is not None else (0, 0))
    held, (gs, d_pre, dxs, counters, dl, router_t) = _buffers(scratch, grad_out.device)
    d_scores, dx = new(T, topk), new(T, d)
    d_w1, d_w2 = torch.empty_like(weight1), torch.empty_like(weight2)
    if info.routing is not None:
        plan_ptrs = _plan_pointers(info.routing)
    else:
        plan_ptrs = _packed_pointers(words, packed_layout(rows, E)[1], device_status(grad_out.get_device()))
    rows_in = x.data_ptr() if info.gathered else xs
    p = _native.ExpertPass(
        T, rp, d, inter, E, topk, _native.ACT_CODES[act], _native.dtype_code(grad_out.dtype), info.gathered, False, True, 0, None,
        rows_in, tail_scores if info.tail else scores.data_ptr(), weight1.data_ptr(), weight2.data_ptr(), *plan_ptrs, None, 0,
        rows_in, pre_act, hidden, ys, None, grad_out.data_ptr(), gs, d_scores.data_ptr(), d_pre, dxs, dx.data_ptr(),
        d_w1.data_ptr(), d_w2.data_ptr())
    p.counters = counters
    steps = [(_native.BWD_FOLD, "rows:combine_bwd", 1),
             (_native.BWD_DOWN, "mgrouped_gemm:wt" if act is None else "mgrouped_gemm:dglu", 1),
             (_native.BWD_UP, "mgrouped_gemm:wt", 1), (_native.BWD_FOLD_DX, "rows:combine", 1),
             (_native.BWD_DW1, "kgrouped_gemm:dw1" + ("+gather" if info.gathered else ""), 1),
             (_native.BWD_DW2, "kgrouped_gemm:dw2", 1)]
    dlogits = None
    if router is not None:
        logits, router_weight, indices = router
        dlogits = new(T, (E + 7) // 8 * 8)
        p.logits, p.router_w = logits.data_ptr(), router_weight.data_ptr()
        p.expert_idx = tail_ids if indices is None else indices.data_ptr()
        p.dl, p.dlogits, p.router_t = dl, dlogits.data_ptr(), router_t
        steps.insert(1, (_native.BWD_ROUTER, "router:bwd", 1))
    _native.run_pass("moe_expert_backward", p, steps, rows)
    return dx, d_scores, d_w1, d_w2, dlogits


class ExpertCompute(torch.autograd.Function):
    """``routing`` is a ``RoutingPlan``, or (expert indices [T, topk], num_experts, topk) to be routed as part of the pass: its
    index arrays then live in one allocation and one library call issues every launch.  ``addend`` [T, d] is added by the
    fold."""

    @staticmethod
    def forward(ctx, x, scores, weight1, weight2, routing, act: str, gather_in_gemm: bool, fused_combine: bool, addend=None):
        needs_grad = any(ctx.needs_input_grad[:4])
        out, ctx.info, saved = _forward(x, scores, weight1, weight2, routing, act, gather_in_gemm, fused_combine, needs_grad, addend)
        ctx.save_for_backward(*saved)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        if ctx.info is None:   # only the addend needed a gradient
            return (None,) * 8 + (grad_out,)
        return _backward(ctx.info, ctx.saved_tensors, grad_out)[:4] + (None,) * 4 + (grad_out if ctx.needs_input_grad[8] else None,)


class RoutedLayer(torch.autograd.Function):
    """The layer with a router whose softmax runs over the selected logits: scores and indices with the bits of ``topk_router`` (the
    router's tail as part of the pass, or its torch ops), their backward as part of the experts' backward pass.  The gradient of such
    logits is zero outside the selection, so the router's share of the input gradient is topk scaled rows of the transposed
    router weight, added by the fold in fp32, instead of a dense GEMM and an addition over [T, d]."""

    @staticmethod
    def forward(ctx, x, router_weight, weight1, weight2, router_params, num_experts: int, act: str, gather_in_gemm: bool, addend):
        logits = x @ router_weight
        if tail_in_one_kernel(logits, router_params.topk, x.dtype):
            scores = indices = None
            tail = (logits, router_params.softmax_before_topk, bool(router_params.normalize_routing), None, False)
        else:
            scores, indices = topk_of_logits(logits, router_params, x.dtype)
            indices, tail = indices.contiguous(), None
        out, ctx.info, saved = _forward(x, scores, weight1, weight2, (indices, num_experts, router_params.topk), act,
                                        gather_in_gemm, False, True, addend, tail)
        ctx.save_for_backward(x, logits, router_weight, indices, *saved)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        x, logits, router_weight, indices, *saved = ctx.saved_tensors
        dx, _, d_w1, d_w2, dlogits = _backward(ctx.info, saved, grad_out,
                                               (logits.contiguous(), router_weight.contiguous(), indices))
        d_router = None
        if ctx.needs_input_grad[1]:   # dlogits' rows are padded to whole 16 bytes
            d_router = (x.t() @ dlogits)[:, :router_weight.size(1)].contiguous()
        return dx, d_router, d_w1, d_w2, None, None, None, None, grad_out if ctx.needs_input_grad[8] else None


class DenseExpert(torch.autograd.Function):
    """act(x @ weight1[0]) @ weight2[0]: one expert that every token goes to with weight one.  No row is moved and nothing is
    folded; the grouped GEMMs read ``x`` and write the result where they are.  (As a top-1 layer it copied x, its
    result and both gradients once more: 160 of 18500 us at 8192 tokens of 14 KB.)"""

    @staticmethod
    def forward(ctx, x, weight1, weight2, act):
        _native.require_cuda(x, weight1, weight2)
        T, d = x.shape
        n1, inter = weight1.size(2), weight2.size(1)
        assert weight1.size(0) == 1 and weight2.size(0) == 1
        assert weight1.size(1) == d and weight2.size(2) == d, "weight shapes do not match the input"
        assert n1 == (2 * inter if is_glu(act) else inter), "weight1 width does not match weight2 and the activation"
        x, weight1, weight2 = x.contiguous(), weight1.contiguous(), weight2.contiguous()
        needs_grad = any(ctx.needs_input_grad[:3])
        rp, offsets, num_words = packed_layout(T, 1)
        words = torch.empty(num_words, dtype=torch.int32, device=x.device)
        groups = torch.arange(0, T + 1, T, dtype=torch.int32, device=x.device)   # {0, T}
        new = lambda *shape: torch.empty(shape, dtype=x.dtype, device=x.device)
        pre_act = new(rp, n1) if (act is not None and needs_grad) else None
        hidden, out = new(rp, inter), new(T, d)
        p = DenseExpert._pass(x, weight1, weight2, act, words, groups, offsets, rp, needs_grad)
        p.pre_act, p.hidden, p.out = _native._ptr(pre_act), hidden.data_ptr(), out.data_ptr()
        _native.run_pass("moe_expert_forward", p, [
            (_native.FWD_ROUTE, "routing", 1), (_native.FWD_UP, "mgrouped_gemm:" + ("glu" if is_glu(act) else "plain"), 1),
            (_native.FWD_DOWN, "mgrouped_gemm:plain", 1)], T)
        if needs_grad:
            ctx.act = act
            ctx.save_for_backward(x, weight1, weight2, pre_act, hidden, words, groups)
        return out

    @staticmethod
    def _pass(x, weight1, weight2, act, words, groups, offsets, rp, keep):
        group_ptr, *plan_ptrs = _packed_pointers(words.data_ptr(), offsets, device_status(x.get_device()))
        return _native.ExpertPass(
            x.size(0), rp, x.size(1), weight2.size(1), 1, 1, _native.ACT_CODES[act], _native.dtype_code(x.dtype), 0, 0, keep, 1,
            None, x.data_ptr(), None, weight1.data_ptr(), weight2.data_ptr(), groups.data_ptr(), *plan_ptrs)

    @staticmethod
    def backward(ctx, grad_out):
        x, weight1, weight2, pre_act, hidden, words, groups = ctx.saved_tensors
        T, d = x.shape
        rp, offsets, _ = packed_layout(T, 1)
        grad_out = grad_out.contiguous()
        d_pre = torch.empty(rp, weight1.size(2), dtype=x.dtype, device=x.device)
        dx, d_w1, d_w2 = torch.empty_like(x), torch.empty_like(weight1), torch.empty_like(weight2)
        p = DenseExpert._pass(x, weight1, weight2, ctx.act, words, groups, offsets, rp, True)
        p.pre_act, p.hidden, p.grad_out = _native._ptr(pre_act), hidden.data_ptr(), grad_out.data_ptr()
        p.d_pre, p.dx, p.d_w1, p.d_w2 = d_pre.data_ptr(), dx.data_ptr(), d_w1.data_ptr(), d_w2.data_ptr()
        _native.run_pass("moe_expert_backward", p, [
            (_native.BWD_DOWN, "mgrouped_gemm:wt" if ctx.act is None else "mgrouped_gemm:dglu", 1),
            (_native.BWD_UP, "mgrouped_gemm:wt", 1), (_native.BWD_DW1, "kgrouped_gemm:dw1", 1),
            (_native.BWD_DW2, "kgrouped_gemm:dw2", 1)], T)
        return dx, d_w1, d_w2, None


# Fusing the row gather into the gate/up GEMM's loads saves the copy of T*k rows into the expert-sorted layout
# (and, in training, keeps only the [T, d] input instead of the [R, d] copy for the weight1 gradient) -- but the 32
# four-row gather copies that replace one 128-row tile copy per stage cost ~95 cycles each on B200, which makes the
# gate/up GEMM 3.3x slower at the Mixtral shape (10.2 ms against 3.1 ms; the copy it saves takes 0.05 ms).  So the
# copy-first form is the default and the fused gather is for callers that are short of memory.
GATHER_IN_GEMM_DEFAULT = False


def expert_compute(x, scores, weight1, weight2, plan: RoutingPlan, act, gather_in_gemm=None,
                   fused_combine: bool = False) -> torch.Tensor:
    """out[t] = sum_s scores[t,s] * (act(x[t] @ weight1[e]) @ weight2[e]),  e = expert of (t, s).

    ``gather_in_gemm``: token rows are gathered by the gate/up GEMM's operand loads (tile::gather4) instead of being
    copied into the expert-sorted layout first (None = the package default).  ``fused_combine``: when no gradient
    is needed, the down GEMM's epilogue multiplies each row by its router weight and adds it into the output
    (vector reductions; the order of the k additions is not fixed, so the result is not bit-reproducible);
    ignored when a gradient is required."""
    if gather_in_gemm is None:
        gather_in_gemm = GATHER_IN_GEMM_DEFAULT
    return ExpertCompute.apply(x, scores, weight1, weight2, plan, None if act is None else str(act), bool(gather_in_gemm),
                               bool(fused_combine), None)


def dense_expert(x, weight1, weight2, act) -> torch.Tensor:
    """One expert for every token: ``weight1`` [1, d, I or 2I], ``weight2`` [1, I, d]."""
    return DenseExpert.apply(x, weight1, weight2, None if act is None else str(act))


def routed_expert_compute(x, scores, weight1, weight2, indices, num_experts: int, topk: int, act, gather_in_gemm=None,
                          fused_combine: bool = False, addend=None) -> torch.Tensor:
    """``expert_compute`` of a routing decision given as expert indices (int64 [T, topk]) instead of a plan; ``addend`` (like the
    output, not with ``fused_combine``) is added to the result."""
    _native.require_cuda(indices)
    assert indices.dtype is torch.int64, "expert indices must be int64 (what torch.topk returns)"
    if gather_in_gemm is None:
        gather_in_gemm = GATHER_IN_GEMM_DEFAULT
    return ExpertCompute.apply(x, scores, weight1, weight2, (indices, num_experts, topk), None if act is None else str(act),
                               bool(gather_in_gemm), bool(fused_combine), addend)


_PLAIN = (torch.Tensor, torch.nn.Parameter)
# Up to here the router joins the pass.  What that costs is topk scaled rows per token in the fold of dX instead of a dense GEMM
# whose result the fold adds (us, fold with the rows / GEMM + fold with the result: 16384 tokens x 4 of 4 KB 71 / 90, 8192 x 2 of
# 8 KB 42 / 68, 4096 x 6 of 8 KB 69 / 74, 8192 x 8 of 4 KB 77 / 78, 8192 x 8 of 14 KB 235 / 225); it grows with topk, the GEMM does
# not.  What it saves is the router's seven element-wise launches.  Whole training passes with 8 slots and 64 experts, joined / not:
# 128 tokens of 4 KB 572 / 603, 1024 of 4 KB 682 / 716, 1024 of 14 KB 4563 / 4747, and equal within 4 % of spread at 8192 tokens
# (4 KB 2764 / 2798, 14 KB 18782 / 18590).  More slots were not measured and keep the composed form.
ROUTER_ROWS_IN_FOLD = 8


def router_joins_the_pass(x, router_params, num_experts: int, topk: int) -> bool:
    """Whether ``routed_layer`` stands for the router as well: plain 16-bit CUDA tensors, softmax over the selected logits, a
    gradient wanted.  Everything else (softmax over all experts has a dense gradient; autocast, mixed types, tensor
    subclasses and the fp32 router are torch's business) goes through the router's torch ops."""
    if type(router_params) is not TopkRouterParams or router_params.softmax_before_topk or not torch.is_grad_enabled():
        return False
    w = router_params.router_weight
    return (type(x) in _PLAIN and type(w) in _PLAIN and (x.requires_grad or w.requires_grad) and x.is_cuda and w.is_cuda
            and x.dtype in (torch.bfloat16, torch.float16) and w.dtype is x.dtype and x.dim() == 2 and w.dim() == 2
            and x.size(0) > 0 and w.size(1) == num_experts and router_params.topk == topk and topk <= ROUTER_ROWS_IN_FOLD
            and not torch.is_autocast_enabled("cuda"))


def routed_layer(x, router_params, weight1, weight2, num_experts: int, act, gather_in_gemm=None, addend=None) -> torch.Tensor:
    """Router and experts in one differentiable step (see ``router_joins_the_pass``)."""
    if gather_in_gemm is None:
        gather_in_gemm = GATHER_IN_GEMM_DEFAULT
    return RoutedLayer.apply(x, router_params.router_weight, weight1, weight2, router_params, num_experts,
                             None if act is None else str(act), bool(gather_in_gemm), addend)


def router_and_experts_at_once(x, router_params, weight1, weight2, num_experts: int, topk: int, addend=None) -> bool:
    """Whether ``inference_pass`` stands for router and experts: plain 16-bit CUDA tensors and nothing that has to see the single
    steps (no gradient, no transform, no tracing, no mode)."""
    if type(router_params) not in (TopkRouterParams, ErnieRouterParams):
        return False
    tensors = (x, router_params.router_weight, weight1, weight2) + (() if addend is None else (addend,))
    if not all(type(t) in _PLAIN and t.is_cuda for t in tensors):
        return False
    if torch.is_grad_enabled() and any(t.requires_grad for t in tensors):
        return False
    return (x.dtype in (torch.bfloat16, torch.float16) and x.dim() == 2 and x.size(0) > 0
            and router_params.router_weight.dim() == 2 and router_params.router_weight.size(1) == num_experts
            and router_params.topk == topk and nothing_watches(x))


def inference_pass(x, router_params, weight1, weight2, num_experts: int, topk: int, act, gather_in_gemm=None,
                   fused_combine: bool = False, addend=None, fused_router: bool = False) -> torch.Tensor:
    """Router and experts without gradients: one allocation besides the result and the logits, and one library call after the
    logits' GEMM."""
    if gather_in_gemm is None:
        gather_in_gemm = GATHER_IN_GEMM_DEFAULT
    scores = indices = tail = None
    if type(router_params) is ErnieRouterParams:
        assert router_params.router_weight.dtype is torch.float32
        with torch.autocast(device_type="cuda", enabled=False):
            logits = x.float() @ router_params.router_weight
        if tail_in_one_kernel(logits, router_params.topk, x.dtype, router_params.bias):
            tail = (logits, True, 2, router_params.bias, False)
        else:
            scores, indices = ernie_router(x, router_params)
    else:
        logits = x @ router_params.router_weight
        if tail_in_one_kernel(logits, router_params.topk, x.dtype):
            tail = (logits, router_params.softmax_before_topk, bool(router_params.normalize_routing), None, fused_router)
        elif fused_router:
            scores, indices = fused_topk_of_logits(logits, router_params)
        else:
            scores, indices = topk_of_logits(logits, router_params, x.dtype)
    # (topk is the layer's: the router's may be anything that torch.topk takes and that equals it)
    return _forward(x, scores, weight1, weight2, (indices, num_experts, topk), None if act is None else str(act),
                    bool(gather_in_gemm), bool(fused_combine), False, addend, tail)[0]
