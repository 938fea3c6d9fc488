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

import torch

from moe_explore import _native
from moe_explore.functional.activation import is_glu
from moe_explore.routing_plan import RoutingPlan, device_status, packed_layout


def _plan_pointers(plan: RoutingPlan):
    return tuple(t.data_ptr() for t in (plan.group_indices, plan.pad_offsets, plan.row_src, plan.dst_row, plan.mtile_expert,
                                        plan.tile_pairs, plan.num_mtiles, plan.status))


def _packed_pointers(words: torch.Tensor, offsets, status: torch.Tensor):
    base = words.data_ptr()
    return tuple(base + o for o in offsets) + (status.data_ptr(),)


class ExpertCompute(torch.autograd.Function):
    """``routing`` is a ``RoutingPlan``, or (expert indices [T, topk], num_experts, topk) to be routed as part of the pass: its
    index arrays then live in one allocation and one library call issues every launch."""

    @staticmethod
    def forward(ctx, x, scores, weight1, weight2, routing, act: str, gather_in_gemm: bool, fused_combine: bool):
        _native.require_cuda(x, scores, weight1, weight2)
        assert x.dim() == 2 and weight1.dim() == 3 and weight2.dim() == 3
        T, d = x.shape
        E, d1, n1 = weight1.shape
        inter = weight2.size(1)
        assert d1 == d and weight2.size(0) == E and weight2.size(2) == d, "weight shapes do not match the input"
        assert n1 == (2 * inter if is_glu(act) else inter), "weight1 width does not match weight2 and the activation"
        planned = isinstance(routing, RoutingPlan)
        if planned:
            topk = routing.topk
            assert routing.num_rows == T * topk and routing.num_experts == E
        else:
            indices, num_experts, topk = routing
            flat = indices.reshape(-1).contiguous()
            assert flat.numel() == T * topk and num_experts == E
        x = x.contiguous()
        scores = scores.to(x.dtype).contiguous()
        weight1 = weight1.contiguous()
        weight2 = weight2.contiguous()
        code = _native.dtype_code(x.dtype)
        act_code = _native.ACT_CODES[act]
        rows = T * topk
        new = lambda *shape: torch.empty(shape, dtype=x.dtype, device=x.device)
        needs_grad = any(ctx.needs_input_grad[:4])
        fold = not fused_combine or needs_grad   # the backward pass needs the per-slot rows for the router-weight gradient

        steps = []
        words = workspace = None
        if planned:
            rp = routing.padded_rows
            ids = None
            plan_ptrs = _plan_pointers(routing)
        else:
            rp, offsets, num_words = packed_layout(rows, E)
            words = torch.empty(num_words, dtype=torch.int32, device=x.device)
            status = device_status(x.get_device())
            plan_ptrs = _packed_pointers(words, offsets, status)
            ids = flat.data_ptr()
            if rows > _native.ROUTE_ONE_LAUNCH_ROWS:
                workspace = torch.empty(max(_native.routing_workspace_bytes(rows, E), 16), dtype=torch.uint8, device=x.device)
            steps.append((_native.FWD_ROUTE, "routing", 1 if workspace is None else 3))
        xs = None if gather_in_gemm else new(rp, d)
        # the un-activated product, needed by the backward pass (not kept for inference or without an activation)
        pre_act = new(rp, n1) if (act is not None and needs_grad) else None
        hidden = new(rp, inter)
        ys = new(rp, d) if fold else None
        out = new(T, d)
        kind = "glu" if is_glu(act) else "plain"
        if not gather_in_gemm:
            steps.append((_native.FWD_DISPATCH, "rows:gather", 1))
        steps.append((_native.FWD_UP, "mgrouped_gemm:" + kind + ("+gather" if gather_in_gemm else ""), 1))
        if fold:
            steps.append((_native.FWD_DOWN, "mgrouped_gemm:plain", 1))
            steps.append((_native.FWD_FOLD, "rows:combine", 1))
        else:
            steps.append((_native.FWD_DOWN, "mgrouped_gemm:combine", 1))
        ptr = _native._ptr
        _native.run_pass("moe_expert_forward", _native.ExpertPass(
            T, rp, d, inter, E, topk, act_code, code, gather_in_gemm, not fold, needs_grad, ids, x.data_ptr(), scores.data_ptr(),
            weight1.data_ptr(), weight2.data_ptr(), *plan_ptrs, ptr(workspace),
            0 if workspace is None else workspace.numel(), ptr(xs), ptr(pre_act), hidden.data_ptr(), ptr(ys), out.data_ptr()),
            steps, rows)
        if needs_grad:
            ctx.sizes = (T, d, inter, E, topk, rp, n1)
            ctx.routing = routing if planned else None
            ctx.act = act
            ctx.gathered = bool(gather_in_gemm)
            ctx.save_for_backward(x if gather_in_gemm else xs, pre_act, hidden, ys, scores, weight1, weight2, words)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        xs, pre_act, hidden, ys, scores, weight1, weight2, words = ctx.saved_tensors
        T, d, inter, E, topk, rp, n1 = ctx.sizes
        act = ctx.act
        rows = T * topk
        grad_out = grad_out.contiguous()
        new = lambda *shape: torch.empty(shape, dtype=grad_out.dtype, device=grad_out.device)

        gs, d_scores, d_pre, dxs, dx = new(rp, d), new(T, topk), new(rp, n1), new(rp, d), new(T, d)
        d_w1, d_w2 = torch.empty_like(weight1), torch.empty_like(weight2)
        if ctx.routing is not None:
            plan_ptrs = _plan_pointers(ctx.routing)
        else:
            plan_ptrs = _packed_pointers(words, packed_layout(rows, E)[1], device_status(words.get_device()))
        ptr = _native._ptr
        _native.run_pass("moe_expert_backward", _native.ExpertPass(
            T, rp, d, inter, E, topk, _native.ACT_CODES[act], _native.dtype_code(grad_out.dtype), ctx.gathered, False, True, None,
            xs.data_ptr(), scores.data_ptr(), weight1.data_ptr(), weight2.data_ptr(), *plan_ptrs, None, 0, xs.data_ptr(),
            ptr(pre_act), hidden.data_ptr(), ys.data_ptr(), None, grad_out.data_ptr(), gs.data_ptr(), d_scores.data_ptr(),
            d_pre.data_ptr(), dxs.data_ptr(), dx.data_ptr(), d_w1.data_ptr(), d_w2.data_ptr()),
            [(_native.BWD_FOLD, "rows:combine_bwd", 1),
             (_native.BWD_DOWN, "mgrouped_gemm:wt" if act is None else "mgrouped_gemm:dglu", 1),
             (_native.BWD_UP, "mgrouped_gemm:wt", 1), (_native.BWD_FOLD_DX, "rows:combine", 1),
             (_native.BWD_DW1, "kgrouped_gemm:dw1" + ("+gather" if ctx.gathered else ""), 1),
             (_native.BWD_DW2, "kgrouped_gemm:dw2", 1)], rows)
        return dx, d_scores, d_w1, d_w2, None, None, None, None


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
                               bool(fused_combine))


def routed_expert_compute(x, scores, weight1, weight2, indices, num_experts: int, topk: int, act, gather_in_gemm=None,
                          fused_combine: bool = False) -> torch.Tensor:
    """``expert_compute`` of a routing decision given as expert indices (int64 [T, topk]) instead of a plan."""
    _native.require_cuda(indices)
    assert indices.dtype is torch.int64, "expert indices must be int64 (what torch.topk returns)"
    if gather_in_gemm is None:
        gather_in_gemm = GATHER_IN_GEMM_DEFAULT
    return ExpertCompute.apply(x, scores, weight1, weight2, (indices, num_experts, topk), None if act is None else str(act),
                               bool(gather_in_gemm), bool(fused_combine))
