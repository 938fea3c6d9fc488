"""Token -> expert routing.

Defined by torch ops: the reference computes its routing with the same ops (src/moe_explore/router.py:9-54), so running
them on the same device gives bit-identical top-k indices and scores, which the expert-compute kernels downstream depend
on.  Where nothing is differentiated or traced, one kernel takes the place of the ops after the linear layer and leaves the
same bits (``moe_router_tail``).  ``torch.compile`` decoration is dropped (no tracing compiler on this path).
"""
from __future__ import annotations

import torch
import torch.nn.functional as F
from torch.autograd import forward_ad

from moe_explore import _native
from moe_explore.params import ErnieRouterParams, RouterParams, TopkRouterParams


def softmax(x: torch.Tensor) -> torch.Tensor:
    """fp32 softmax over the last dim (router.py:5-7)."""
    return F.softmax(x, dim=-1, dtype=torch.float32)


def router(input: torch.Tensor, params: RouterParams):
    """Dispatch on the parameter type (router.py:9-15). Returns (scores [T,k], indices [T,k] int64)."""
    if isinstance(params, TopkRouterParams):
        return topk_router(input, params)
    if isinstance(params, ErnieRouterParams):
        return ernie_router(input, params)
    raise ValueError(f"Unsupported router type: {type(params)}")


def topk_router(input: torch.Tensor, router_params: TopkRouterParams):
    """Linear logits -> (softmax ->) top-k (-> softmax over the k) (-> renormalise) (router.py:17-35)."""
    return topk_of_logits(input @ router_params.router_weight, router_params, input.dtype)


def topk_of_logits(logits: torch.Tensor, router_params: TopkRouterParams, dtype: torch.dtype):
    """Everything of ``topk_router`` after the linear layer."""
    if tail_in_one_kernel(logits, router_params.topk, dtype):
        return _native.router_tail(logits, router_params.topk, bool(router_params.softmax_before_topk),
                                   bool(router_params.normalize_routing))
    if router_params.softmax_before_topk:
        logits = softmax(logits)
    scores, indices = torch.topk(logits, k=router_params.topk, dim=-1, sorted=False)
    if not router_params.softmax_before_topk:
        scores = softmax(scores)
    if router_params.normalize_routing:
        scores = scores / scores.sum(dim=-1, keepdim=True)
    return scores.to(dtype), indices


def _only_default_devices() -> bool:
    """The torch function modes in force are at most those of ``torch.set_default_device`` and ``with torch.device(...)``: they
    choose where factory calls without a device allocate, and the calls here name theirs."""
    return (torch._C._len_torch_function_stack() == 0
            or all(type(m) is torch.utils._device.DeviceContext for m in torch.overrides._get_current_function_mode_stack()))


def nothing_watches(*tensors: torch.Tensor) -> bool:
    """No transform, tracer or mode has to see the single ops on these tensors, and they lie on the current device.  (Some of the
    names are private to torch: one that is missing means that something may watch.)"""
    if torch.compiler.is_compiling():   # first: the names below are not traceable, and a graph without breaks may be wanted
        return False
    try:
        return (forward_ad._current_level < 0 and not any(map(torch._C._functorch.is_functorch_wrapped_tensor, tensors))
                and torch._C._len_torch_dispatch_stack() == 0 and _only_default_devices() and not torch.jit.is_tracing()
                and all(t.get_device() == torch.cuda.current_device() for t in tensors))
    except AttributeError:
        return False


def tail_in_one_kernel(logits: torch.Tensor, topk, dtype: torch.dtype, bias=None) -> bool:
    """Plain logits in the result's type (with a bias: in fp32), without a gradient, that nothing watches.  (One token to 16384 x 60
    experts: 2 to 8 us for what takes 10 to 48 in four to six launches.)"""
    if bias is not None and not (type(bias) in (torch.Tensor, torch.nn.Parameter) and bias.dtype is torch.float32
                                 and bias.get_device() == logits.get_device() and bias.dim() == 1
                                 and bias.size(0) == logits.size(-1) and bias.is_contiguous()):
        return False
    return (type(logits) is torch.Tensor and logits.is_cuda and logits.dtype is (dtype if bias is None else torch.float32)
            and dtype in (torch.bfloat16, torch.float16, torch.float32) and logits.dim() == 2 and logits.size(0) > 0
            and type(topk) is int and 0 < topk <= min(logits.size(1), _native.ROUTER_TAIL_TOPK)
            and logits.size(1) <= _native.ROUTER_TAIL_EXPERTS and logits.is_contiguous()
            and not (logits.requires_grad and torch.is_grad_enabled())
            and (nothing_watches(logits) if bias is None else nothing_watches(logits, bias)))


class _FusedTopk(torch.autograd.Function):
    """scores, indices = fused router tail of ``logits``; differentiable with respect to the logits."""

    @staticmethod
    def forward(ctx, logits, topk, softmax_before_topk, normalize_routing):
        from moe_explore import _native

        scores, indices, _ = _native.router_topk(logits, topk, softmax_before_topk, normalize_routing)
        ctx.save_for_backward(logits, indices)
        ctx.cfg = (softmax_before_topk, normalize_routing)
        ctx.mark_non_differentiable(indices)
        return scores, indices

    @staticmethod
    def backward(ctx, d_scores, _d_indices):
        # the scores as a differentiable torch function of the logits GIVEN the selection (gather, not top-k)
        logits, indices = ctx.saved_tensors
        softmax_before_topk, normalize_routing = ctx.cfg
        with torch.enable_grad():
            leaf = logits.detach().requires_grad_(True)
            if softmax_before_topk:
                picked = torch.gather(softmax(leaf), -1, indices)
            else:
                picked = softmax(torch.gather(leaf, -1, indices))
            if normalize_routing:
                picked = picked / picked.sum(dim=-1, keepdim=True)
            picked.to(logits.dtype).backward(d_scores)
        return leaf.grad, None, None, None


def fused_topk_router(input: torch.Tensor, router_params: TopkRouterParams):
    """``topk_router`` with everything after the logits GEMM in ONE kernel (softmax, top-k, softmax over the k,
    renormalisation, cast).  Opt-in: its tie rule is its own (equal logits are taken in ascending expert index; the
    k results come in descending score order, where ``torch.topk(sorted=False)`` leaves the order unspecified), so
    on inputs with tied logits among the selected values the indices can differ from ``topk_router``'s; without
    such ties the set of experts per token is the same and the scores agree to one rounding of the 16-bit type.
    (router.py:17-35)"""
    return fused_topk_of_logits(input @ router_params.router_weight, router_params)


def fused_topk_of_logits(logits: torch.Tensor, router_params: TopkRouterParams):
    """Everything of ``fused_topk_router`` after the linear layer."""
    return _FusedTopk.apply(logits, router_params.topk, bool(router_params.softmax_before_topk),
                            bool(router_params.normalize_routing))


def ernie_router(input: torch.Tensor, router_params: ErnieRouterParams):
    """All-fp32 router with a selection-only bias and clamp-normalised weights (router.py:37-54)."""
    assert router_params.router_weight.dtype is torch.float32
    with torch.autocast(device_type=input.device.type, enabled=False):
        logits = input.float() @ router_params.router_weight
        if tail_in_one_kernel(logits, router_params.topk, input.dtype, router_params.bias):
            return _native.router_tail(logits, router_params.topk, True, 2, router_params.bias, input.dtype)
        probs = softmax(logits)
        _, indices = torch.topk(probs + router_params.bias, k=router_params.topk, dim=-1, sorted=False)
        picked = torch.gather(probs, dim=-1, index=indices)
        picked = picked / torch.clamp(picked.sum(dim=-1, keepdim=True), min=1e-12)
        return picked.to(input.dtype), indices
