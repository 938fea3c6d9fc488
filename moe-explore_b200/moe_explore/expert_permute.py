"""Routing metadata and the stand-alone permute helpers.

Same names and return types as the reference (src/moe_explore/expert_permute.py:8-68).  The
sort is the library's stable counting sort, so ``indices`` equals
``torch.sort(flat_expert_indices, stable=True).indices`` bit for bit (the reference calls a
non-stable ``argsort``, whose order inside an expert is unspecified).
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Tuple, Union

import torch

from moe_explore import _native
from moe_explore.functional.scale_and_reduce import scale_and_reduce
from moe_explore.routing_plan import build_routing_plan, device_status


@dataclass
class GroupedTokens:
    tokens: torch.Tensor
    group_indices: torch.Tensor
    indices: torch.Tensor


@dataclass
class PermToGroupIndices:
    group_indices: torch.Tensor
    indices: torch.Tensor


def get_token_indices(expert_indices: torch.Tensor, topk: int, num_experts: int, zero_prefix: bool = False) -> PermToGroupIndices:
    """``expert_indices`` int64 [T, topk] -> per-expert row ranges and the permutation that sorts
    the flat (token, slot) positions by expert (expert_permute.py:19-41).

    ``zero_prefix=True``: ``group_indices`` is int32 [E+1] starting at 0; otherwise the inclusive
    cumulative counts, int64 [E] (what ``counts.cumsum`` yields in the reference)."""
    plan = build_routing_plan(expert_indices, num_experts, topk, want_perm=True)
    if zero_prefix:
        groups = plan.group_indices
    else:
        groups = plan.group_indices[1:].to(torch.int64)
    return PermToGroupIndices(group_indices=groups, indices=plan.perm)


def row_gather(tokens: torch.Tensor, indices: torch.Tensor) -> torch.Tensor:
    """``out[r] = tokens[indices[r]]`` (triton_kernels/row_gather_scatter.py:36-58)."""
    _native.require_cuda(tokens, indices)
    assert tokens.dim() == 2 and indices.dim() == 1
    out = torch.empty(indices.numel(), tokens.size(1), dtype=tokens.dtype, device=tokens.device)
    _native.unpad_rows(tokens.contiguous(), indices.to(torch.int32), out)
    return out


def row_scatter(tokens: torch.Tensor, indices: torch.Tensor) -> torch.Tensor:
    """``out[indices[r]] = tokens[r]``; ``indices`` must be a permutation (triton_kernels/row_gather_scatter.py:91-116), but for
    entries of -1 (positions ``get_token_indices`` dropped): their rows go nowhere and the rows of ``out`` that nothing
    reaches are zero.  An entry past the end is reported through the device's status word."""
    inverse = _inverse(tokens, indices)
    out = torch.empty_like(tokens)
    _native.unpad_rows(tokens.contiguous(), inverse, out)
    return out


def _inverse(tokens: torch.Tensor, indices: torch.Tensor) -> torch.Tensor:
    _native.require_cuda(tokens, indices)
    assert tokens.dim() == 2 and indices.dim() == 1 and indices.numel() == tokens.size(0)
    inverse = torch.empty(indices.numel(), dtype=torch.int32, device=tokens.device)
    _native.inverse_rows(indices.to(torch.int64).contiguous(), inverse, device_status(tokens.get_device()))
    return inverse


def expert_input_permute(tokens: torch.Tensor, expert_indices: torch.Tensor, num_experts: int, topk: int) -> GroupedTokens:
    """Gather token rows into expert order (expert_permute.py:43-56)."""
    found = get_token_indices(expert_indices, topk, num_experts, zero_prefix=True)
    assert tokens.dim() == 2
    grouped = torch.empty(found.indices.numel(), tokens.size(1), dtype=tokens.dtype, device=tokens.device)
    _native.index_rows(tokens.contiguous(), found.indices, grouped, div=topk)
    return GroupedTokens(tokens=grouped, group_indices=found.group_indices, indices=found.indices)


def expert_output_permute(grouped_tokens: GroupedTokens, expert_scores: torch.Tensor, topk: int,
                          output_shape: Union[Tuple[int], torch.Size]) -> torch.Tensor:
    """Scatter expert-ordered rows back to (token, slot) order and fold the slots with the router
    weights (expert_permute.py:58-68)."""
    tokens = grouped_tokens.tokens
    if torch.is_grad_enabled() and expert_scores.requires_grad:
        # the gradient of the scores needs the rows in (token, slot) order
        tokens = row_scatter(tokens, grouped_tokens.indices)
        return scale_and_reduce(tokens, expert_scores, expert_scores.size(0), topk, tokens.size(1))
    # Without it the fold reads the expert-ordered rows where they are: the un-permuted copy (every row written and read
    # once more) was 73 of 232 us at 65536 rows of 4 KB and saved nothing.
    assert tokens.dim() == 2
    return _FoldGrouped.apply(tokens.detach(), expert_scores, grouped_tokens.indices, topk)


class _FoldGrouped(torch.autograd.Function):
    """out[t] = sum_s scores[t, s] * tokens[position of (t, s) in ``indices``]; only reached without gradients."""

    @staticmethod
    def forward(ctx, tokens, scores, indices, topk):
        inverse = _inverse(tokens, indices)
        T = scores.size(0)
        assert tokens.size(0) == T * topk and scores.shape == (T, topk)
        _native.require_cuda(scores)
        out = torch.empty(T, tokens.size(1), dtype=tokens.dtype, device=tokens.device)
        _native.combine_topk(tokens.contiguous(), scores.to(tokens.dtype).contiguous(), inverse, out, topk)
        return out
