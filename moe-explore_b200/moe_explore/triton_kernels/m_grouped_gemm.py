"""Ragged M-grouped GEMM with optional fused row gather / scatter and activation epilogue.

Drop-in for the reference's Triton wrapper (src/moe_explore/triton_kernels/m_grouped_gemm.py:16-31,
332-393): same ``MGroupedGEMMParams`` fields and the same ``m_grouped_gemm(token, params,
autotune_mode=None)`` call.  The module keeps its reference path although nothing here is Triton:
the contraction runs on the library's tcgen05 kernel over the padded expert-sorted layout.
``autotune_mode`` is accepted and ignored (tile shapes are fixed at build time).
"""
from __future__ import annotations

import functools
from dataclasses import dataclass
from typing import Optional

import torch

from moe_explore import _native
from moe_explore.functional.activation import is_glu
from moe_explore.routing_plan import device_status


@dataclass
class MGroupedGEMMParams:
    weight: torch.Tensor                      # [E, K, N]
    group_indices: torch.Tensor               # int32 [E+1], exclusive prefix of rows per expert
    permute_indices: Optional[torch.Tensor]   # int64 [T*topk], required with gather or scatter
    gather: bool                              # input row of sorted position r is token[permute_indices[r] // topk]
    scatter: bool                             # output row of sorted position r is written at permute_indices[r]
    # With gather or scatter ``num_tokens`` is the token count BEFORE routing (T); otherwise it is
    # simply the number of input rows.
    num_tokens: int
    topk: int
    shared_weight: Optional[torch.Tensor] = None
    scales: Optional[torch.Tensor] = None     # carried for the caller; not applied here
    activation: Optional[str] = None


def m_grouped_gemm(token: torch.Tensor, params: MGroupedGEMMParams, autotune_mode=None) -> torch.Tensor:
    """Rows [g[e], g[e+1]) of the (optionally gathered) input times ``weight[e]``, optional activation epilogue,
    optional scatter of the output rows.  As in the reference kernel the scatter happens inside the GEMM's epilogue
    (m_grouped_gemm.py:168-172): no un-scattered copy of the output exists.  Gathered input rows are copied into
    128-row-aligned expert segments first (one HBM-bound pass) so that the GEMM loads whole tiles; rows that are in expert
    order already are read where they are."""
    assert token.dim() == 2
    assert params.weight.dim() == 3
    assert token.size(1) == params.weight.size(1)
    if params.gather or params.scatter:
        assert params.permute_indices is not None
    _native.require_cuda(token, params.weight, params.group_indices)

    num_experts, k_dim, n_dim = params.weight.shape
    rows = params.num_tokens * params.topk if (params.gather or params.scatter) else params.num_tokens
    act = None if params.activation is None else str(params.activation)
    assert act in _native.ACT_CODES, f"Invalid activation: {act}"
    out_cols = n_dim // 2 if is_glu(act) else n_dim
    out = torch.empty(rows, out_cols, dtype=token.dtype, device=token.device)
    if rows == 0:
        return out

    assert params.group_indices.dim() == 1 and params.group_indices.numel() == num_experts + 1
    groups = params.group_indices.to(torch.int32).contiguous()
    token = token.contiguous()
    weight = params.weight.contiguous()
    perm = None
    if params.gather or params.scatter:
        _native.require_cuda(params.permute_indices)
        perm = params.permute_indices.to(torch.int64).contiguous()
        assert perm.numel() >= rows, "permute_indices is shorter than the routed rows"
    rp, offsets, words = _maps_layout(rows, num_experts)
    maps = torch.empty(words, dtype=torch.int32, device=token.device)
    base = maps.data_ptr()
    padded = torch.empty(rp, k_dim, dtype=token.dtype, device=token.device) if params.gather else None
    ptr = _native._ptr
    steps = [(_native.ROWS_LAYOUT, "routing", 1)]
    if params.gather:
        # (the gather could ride on the GEMM's operand loads -- mgrouped_gemm_gather -- but four-row gather copies are several
        # times slower than 128-row tile copies)
        steps.append((_native.ROWS_GATHER, "rows:gather", 1))
    steps.append((_native.ROWS_GEMM, "mgrouped_gemm:scatter", 1))
    _native.run_pass("moe_rows_gemm", _native.RowsPass(
        rows, token.size(0), num_experts, k_dim, n_dim, params.topk if params.gather else 1, _native.ACT_CODES[act],
        _native.dtype_code(token.dtype), bool(params.gather), bool(params.scatter), token.data_ptr(), weight.data_ptr(),
        out.data_ptr(), groups.data_ptr(), ptr(perm), *[base + o for o in offsets[:-1]],
        device_status(token.get_device()).data_ptr(), ptr(padded), base + offsets[-1]), steps, rows)
    return out


@functools.lru_cache(maxsize=256)
def _maps_layout(rows: int, num_experts: int):
    """(padded rows, byte offsets of pad_offsets, in_rows, out_rows, mtile_expert, tile_pairs, num_mtiles, work counters, int32
    words)."""
    rp = _native.padded_rows_bound(rows, num_experts)
    tiles = rp // _native.TILE_M
    offsets, words = [], 0
    for n in (num_experts + 1, rp, rp, tiles, tiles + num_experts + 1, 4, _native.WORK_COUNTERS):
        offsets.append(4 * words)
        words += (n + 3) // 4 * 4
    return rp, tuple(offsets), words
