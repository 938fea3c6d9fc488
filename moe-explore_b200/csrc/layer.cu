// The expert part of a layer pass in one host call: the launches of moe_expert_forward / moe_expert_backward are the ones a caller
// could make one by one through the entry points below; issuing them from native code is what a pass over a few tokens
// is bound by (from Python, each call costs 5-12 us of argument handling against 2-3 us for the launch itself).
#include "common.cuh"

namespace moe {

// `counts` for a contraction that claims its work items from word `i`.
static RowCounts claiming(const RowCounts& counts, uint32_t* counters, int i) {
  RowCounts c = counts;
  c.work_counter = counters != nullptr ? counters + i : nullptr;
  return c;
}

static bool glu(int act) { return act == MOE_ACT_SWIGLU || act == MOE_ACT_GEGLU; }

}  // namespace moe

using namespace moe;

extern "C" size_t moe_expert_pass_size(void) { return sizeof(moe_expert_pass); }

extern "C" int moe_expert_forward(const moe_expert_pass* p, int steps, void* stream) {
  MOE_CHECK_ARG(p != nullptr, "moe_expert_forward: null pointer argument");
  const int up_cols = glu(p->act) ? 2 * p->inter : p->inter;
  const int64_t rows = p->num_tokens * p->topk;
  const Chain chain;
  if (p->identity) {
    // One expert, weight one: no row moves and nothing is folded.  The GEMMs read x and write out where they are.
    RowCounts in{p->pad_offsets, p->group_indices};
    in.routed_rows = p->num_tokens;
    RowCounts out = in;
    in.a_rows = out.out_rows = p->num_tokens;
    in.settled = (steps & MOE_FWD_ROUTE) == 0;
    out.settled = in.settled || (steps & MOE_FWD_UP) != 0;  // the contraction before waited for the layout
    if (steps & MOE_FWD_ROUTE)
      MOE_STEP(moe_layout_from_groups(p->group_indices, p->num_tokens, 1, p->pad_offsets, nullptr, nullptr, p->mtile_expert,
                                      p->tile_pairs, p->num_mtiles, p->status, stream));
    if (steps & MOE_FWD_UP)
      MOE_STEP(mgrouped_gemm(p->x, p->w1, p->hidden, p->pre_act, p->mtile_expert, p->tile_pairs, p->num_mtiles, p->padded_rows,
                             p->d, up_cols, 1, 0, p->act, p->dtype, 0, 1, nullptr, p->status, stream, in));
    if (steps & MOE_FWD_DOWN)
      MOE_STEP(mgrouped_gemm(p->hidden, p->w2, p->out, nullptr, p->mtile_expert, p->tile_pairs, p->num_mtiles, p->padded_rows,
                             p->inter, p->d, 1, 0, MOE_ACT_NONE, p->dtype, 0, 1, nullptr, p->status, stream, out));
    return MOE_OK;
  }
  RowCounts counts{p->pad_offsets, p->group_indices};
  counts.routed_rows = rows;
  uint32_t* const counters = p->gather ? nullptr : reinterpret_cast<uint32_t*>(p->counters);
  // (the dispatch waits for the routing before it lets the contraction up, and so does a contraction)
  counts.settled = (steps & MOE_FWD_ROUTE) == 0 || ((steps & MOE_FWD_DISPATCH) != 0 && !p->gather);
  if (steps & MOE_FWD_TAIL) {
    void* const scores = const_cast<void*>(p->scores);
    int64_t* const experts = const_cast<int64_t*>(p->expert_idx);
    if (p->own_tie_rule)
      MOE_STEP(moe_router_topk(p->logits, scores, experts, nullptr, p->num_tokens, p->num_experts, p->topk,
                               p->softmax_before_topk, p->normalize, p->dtype, stream));
    else
      MOE_STEP(moe_router_tail(p->logits, p->router_bias, scores, experts, p->num_tokens, p->num_experts, p->topk,
                               p->softmax_before_topk, p->normalize, p->logits_dtype, p->dtype, stream));
  }
  if (steps & MOE_FWD_ROUTE)
    MOE_STEP(routing_metadata(p->expert_idx, rows, p->num_experts, p->group_indices, nullptr, p->pad_offsets, p->row_src,
                              p->dst_row, p->mtile_expert, p->tile_pairs, p->num_mtiles, p->status, p->workspace,
                              p->workspace_bytes, false, stream));
  // the fused fold adds to zeros; set by the dispatch where that is part of the same call (a memset between the two contractions
  // would keep the second from being chained to the first: 3 us)
  const bool cleared = p->fused_combine && !p->keep && !p->gather && (steps & MOE_FWD_DISPATCH) != 0;
  if ((steps & MOE_FWD_DISPATCH) && !p->gather) {
    // rows do not mix in a forward pass, and only a weight gradient contracts over the padding rows
    if (p->keep)
      MOE_STEP(dispatch_rows(p->x, p->dst_row, p->row_src, p->num_mtiles, p->xs, p->num_tokens, p->topk, p->padded_rows, p->d,
                                 p->dtype, stream, true, counters));
    else
      MOE_STEP(dispatch_rows_only(p->x, p->dst_row, p->xs, p->num_tokens, p->topk, p->d, p->dtype, stream, counters,
                                  cleared ? p->out : nullptr));
  }
  if (steps & MOE_FWD_UP) {
    if (p->gather)
      MOE_STEP(mgrouped_gemm_gather(p->x, p->num_tokens, p->row_src, p->topk, p->w1, p->hidden, p->pre_act, p->mtile_expert,
                                        p->tile_pairs, p->num_mtiles, p->padded_rows, p->d, up_cols, p->num_experts, p->act,
                                        p->dtype, nullptr, p->status, stream, counts));
    else
      MOE_STEP(mgrouped_gemm(p->xs, p->w1, p->hidden, p->pre_act, p->mtile_expert, p->tile_pairs, p->num_mtiles,
                                 p->padded_rows, p->d, up_cols, p->num_experts, 0, p->act, p->dtype, 0, 1, nullptr, p->status,
                                 stream, claiming(counts, counters, 0)));
  }
  if (steps & MOE_FWD_DOWN) {
    if (p->fused_combine) {
      if (!cleared) {
        MOE_CUDA(cudaMemsetAsync(p->out, 0, static_cast<size_t>(p->num_tokens) * p->d * 2, static_cast<cudaStream_t>(stream)));
        chained_launches() = false;  // the memset stands between
      }
      MOE_STEP(mgrouped_gemm_combine(p->hidden, p->w2, p->out, p->row_src, p->scores, p->topk, p->mtile_expert, p->tile_pairs,
                                         p->num_mtiles, p->padded_rows, p->inter, p->d, p->num_experts, 0, p->dtype, nullptr,
                                         p->status, stream, claiming(counts, counters, 1)));
    } else {
      MOE_STEP(mgrouped_gemm(p->hidden, p->w2, p->ys, nullptr, p->mtile_expert, p->tile_pairs, p->num_mtiles, p->padded_rows,
                                 p->inter, p->d, p->num_experts, 0, MOE_ACT_NONE, p->dtype, 0, 1, nullptr, p->status, stream, claiming(counts, counters, 1)));
    }
  }
  if ((steps & MOE_FWD_FOLD) && !p->fused_combine)
    MOE_STEP(combine_topk(p->ys, p->scores, p->dst_row, p->out, p->num_tokens, p->topk, p->d, p->dtype, p->addend, nullptr,
                          nullptr, nullptr, stream));
  return MOE_OK;
}

extern "C" int moe_expert_backward(const moe_expert_pass* p, int steps, void* stream) {
  MOE_CHECK_ARG(p != nullptr, "moe_expert_backward: null pointer argument");
  const int up_cols = glu(p->act) ? 2 * p->inter : p->inter;
  const Chain chain;
  if (p->identity) {
    RowCounts in{p->pad_offsets, p->group_indices};
    in.routed_rows = p->num_tokens;
    RowCounts out = in, right = in;
    in.a_rows = out.out_rows = right.b_rows = p->num_tokens;
    in.settled = out.settled = true;
    if (steps & MOE_BWD_DOWN) {
      if (p->act == MOE_ACT_NONE)
        MOE_STEP(mgrouped_gemm(p->grad_out, p->w2, p->d_pre, nullptr, p->mtile_expert, p->tile_pairs, p->num_mtiles,
                               p->padded_rows, p->d, p->inter, 1, 1, MOE_ACT_NONE, p->dtype, 0, 1, nullptr, p->status, stream, in));
      else
        MOE_STEP(mgrouped_gemm_dglu(p->grad_out, p->w2, p->pre_act, p->d_pre, p->mtile_expert, p->tile_pairs, p->num_mtiles,
                                    p->padded_rows, p->d, p->inter, 1, p->act, p->dtype, 0, 1, nullptr, p->status, stream, in));
    }
    if (steps & MOE_BWD_UP)
      MOE_STEP(mgrouped_gemm(p->d_pre, p->w1, p->dx, nullptr, p->mtile_expert, p->tile_pairs, p->num_mtiles, p->padded_rows,
                             up_cols, p->d, 1, 1, MOE_ACT_NONE, p->dtype, 0, 1, nullptr, p->status, stream, out));
    if (steps & MOE_BWD_DW1)
      MOE_STEP(kgrouped_gemm(p->x, p->d_pre, p->d_w1, p->pad_offsets, p->padded_rows, p->d, up_cols, 1, p->dtype, nullptr,
                             p->status, stream, in));
    if (steps & MOE_BWD_DW2)
      MOE_STEP(kgrouped_gemm(p->hidden, p->grad_out, p->d_w2, p->pad_offsets, p->padded_rows, p->inter, p->d, 1, p->dtype,
                             nullptr, p->status, stream, right));
    return MOE_OK;
  }
  RowCounts counts{p->pad_offsets, p->group_indices};
  counts.routed_rows = p->num_tokens * p->topk;
  counts.settled = true;  // nothing of a backward pass writes the metadata or the weights
  uint32_t* const counters = reinterpret_cast<uint32_t*>(p->counters);
  if (steps & MOE_BWD_FOLD)
    MOE_STEP(combine_bwd_tokens(p->grad_out, p->scores, p->ys, p->dst_row, p->row_src, p->num_mtiles, p->gs, p->d_scores,
                                    p->num_tokens, p->topk, p->d, p->dtype, stream, true, counters));
  if ((steps & MOE_BWD_ROUTER) && p->dl != nullptr)
    MOE_STEP(router_backward(p->logits, p->expert_idx, p->d_scores, p->router_w, p->dl, p->dlogits, p->router_t, p->num_tokens,
                             p->num_experts, p->topk, p->d, p->dtype, stream));
  if (steps & MOE_BWD_DOWN) {
    if (p->act == MOE_ACT_NONE)  // linear "activation": d_pre = gs @ W2^T
      MOE_STEP(mgrouped_gemm(p->gs, p->w2, p->d_pre, nullptr, p->mtile_expert, p->tile_pairs, p->num_mtiles, p->padded_rows,
                                 p->d, p->inter, p->num_experts, 1, MOE_ACT_NONE, p->dtype, 0, 1, nullptr, p->status, stream, claiming(counts, counters, 0)));
    else
      MOE_STEP(mgrouped_gemm_dglu(p->gs, p->w2, p->pre_act, p->d_pre, p->mtile_expert, p->tile_pairs, p->num_mtiles,
                                      p->padded_rows, p->d, p->inter, p->num_experts, p->act, p->dtype, 0, 1, nullptr, p->status,
                                      stream, claiming(counts, counters, 0)));
  }
  if (steps & MOE_BWD_UP)
    MOE_STEP(mgrouped_gemm(p->d_pre, p->w1, p->dxs, nullptr, p->mtile_expert, p->tile_pairs, p->num_mtiles, p->padded_rows,
                               up_cols, p->d, p->num_experts, 1, MOE_ACT_NONE, p->dtype, 0, 1, nullptr, p->status, stream, claiming(counts, counters, 1)));
  if (steps & MOE_BWD_FOLD_DX)
    MOE_STEP(combine_topk(p->dxs, nullptr, p->dst_row, p->dx, p->num_tokens, p->topk, p->d, p->dtype, nullptr, p->dl,
                          p->expert_idx, p->router_t, stream));
  if (steps & MOE_BWD_DW1) {
    if (p->gather)  // x is the layer input in token order: its rows are gathered by the loads again
      MOE_STEP(kgrouped_gemm_gather(p->x, p->num_tokens, p->row_src, p->topk, p->d_pre, p->d_w1, p->pad_offsets,
                                        p->padded_rows, p->d, up_cols, p->num_experts, p->dtype, nullptr, p->status, stream, claiming(counts, counters, 2)));
    else
      MOE_STEP(kgrouped_gemm(p->xs, p->d_pre, p->d_w1, p->pad_offsets, p->padded_rows, p->d, up_cols, p->num_experts, p->dtype,
                                 nullptr, p->status, stream, claiming(counts, counters, 2)));
  }
  if (steps & MOE_BWD_DW2)
    MOE_STEP(kgrouped_gemm(p->hidden, p->gs, p->d_w2, p->pad_offsets, p->padded_rows, p->inter, p->d, p->num_experts, p->dtype,
                               nullptr, p->status, stream, claiming(counts, counters, 3)));
  return MOE_OK;
}
