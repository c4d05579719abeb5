// One layer step from one call: the launches of a step in order, from a description that the
// caller keeps.  A step of a few dozen microseconds is otherwise bound by the host's way from one
// launch to the next: one token on a 16-expert shard, launched call by call, took 69 us through four
// calls from Python and takes 18.5 us through this one, 17 us of it on the GPU.  The stages can be
// called one by one as well (a traced or measured step), with the same launches.
#include "common.cuh"

extern "C" int lm_moe_step_stage(const lm_step* step, int stage, const void* x, const int32_t* topk_ids,
                                 const float* topk_weights, int64_t tokens, void* out, lm_stream_t stream) {
  using namespace lm;
  LM_REQUIRE(step && x && topk_ids && topk_weights && out, "step: null pointer");
  LM_REQUIRE(step->fc1 && step->fc2, "step: null plan");
  LM_REQUIRE(step->kind >= LM_STEP_ONE_TOKEN && step->kind <= LM_STEP_DISPATCH, "step: unknown kind");
  LM_REQUIRE(step->kind != LM_STEP_ONE_TOKEN || tokens == 1, "step: the one-token form takes one token");
  switch (stage) {
    case LM_STAGE_PREPARE:
      if (step->kind == LM_STEP_ONE_TOKEN)
        return lm_decode_prepare(x, topk_ids, topk_weights, step->top_k, step->experts, step->hidden, 1, step->gather,
                                 step->slots, step->table, step->probs, step->padded_offsets, step->scale_pair,
                                 step->qx, step->sfx, stream);
      if (step->kind == LM_STEP_FUSED_PREPARE)
        return lm_dispatch_quantize_decode(x, topk_ids, topk_weights, tokens, step->top_k, step->experts, step->hidden,
                                           step->gather, step->table, step->probs, step->slots, step->padded_offsets,
                                           step->scratch, step->scratch_elems, 128, step->scale_pair, step->qx,
                                           step->sfx, stream);
      return lm_dispatch(topk_ids, topk_weights, tokens, step->top_k, step->experts, step->gather, step->table,
                         step->probs, step->slots, step->padded_offsets, step->scratch, step->scratch_elems, 128,
                         stream);
    case LM_STAGE_QUANTIZE:
      if (step->kind != LM_STEP_DISPATCH) return LM_OK;
      return quantize_scatter(x, tokens, step->hidden, step->top_k, step->slots, topk_ids, step->table, step->experts,
                              step->scale_pair, step->qx, step->sfx, step->gather, step->sf_tokens, stream);
    case LM_STAGE_FC1:
      return lm_gemm_launch(step->fc1, stream);
    case LM_STAGE_FC2:
      return lm_gemm_launch(step->fc2, stream);
    case LM_STAGE_COMBINE:
      return lm_finalize(step->routed_out, step->slots, step->probs, out, tokens, step->top_k, step->hidden,
                         step->hidden, step->hidden, nullptr, step->combine_pdl, stream);
  }
  return set_error(LM_ERR_INVALID, "step: unknown stage");
}

extern "C" int lm_moe_step(const lm_step* step, const void* x, const int32_t* topk_ids, const float* topk_weights,
                           int64_t tokens, void* out, lm_stream_t stream) {
  for (int stage = LM_STAGE_PREPARE; stage <= LM_STAGE_COMBINE; ++stage) {
    const int rc = lm_moe_step_stage(step, stage, x, topk_ids, topk_weights, tokens, out, stream);
    if (rc != LM_OK) return rc;
  }
  return LM_OK;
}
