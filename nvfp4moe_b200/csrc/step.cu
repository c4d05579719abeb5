// One layer step from one call: the launches of a step in order, from a description that the
// caller keeps.  A step of a few dozen microseconds is otherwise bound by the host's way from one
// launch to the next: one token on a 16-expert shard, launched call by call, took 69 us through four
// calls from Python and takes 18.5 us through this one, 17 us of it on the GPU.
#include "common.cuh"

extern "C" int lm_moe_step(const lm_step* step, const void* x, const int32_t* topk_ids, const float* topk_weights,
                           int64_t tokens, void* out, lm_stream_t stream) {
  using namespace lm;
  LM_REQUIRE(step && x && topk_ids && topk_weights && out, "step: null pointer");
  LM_REQUIRE(step->fc1 && step->fc2, "step: null plan");
  int rc;
  switch (step->kind) {
    case LM_STEP_ONE_TOKEN:
      LM_REQUIRE(tokens == 1, "step: the one-token form takes one token");
      rc = lm_decode_prepare(x, topk_ids, topk_weights, step->top_k, step->experts, step->hidden, 1, step->gather,
                             step->slots, step->table, step->probs, step->padded_offsets, step->scale_pair, step->qx,
                             step->sfx, stream);
      break;
    case LM_STEP_FUSED_PREPARE:
      rc = lm_dispatch_quantize_decode(x, topk_ids, topk_weights, tokens, step->top_k, step->experts, step->hidden,
                                       step->gather, step->table, step->probs, step->slots, step->padded_offsets,
                                       step->scratch, step->scratch_elems, 128, step->scale_pair, step->qx, step->sfx,
                                       stream);
      break;
    case LM_STEP_DISPATCH:
      rc = lm_dispatch(topk_ids, topk_weights, tokens, step->top_k, step->experts, step->gather, step->table,
                       step->probs, step->slots, step->padded_offsets, step->scratch, step->scratch_elems, 128, stream);
      if (rc == LM_OK)
        rc = quantize_scatter(x, tokens, step->hidden, step->top_k, step->slots, topk_ids, step->table, step->experts,
                              step->scale_pair, step->qx, step->sfx, step->gather, step->sf_tokens, stream);
      break;
    default:
      return set_error(LM_ERR_INVALID, "step: unknown kind");
  }
  if (rc == LM_OK) rc = lm_gemm_launch(step->fc1, stream);
  if (rc == LM_OK) rc = lm_gemm_launch(step->fc2, stream);
  if (rc == LM_OK)
    rc = lm_finalize(step->routed_out, step->slots, step->probs, out, tokens, step->top_k, step->hidden, step->hidden,
                     step->hidden, nullptr, step->combine_pdl, stream);
  return rc;
}
