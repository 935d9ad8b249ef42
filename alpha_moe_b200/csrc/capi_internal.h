// Shared by the C ABI library and the torch operator library: the per-thread error message behind
// alpha_moe_b200_last_error(), and the layer call for a caller that keeps its scratch to itself.
#pragma once

#include <cstdint>

namespace amoe_capi {
// Stores a printf-style message for the calling thread and returns `code`.
int fail(int code, const char* fmt, ...);

// alpha_moe_b200_fused_experts.  keep_schedule: whether sorted_token_ids, expert_ids and num_tokens_post_padded hold the schedule
// afterwards in every case; without it an operator that makes the schedule itself does not write it out.
int fused_experts(void* hidden_states, void* x_fp8, float* x_scale, const void* w, const float* w_scale, const void* w2,
                  const float* w2_scale, const int32_t* topk_ids, const float* topk_weights, int top_k, int M, int K, int N,
                  int num_experts, int32_t* sorted_token_ids, int32_t* expert_ids, int32_t* num_tokens_post_padded,
                  void* align_workspace, int block_m, int block_n, int warp_n, int stages, float scaling_factor, void* stream,
                  bool keep_schedule);
}  // namespace amoe_capi
