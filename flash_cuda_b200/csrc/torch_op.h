// torch_op.h — the implementation of the torch op `fwd`, for callers inside this package (torch_direct.cpp).
#pragma once
#include <ATen/core/Tensor.h>

#include <optional>
#include <utility>

namespace fa_b200 {

// The op's arguments in the op's order; returns (out, lse).
std::pair<at::Tensor, at::Tensor> attention(
    at::Tensor q, at::Tensor k, at::Tensor v, std::optional<at::Tensor> k_new, std::optional<at::Tensor> v_new,
    std::optional<at::Tensor> q_v, std::optional<at::Tensor> out_, std::optional<at::Tensor> cu_seqlens_q,
    std::optional<at::Tensor> cu_seqlens_k, std::optional<at::Tensor> cu_seqlens_k_new, std::optional<at::Tensor> seqused_q,
    std::optional<at::Tensor> seqused_k, std::optional<int64_t> max_seqlen_q, std::optional<int64_t> max_seqlen_k,
    std::optional<at::Tensor> page_table, std::optional<at::Tensor> kv_batch_idx, std::optional<at::Tensor> leftpad_k,
    std::optional<at::Tensor> rotary_cos, std::optional<at::Tensor> rotary_sin, std::optional<at::Tensor> seqlens_rotary,
    std::optional<at::Tensor> q_descale, std::optional<at::Tensor> k_descale, std::optional<at::Tensor> v_descale,
    double softmax_scale, bool is_causal, int64_t window_size_left, int64_t window_size_right, double softcap,
    bool is_rotary_interleaved, std::optional<at::Tensor> scheduler_metadata, int64_t num_splits,
    std::optional<bool> pack_gqa, int64_t sm_margin, std::optional<at::Tensor> s_aux, int64_t cp_world_size, int64_t cp_rank,
    std::optional<at::Tensor> cp_tot_seqused_k);

}  // namespace fa_b200
