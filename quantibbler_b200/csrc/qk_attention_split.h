// Float32 attention as sums of 16-bit products on tcgen05 (qk_attention_split.cu).
#pragma once

#include "qk_common.h"

namespace qk {
// Whether the exact attention face can take this call here (sizes, masks, no graph being recorded).
bool attention_split_takes(qk_ctx *c, const qk_attention_shape *s, int causal);
qk_status attention_split_exact(qk_ctx *c, const float *q, const float *k, const float *v, float *out,
                                const qk_attention_shape *s, int causal);
// Causal attention of n_tokens new positions of sequence slot `seq` against its bfloat16 cache, heads of 128.
qk_status attention_split_cached(qk_ctx *c, const float *q, const void *cache_k, const void *cache_v, size_t seq,
                                 size_t first_position, size_t n_tokens, size_t n_heads, size_t n_kv_heads, size_t s_max,
                                 float *out);
}  // namespace qk
