// Float32 attention as sums of 16-bit products on tcgen05 (qk_attention_split.cu).
#pragma once

#include "qk_common.h"

namespace qk {
// Whether the exact attention face can take this call here (sizes, masks, no graph being recorded).
bool attention_split_takes(qk_ctx *c, const qk_attention_shape *s, int causal);
// QK_ERR_ALLOC: no memory for the terms (as much as k and v take, more for heads below 64 channels); nothing is launched.
// *marked: rows that the caller has to compute again, one bit each, [batch x heads][tiles of 128 rows][4 words] on
// the device, valid in stream order until the context's next call.
qk_status attention_split_exact(qk_ctx *c, const float *q, const float *k, const float *v, float *out,
                                const qk_attention_shape *s, int causal, const uint32_t **marked);
}  // namespace qk
