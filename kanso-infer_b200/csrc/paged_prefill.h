// Prompt attention over the quantised pool in tiles of query rows (paged_prefill.cu).
#pragma once
#include "ctx.h"

namespace kanso {
// Arguments as kanso_cuda_paged_attention_prefill's, checked. *handled = false, nothing launched: the
// call is outside this kernel's range or has too few query tokens per sequence to fill its tiles.
int32_t launch_paged_prefill(kanso_cuda_ctx* ctx, const kanso_cuda_kv* kv, uint32_t layer,
                             const float* q, const uint32_t* tables, const uint32_t* ctx_lens,
                             const uint32_t* q_lens, float* out,
                             const kanso_paged_attention_params* p, bool* handled);
}  // namespace kanso
