// Attention forward for few query rows and for small problems (attn_rows.cu).
#pragma once
#include "host_common.h"

namespace wk {

// Whether this (valid) call is one of few query rows or small enough for the kernels of attn_rows.cu and attn_decode.cu.
bool attn_rows_applies(const wk_attn_fwd_args* a);
// Whether they are then ahead of the kernels with tiles of 128 rows.
bool attn_rows_ahead(const wk_attn_fwd_args* a, bool bf16, int sms);
// The FP8 kernel for at most a few dozen packed rows against many keys (attn_decode.cu).
int launch_attn_decode(const wk_attn_fwd_args* a, cudaStream_t stream);
// Into how many CTAs it divides the keys, with `units` of (KV heads of the batch x groups of packed rows).
int attn_decode_splits(const wk_attn_fwd_args* a, int64_t units, int sms);
int launch_attn_rows(const wk_attn_fwd_args* a, bool bf16, cudaStream_t stream);

}  // namespace wk
