// Attention forward for few query rows and for small problems (attn_rows.cu).
#pragma once
#include "host_common.h"

namespace wk {

// Whether the kernel should take this (valid) call instead of the 128-row tensor-core kernels.
bool attn_rows_applies(const wk_attn_fwd_args* a, bool bf16);
// The FP8 kernel for at most a few dozen packed rows against many keys (attn_decode.cu).
int launch_attn_decode(const wk_attn_fwd_args* a, cudaStream_t stream);
int launch_attn_rows(const wk_attn_fwd_args* a, bool bf16, cudaStream_t stream);

}  // namespace wk
