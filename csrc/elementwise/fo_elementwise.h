// Host launchers of the decoder layer's element-wise kernels (rotary embedding, SwiGLU).  The
// reference ships no model beyond a linear layer and a norm, so these have no counterpart there.
#pragma once
#include <cuda_runtime.h>

namespace fo {

// Rotary embedding in place over the first `heads` heads of every row of QKV [tokens, row_elems]
// (16-bit storage, fp32 math, adjacent pairs rotate): position = row % seq.  head_dim % 8 == 0.
cudaError_t rope_launch(void* QKV, int tokens, int seq, int heads, int head_dim, int row_elems, float theta, bool bf16,
                        cudaStream_t stream);

// Y[rows, f] = round16(round16(silu(GU[:, :f])) * GU[:, f:]), GU [rows, 2 f] row-major.  f % 8 == 0.
cudaError_t swiglu_launch(const void* GU, void* Y, int rows, int f, bool bf16, int sm_count, cudaStream_t stream);

}  // namespace fo
