// Gated DeltaNet over a chunk in blocks of 64 tokens on the tensor cores (dn_chunk.cu); used by launch_dn_prefill.
#pragma once
#include "common.cuh"

namespace nvfp4 {

// Whether n tokens of nv value heads are faster this way than four tokens at a time (prefill.cu).
bool dn_chunk_takes(int n, int nv);

// Bytes of workspace for n tokens (a multiple of 256).
long long dn_chunk_work_bytes(int n, int nk, int nv);

// The recurrence over n tokens: conv_out [n][conv_dim] (conv + silu, fp16), x / ld / A_log / dt_bias as for
// launch_dn_prefill, work 256-byte aligned; state is updated, o_out [n][nv * 128] gets the outputs (fp16).
cudaError_t dn_chunk_launch(const __half* conv_out, int conv_dim, const __half* x, long long ld, const __half* A_log,
                            const __half* dt_bias, float* state, void* work, __half* o_out, int n, int nk, int nv,
                            cudaStream_t st);

}  // namespace nvfp4
