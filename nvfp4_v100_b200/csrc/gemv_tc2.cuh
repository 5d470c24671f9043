// GEMV of two activations on the tensor cores (gemv_tc2.cu).
#pragma once
#include "common.cuh"

namespace nvfp4 {

// Whether GEMVs may read weights before the kernel in front of them has finished (gemv.cu: bit 1 of
// nvfp4_b200_gemv_config's flags turns it off).
bool gemv_reads_ahead();

// Two activations (16 digit columns each): out[m] = W[m] . act0, out[M + m] = W[m] . act1; interleaved: act0 holds
// K (act0[k], act1[k]) pairs.  Returns 0, -2 where it does not take the problem (the register-streaming kernel then
// does), -3 without a tensor-map encoder, or the launch error.
int gemv_tc2_launch(const uint8_t* packed, const uint8_t* scales, const void* act0, const void* act1, bool interleaved,
                    void* out, int M, int K, cudaStream_t st);
int gemv_tc2_status(int reset);

}  // namespace nvfp4
