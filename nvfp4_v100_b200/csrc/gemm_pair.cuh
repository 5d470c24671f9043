// W4A16 GEMM on CTA pairs for more than 128 tokens (gemm_pair.cu): what the entry points in gemm.cu call.
#pragma once
#include "common.cuh"

namespace nvfp4 {

// Whether the kernel takes this product (sizes and alignment).
bool gemm_pair_takes(const uint8_t* packed, const uint8_t* scales, int N, int K);

// Whether it is the faster one where gemm.cu has 256-row tiles for the shape (both give the same bits).
bool gemm_pair_beats_tiles(int M, int N, int K, int out_mode);

// Whether GEMM_OUT_TM_SILU is possible (more tiles than pairs of SMs) and faster than GEMM_OUT_TM and a pass after it.
bool gemm_pair_fuses_silu(int M, int N, int K);

// act: token-major [n_tokens][ld_act] (in_tm) or token-minor [K][ld_act]; N = tokens the output holds in
// feature-major mode, n_tokens = tokens written in token-major mode.  0, -3, or a cudaError_t.
int gemm_pair_launch(const uint8_t* packed, const uint8_t* scales, const __half* act, long long ld_act,
                     bool in_tm, __half* out, int ld_out, int M, int N, int n_tokens, int K, int out_mode,
                     cudaStream_t st);

// Dynamic shared memory of a launch, the most that any kernel behind the GEMM entry points asks for.
int gemm_pair_shared_bytes();

// 0 or 1 + the id of the first bounded wait that ran out.  Synchronises the device.
int gemm_pair_status(int reset);

}  // namespace nvfp4
