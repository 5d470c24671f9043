// W4A16 GEMM for few tokens (gemm_few.cu): what the entry points in gemm.cu call.
#pragma once
#include "common.cuh"

namespace nvfp4 {

constexpr int GEMM_FEW_MAX_TOKENS = 128;

// Whether the few-token kernel takes this product (sizes and alignment).
bool gemm_few_takes(const uint8_t* packed, const uint8_t* scales, int N, int K);

// act: token-major [N][ld_act] (in_tm) or token-minor [K][ld_act]; N = tokens the output holds in
// feature-major mode, n_out = tokens written in token-major mode.  0, -3, or a cudaError_t.
int gemm_few_launch(const uint8_t* packed, const uint8_t* scales, const __half* act, long long ld_act,
                    bool in_tm, __half* out, int ld_out, int M, int N, int n_tokens, int K, int out_mode,
                    cudaStream_t st);

// 0 or 1 + the id of the first bounded wait that ran out.  Synchronises the device.
int gemm_few_status(int reset);

}  // namespace nvfp4
