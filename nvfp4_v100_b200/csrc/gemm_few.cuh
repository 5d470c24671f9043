// W4A16 GEMM for few tokens (gemm_few.cu): what the entry points in gemm.cu call.
#pragma once
#include "common.cuh"

namespace nvfp4 {

// One token tile.  Above it the CTA-pair kernel, which needs enough rows to fill the GPU: 136 tokens 16480 x
// 5120 25.4 us against 35.8 with two token tiles here, 34816 x 5120 51.3 / 71.4.  Narrow matrices lie the other
// way up to 256 tokens: gemm_few_takes_two.
constexpr int GEMM_FEW_MAX_TOKENS = 128;

// Whether the few-token kernel takes this product (sizes and alignment).
bool gemm_few_takes(const uint8_t* packed, const uint8_t* scales, int N, int K);

// Whether the kernel is the faster one for this product of 129 to 256 tokens (its sums over K are in another order than
// those of the kernels it then replaces).
bool gemm_few_takes_two(const uint8_t* packed, const uint8_t* scales, int M, int N, int K);

// act: token-major [N][ld_act] (in_tm) or token-minor [K][ld_act]; N = tokens the output holds in
// feature-major mode, n_out = tokens written in token-major mode.  0, -3, or a cudaError_t.
int gemm_few_launch(const uint8_t* packed, const uint8_t* scales, const __half* act, long long ld_act,
                    bool in_tm, __half* out, int ld_out, int M, int N, int n_tokens, int K, int out_mode,
                    cudaStream_t st);

// 0 or 1 + the id of the first bounded wait that ran out.  Synchronises the device.
int gemm_few_status(int reset);

// Clusters of `split` CTAs (1 to 8) that run at once with two CTAs per SM.
int gemm_few_clusters(int dev, int split);

}  // namespace nvfp4
