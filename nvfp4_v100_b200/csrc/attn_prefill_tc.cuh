// Tensor-core attention of a prefill chunk (attn_prefill_tc.cu): what launch_attn_prefill calls.
#pragma once
#include "common.cuh"

namespace nvfp4 {

// (token, key) pairs of a chunk from which the tensor-core kernel is the faster one: 64 tokens of an
// empty cache 25.7 -> 18.2 us, 8 tokens after 511 30.9 -> 12.3; below it the one-query-at-a-time kernel
// takes 8 to 20 us (16 after 64: 11.2, 26 after 64: 20.4) except for a handful of tokens deep in a context.
// (24 heads; with few heads the line lies higher, see attn_prefill_tc_takes.)
constexpr long long ATTN_TC_MIN_PAIRS = 4096;

// Whether the tensor-core kernel takes this call (sizes and alignment).
bool attn_prefill_tc_takes(const void* q, const void* keys, const void* values, const void* gate, const void* out,
                           int len0, int n_tokens, int hq, int hkv);

// The arguments of launch_attn_prefill, already checked.  0, -3, or a cudaError_t.
int attn_prefill_tc_launch(const __half* q, const __half* keys, const __half* values, int len0, int n_tokens,
                           const __half* gate, __half* out, int max_len, int hq, int hkv, float scale,
                           cudaStream_t st);

// 0 or 1 + the id of the first bounded wait that ran out.  Synchronises the device.
int attn_prefill_tc_status(int reset);

}  // namespace nvfp4
