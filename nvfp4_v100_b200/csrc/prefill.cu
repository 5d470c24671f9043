// Chunked prefill around the tensor-core GEMM: everything a prompt chunk needs between the GEMMs,
// with the arithmetic (formulas and fp16 rounding points) of the decode-step kernels, so that a
// prompt fed through here leaves the KV cache, the conv window and the recurrent state as feeding
// it token by token through the decode step would, up to the GEMM-vs-GEMV summation order.
//
// The reference prefills through the third-party model code (pipeline/_qwen38_infer.py:796-809:
// 512-token chunks, every Linear running launch_nvfp4_gemmtc_v5, attention and the gated delta
// rule in PyTorch).  Here the chunk's activations are token-major [tokens][features] between the
// operators and at the GEMMs (launch_nvfp4_gemm_w4a16_ex, launch_nvfp4_gemm_silu):
//   transpose_f16 / add_transposed   layout changes around launch_nvfp4_gemmtc_v5 (the second fused with
//                                    the residual add), for a caller that keeps to that entry point
//   embed_rows                       token ids -> embedding rows
//   silu_mul_tokens, silu_mul_rows   gate/up (interleaved by 8) -> activations, token-major and token-minor
//   dn_conv_tokens, dn_block, dn_scan, dn_post   one Gated-DeltaNet layer over a chunk:
//       causal conv + silu over the chunk with the carried window; q/k L2 norm, beta, decay;
//       the recurrence S_t = S_{t-1} e^{g_t} + k_t (v_t - S_{t-1} e^{g_t} k_t) beta_t, o_t = S_t q_t
//       run over the chunk in blocks of four tokens with every state row in registers (rows are
//       independent: 16 lanes own two rows, 8 dims each; 6144 rows of the full model), longer chunks in
//       blocks of 64 on the tensor cores (dn_chunk.cu); gated norm.
// Attention uses the chunk forms of attn_prep (decode_ops.cu) and launch_attn_prefill: the tensor-core
// kernel (attn_prefill_tc.cu) or, for small chunks, attn_prefill_group_kernel (fused_ops.cu).
#include <algorithm>
#include <cstdio>

#include "common.cuh"
#include "dn_chunk.cuh"

namespace nvfp4 {


// dst[c][r] = src[r][c] for r < R, c < C; dst rows are ld_dst long and columns R .. ld_dst-1 are
// zero-filled (the GEMM reads whole rows).  src rows are ld_src long.
__global__ void __launch_bounds__(256)
transpose_f16_kernel(const __half* __restrict__ src, long long ld_src, __half* __restrict__ dst,
                     long long ld_dst, int R, int C) {
    pdl_prologue();
    PDL_FRESH(src); PDL_FRESH(dst);
    __shared__ __half tile[64][66];
    const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
    // read 64 rows x 64 columns: a thread reads two adjacent columns (one 4-byte load)
    for (int i = ty; i < 64; i += 8) {
        const int r = r0 + i, c = c0 + tx * 2;
        __half2 v = __floats2half2_rn(0.0f, 0.0f);
        if (r < R) {
            if (c + 1 < C && ((ld_src | c) & 1) == 0) {
                v = *reinterpret_cast<const __half2*>(src + (size_t)r * ld_src + c);
            } else {
                const __half lo = (c < C) ? src[(size_t)r * ld_src + c] : __float2half(0.0f);
                const __half hi = (c + 1 < C) ? src[(size_t)r * ld_src + c + 1] : __float2half(0.0f);
                v = __halves2half2(lo, hi);
            }
        }
        tile[i][tx * 2] = __low2half(v);
        tile[i][tx * 2 + 1] = __high2half(v);
    }
    __syncthreads();
    for (int i = ty; i < 64; i += 8) {
        const int c = c0 + i, r = r0 + tx * 2;
        if (c >= C) continue;
        __half* d = dst + (size_t)c * ld_dst + r;
        if (r + 1 < ld_dst && ((ld_dst | r) & 1) == 0) {
            *reinterpret_cast<__half2*>(d) = __halves2half2(tile[tx * 2][i], tile[tx * 2 + 1][i]);
        } else {
            if (r < ld_dst) d[0] = tile[tx * 2][i];
            if (r + 1 < ld_dst) d[1] = tile[tx * 2 + 1][i];
        }
    }
}

// h[t][c] = f16(f32(h[t][c]) + f32(dT[c][t])) for t < n, c < C: the residual add, reading the
// GEMM's token-minor output (rows ldT long).
__global__ void __launch_bounds__(256)
add_transposed_kernel(__half* __restrict__ h, const __half* __restrict__ dT, long long ldT, int n,
                      int C) {
    pdl_prologue();
    PDL_FRESH(h); PDL_FRESH(dT);
    __shared__ __half tile[64][66];
    const int t0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int i = ty; i < 64; i += 8) {          // rows of dT: feature c0 + i, tokens t0 ..
        const int c = c0 + i;
        const int t = t0 + tx * 2;
        __half lo = __float2half(0.0f), hi = lo;
        if (c < C) {
            if (t < n) lo = dT[(size_t)c * ldT + t];
            if (t + 1 < n) hi = dT[(size_t)c * ldT + t + 1];
        }
        tile[i][tx * 2] = lo;
        tile[i][tx * 2 + 1] = hi;
    }
    __syncthreads();
    for (int i = ty; i < 64; i += 8) {          // rows of h: token t0 + i, features c0 ..
        const int t = t0 + i;
        if (t >= n) continue;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int c = c0 + tx * 2 + u;
            if (c < C) {
                __half* p = h + (size_t)t * C + c;
                *p = __float2half(__half2float(*p) + __half2float(tile[tx * 2 + u][i]));
            }
        }
    }
}

// out[t][:] = table[ids[t]][:]
__global__ void __launch_bounds__(256)
embed_rows_kernel(const __half* __restrict__ table, const long long* __restrict__ ids,
                  __half* __restrict__ out, int hidden, long long vocab) {
    pdl_prologue();
    PDL_FRESH(table); PDL_FRESH(ids); PDL_FRESH(out);
    long long id = ids[blockIdx.y];
    if (id < 0) id = 0;
    if (id >= vocab) id = vocab - 1;
    const int i = (blockIdx.x * 256 + threadIdx.x) * 8;
    const __half* src = table + (size_t)id * hidden;
    __half* dst = out + (size_t)blockIdx.y * hidden;
    if (i + 8 <= hidden && (hidden & 7) == 0) {
        *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(src + i);
    } else {
        for (int j = i; j < hidden && j < i + 8; j++) dst[j] = src[j];
    }
}

// Token-minor gate/up rows, interleaved in groups of 8 (rows 16j..16j+7 gate, 16j+8..16j+15 up),
// to activation rows: act[8j + r][t] = f16( f32(f16(silu(g))) * u ), the silu_mul_kernel chain.
// W tokens a thread: eight with 16-byte accesses (N a multiple of 8, 16-byte aligned matrices), two with
// 4-byte ones (N even), or two with single ones (ODD).  flat: rows and token groups share the grid's x, so
// many short rows leave no CTA nearly empty (17408 rows of 27 tokens 18.3 -> 3.1 us against a CTA per row);
// otherwise a row is blockIdx.y, which saves the division where the rows' CTAs run at once anyway.
template <int W, bool ODD>
__global__ void __launch_bounds__(256)
silu_mul_rows_kernel(const __half* __restrict__ gu, __half* __restrict__ act, int inter, int N, bool flat) {
    pdl_prologue();
    PDL_FRESH(gu); PDL_FRESH(act);
    const unsigned groups = ((unsigned)N + W - 1) / W, id = blockIdx.x * 256 + threadIdx.x;
    const unsigned row = flat ? id / groups : blockIdx.y, group = flat ? id % groups : id;
    if (row >= (unsigned)inter || group >= groups) return;
    const size_t t = (size_t)group * W, grow = (size_t)(row >> 3) * 16 + (row & 7);
    const __half* g = gu + grow * N + t;
    const __half* u = gu + (grow + 8) * N + t;
    __half* o = act + (size_t)row * N + t;
    if constexpr (W == 8) {
        const uint4 gv = *reinterpret_cast<const uint4*>(g), uv = *reinterpret_cast<const uint4*>(u);
        const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
        uint32_t ow[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 gf = __half22float2(*reinterpret_cast<const __half2*>(&gw[k]));
            const float2 uf = __half22float2(*reinterpret_cast<const __half2*>(&uw[k]));
            const __half2 r = __floats2half2_rn(round_f16(silu_pf(gf.x)) * uf.x, round_f16(silu_pf(gf.y)) * uf.y);
            ow[k] = *reinterpret_cast<const uint32_t*>(&r);
        }
        *reinterpret_cast<uint4*>(o) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    } else if constexpr (!ODD) {
        const float2 gf = __half22float2(*reinterpret_cast<const __half2*>(g));
        const float2 uf = __half22float2(*reinterpret_cast<const __half2*>(u));
        *reinterpret_cast<__half2*>(o) =
            __floats2half2_rn(round_f16(silu_pf(gf.x)) * uf.x, round_f16(silu_pf(gf.y)) * uf.y);
    } else {
        const bool two = t + 1 < (size_t)N;
        const float g0 = __half2float(g[0]), u0 = __half2float(u[0]);
        const float g1 = two ? __half2float(g[1]) : 0.0f, u1 = two ? __half2float(u[1]) : 0.0f;
        o[0] = __float2half(round_f16(silu_pf(g0)) * u0);
        if (two) o[1] = __float2half(round_f16(silu_pf(g1)) * u1);
    }
}

// The same for token-major rows: sixteen neighbours (eight gates, their eight ups) make eight results.
__global__ void __launch_bounds__(256)
silu_mul_tokens_kernel(const __half* __restrict__ gu, __half* __restrict__ act, long long pieces) {
    pdl_prologue();
    PDL_FRESH(gu); PDL_FRESH(act);
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= pieces) return;
    const uint4 gv = reinterpret_cast<const uint4*>(gu)[2 * i], uv = reinterpret_cast<const uint4*>(gu)[2 * i + 1];
    const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
    uint32_t ow[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 gf = __half22float2(*reinterpret_cast<const __half2*>(&gw[k]));
        const float2 uf = __half22float2(*reinterpret_cast<const __half2*>(&uw[k]));
        const __half2 r = __floats2half2_rn(round_f16(silu_pf(gf.x)) * uf.x, round_f16(silu_pf(gf.y)) * uf.y);
        ow[k] = *reinterpret_cast<const uint32_t*>(&r);
    }
    reinterpret_cast<uint4*>(act)[i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

// ---------------------------------------------------------------------------------------------
// Gated DeltaNet over a chunk.  x: token-major in-projection output, row t =
// [ mixed (conv_dim = 2 key_dim + nv*128) | z (nv*128) | b (nv) | a (nv) ], ld halves per row.
// ---------------------------------------------------------------------------------------------
#define PF_DK 128

// four halves (inputs, a channel's window or weights): one 8-byte access where the pointer allows it
__device__ __forceinline__ uint2 ld_half4(const __half* p) {
    if (((uintptr_t)p & 7) == 0) return *reinterpret_cast<const uint2*>(p);
    const __half2 lo = __halves2half2(p[0], p[1]), hi = __halves2half2(p[2], p[3]);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// conv[t][c] = f16(silu(w0 x[t-3] + w1 x[t-2] + w2 x[t-1] + w3 x[t])), inputs before the chunk
// taken from the carried window state[c][0..3] (state[c][3] is the newest).  A thread owns four
// adjacent channels and T tokens, so every input is loaded once (8 bytes at a time) plus the three before
// its first token.  T = 8 for long chunks (512 tokens of 10240 channels 24.1 -> 11.2 us against a thread
// per channel and token); short ones would leave most SMs empty and take T = 2.  WIDE: x is 8-byte aligned
// (it may start at any element; deciding per load instead costs a layer of 512 tokens 1 us).
template <int T, bool WIDE>
__global__ void __launch_bounds__(128)
dn_conv_tokens_kernel(const __half* __restrict__ x, long long ld, const __half* __restrict__ conv_w,
                      const __half* __restrict__ conv_state, __half* __restrict__ conv_out,
                      int conv_dim, int n) {
    pdl_prologue();
    PDL_FRESH(x); PDL_FRESH(conv_w); PDL_FRESH(conv_state); PDL_FRESH(conv_out);
    const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
    const int t0 = blockIdx.y * T;
    if (c >= conv_dim) return;
    auto unpack = [](const uint2 u, float (&f)[4]) {
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
        const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        f[0] = lo.x; f[1] = lo.y; f[2] = hi.x; f[3] = hi.y;
    };
    float w[4][4];                     // channel, tap
#pragma unroll
    for (int e = 0; e < 4; e++) unpack(ld_half4(conv_w + (size_t)(c + e) * 4), w[e]);
    float win[T + 3][4];               // token t0 - 3 + i, channel
#pragma unroll
    for (int i = 0; i < T + 3; i++) {
        const int t = t0 - 3 + i;
        uint2 u = make_uint2(0u, 0u);
        if (t >= 0 && t < n) u = WIDE ? *reinterpret_cast<const uint2*>(x + (size_t)t * ld + c) : ld_half4(x + (size_t)t * ld + c);
        unpack(u, win[i]);
    }
    if (t0 < 3) {                      // (T = 2: the second strip still reaches back to the carried window)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            float old[4];
            unpack(ld_half4(conv_state + (size_t)(c + e) * 4), old);
#pragma unroll
            for (int i = 0; i < 3; i++)          // input t < 0 is old[4 + t]
                if (t0 == 0) win[i][e] = old[1 + i];
                else if (t0 == 2 && i == 0) win[i][e] = old[3];
        }
    }
#pragma unroll
    for (int i = 0; i < T; i++) {
        if (t0 + i >= n) break;
        float r[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            float acc = w[e][0] * win[i][e];
            acc = fmaf(w[e][1], win[i + 1][e], acc);
            acc = fmaf(w[e][2], win[i + 2][e], acc);
            acc = fmaf(w[e][3], win[i + 3][e], acc);
            r[e] = silu_pf(acc);
        }
        const __half2 lo = __floats2half2_rn(r[0], r[1]), hi = __floats2half2_rn(r[2], r[3]);
        *reinterpret_cast<uint2*>(conv_out + (size_t)(t0 + i) * conv_dim + c) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
}

// The recurrence is evaluated in blocks of DNB tokens (see dn_scan_kernel); per value head and block
// dn_block_kernel leaves these coefficients, with P(j..i) = e^g_j ... e^g_i:
//   c[i][m] = P(m+1..i) k_i . k_m for m < i, 0 above
//   d[i][j] = P(j+1..i) q_i . k_j for j <= i, 0 above
//   gam[i]  = P(0..i)       (what is left of the state that enters the block when token i sees it)
//   tail[i] = P(i+1..DNB-1) (what is left of token i's update when the block ends)
// Tokens past the end of the chunk count as k = q = 0, beta = 0, e^g = 1: they change nothing.
#define DNB 4
struct __align__(16) DnBlock {
    float c[DNB][4];
    float d[DNB][4];
    float gam[DNB];
    float tail[DNB];
    float beta[DNB];
};

// One warp per (key head, block of DNB tokens): L2-normalised q (x 128^-1/2) and k as fp32, their
// products inside the block, and for each value head of the key head beta = f16(sigmoid(b)), the
// decay e^g with g = -exp(A_log) softplus(a + dt_bias), and the block's coefficients.
__global__ void __launch_bounds__(128)
dn_block_kernel(const __half* __restrict__ conv_out, int conv_dim, const __half* __restrict__ x,
                long long ld, const __half* __restrict__ A_log, const __half* __restrict__ dt_bias,
                float* __restrict__ qn, float* __restrict__ kn, DnBlock* __restrict__ blocks, int nk,
                int nv, int n) {
    pdl_prologue();
    PDL_FRESH(conv_out); PDL_FRESH(x); PDL_FRESH(A_log); PDL_FRESH(dt_bias); PDL_FRESH(qn); PDL_FRESH(kn);
    PDL_FRESH(blocks);
    const int lane = threadIdx.x & 31, kh = blockIdx.x * 4 + (threadIdx.x >> 5), blk = blockIdx.y;
    if (kh >= nk) return;
    const int key_dim = nk * PF_DK, rep = nv / nk;
    float4 q[DNB], k[DNB];
#pragma unroll
    for (int i = 0; i < DNB; i++) {
        const int t = blk * DNB + i;
        float4 qv = make_float4(0.0f, 0.0f, 0.0f, 0.0f), kv = qv;
        if (t < n) {
            const __half* row = conv_out + (size_t)t * conv_dim;
            const uint2 a = *reinterpret_cast<const uint2*>(row + kh * PF_DK + lane * 4);
            const uint2 b = *reinterpret_cast<const uint2*>(row + key_dim + kh * PF_DK + lane * 4);
            const float2 a0 = __half22float2(*reinterpret_cast<const __half2*>(&a.x));
            const float2 a1 = __half22float2(*reinterpret_cast<const __half2*>(&a.y));
            const float2 b0 = __half22float2(*reinterpret_cast<const __half2*>(&b.x));
            const float2 b1 = __half22float2(*reinterpret_cast<const __half2*>(&b.y));
            qv = make_float4(a0.x, a0.y, a1.x, a1.y);
            kv = make_float4(b0.x, b0.y, b1.x, b1.y);
        }
        const float qss = warp_sum(qv.x * qv.x + qv.y * qv.y + qv.z * qv.z + qv.w * qv.w);
        const float kss = warp_sum(kv.x * kv.x + kv.y * kv.y + kv.z * kv.z + kv.w * kv.w);
        const float inv_q = rsqrtf(qss + 1e-6f) * 0.08838834764831845f;
        const float inv_k = rsqrtf(kss + 1e-6f);
        q[i] = make_float4(qv.x * inv_q, qv.y * inv_q, qv.z * inv_q, qv.w * inv_q);
        k[i] = make_float4(kv.x * inv_k, kv.y * inv_k, kv.z * inv_k, kv.w * inv_k);
        // rows up to the end of the block exist in the workspace (zeros past the chunk's end)
        const size_t o = ((size_t)kh * gridDim.y * DNB + t) * PF_DK + lane * 4;      // [key head][token]
        *reinterpret_cast<float4*>(qn + o) = q[i];
        *reinterpret_cast<float4*>(kn + o) = k[i];
    }
    float kk[DNB][DNB], qk[DNB][DNB];
#pragma unroll
    for (int i = 0; i < DNB; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) {
            qk[i][j] = warp_sum(q[i].x * k[j].x + q[i].y * k[j].y + q[i].z * k[j].z + q[i].w * k[j].w);
            kk[i][j] = j < i ? warp_sum(k[i].x * k[j].x + k[i].y * k[j].y + k[i].z * k[j].z + k[i].w * k[j].w) : 0.0f;
        }
    // A lane per (value head, token of the block): its beta and decay, then its row of the coefficients.  (With one
    // lane for a head's four tokens a chunk waits for it: a layer of 5 tokens 14.1 -> 12.7 us, of 512 143.5 -> 142.7.)
    const int i = lane & 3, t = blk * DNB + i;
    float ki[4], qi[4];                            // row i of the products
#pragma unroll
    for (int j = 0; j < DNB; j++) {
        ki[j] = qi[j] = 0.0f;
#pragma unroll
        for (int m = j; m < DNB; m++)
            if (m == i) {
                ki[j] = kk[m][j];
                qi[j] = qk[m][j];
            }
    }
    for (int r0 = 0; r0 < rep; r0 += 8) {
        const int r = r0 + (lane >> 2), h = kh * rep + min(r, rep - 1);
        float e = 1.0f, beta = 0.0f;
        if (t < n) {
            const float decay = -expf(__half2float(A_log[h])), dt = __half2float(dt_bias[h]);
            const __half* row = x + (size_t)t * ld + conv_dim + (size_t)nv * PF_DK;
            beta = round_f16(1.0f / (1.0f + expf(-__half2float(row[h]))));
            e = expf(decay * softplus_pf(__half2float(row[nv + h]) + dt));
        }
        float eg[DNB];
#pragma unroll
        for (int j = 0; j < DNB; j++) eg[j] = __shfl_sync(0xffffffffu, e, (lane & 28) + j);
        float c[4], d[4], p = 1.0f;                // p = P(j+1..i) while j counts down
#pragma unroll
        for (int j = DNB - 1; j >= 0; j--) {
            if (j + 1 < DNB && j < i) p *= eg[j + 1 < DNB ? j + 1 : j];
            c[j] = j < i ? p * ki[j] : 0.0f;
            d[j] = j <= i ? p * qi[j] : 0.0f;
        }
        float tail = 1.0f;
#pragma unroll
        for (int j = DNB - 1; j > 0; j--)
            if (j > i) tail *= eg[j];
        if (r < rep) {
            DnBlock& w = blocks[(size_t)h * gridDim.y + blk];
            *reinterpret_cast<float4*>(w.c[i]) = make_float4(c[0], c[1], c[2], c[3]);
            *reinterpret_cast<float4*>(w.d[i]) = make_float4(d[0], d[1], d[2], d[3]);
            w.gam[i] = p * eg[0];
            w.tail[i] = tail;
            w.beta[i] = beta;
        }
    }
}

// packed fp32 pair arithmetic (two IEEE fp32 operations per instruction)
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(*reinterpret_cast<unsigned long long*>(&d))
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
          "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(*reinterpret_cast<unsigned long long*>(&d))
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return d;
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The recurrence over the chunk, DNB = 4 tokens at a time.  Token by token,
//   delta_t = beta_t (v_t - e^g_t S k_t),  S <- e^g_t S + k_t delta_t,  o_t = S q_t,
// is a chain of two reductions over the lanes per token.  For a block of tokens all dot products can
// be taken with the state that ENTERS it, because what the block's own tokens add to S k_i and S q_i
// is known from their keys (coefficients of dn_block_kernel):
//   delta_i = beta_i (v_i - gam_i S k_i - sum_{m<i} c_im delta_m)
//   o_i = gam_i S q_i + sum_{j<=i} d_ij delta_j,   S <- gam_3 S + sum_i tail_i delta_i k_i
// so a block has ONE reduction and the state is scaled once.  Exact algebra, fp32 throughout.
// Two value rows' 256 state values live in the registers of 16 lanes (lane sub owns dims 64 j + 4 sub
// .. + 3 of both); a warp holds 4 rows.  The 16 sums of a block (8 per row) are reduced transposed:
// a lane gives away the half it will not own, four times (15 shuffles), and ends with one sum.  Bound by
// shared-memory wavefronts (k and q are read by every warp) and the length of the chain: one row in
// 8 lanes needs twice the reads of k and q (162 us for 512 tokens of 48 heads against 131), two rows in
// 8 lanes leave half of the warps (slower still); one token at a time took 231.
// Operands of SCAN_TB tokens are staged in shared memory by cp.async, double buffered, so the chain
// never waits on global memory.  o[t][h*128 + row] = f16(o_t[row]).
#define SCAN_WARPS 4
#define SCAN_ROWS (SCAN_WARPS * 4)
#define SCAN_TB 16
#define SCAN_NB (SCAN_TB / DNB)

struct ScanStage {
    float k[SCAN_TB][PF_DK];
    float q[SCAN_TB][PF_DK];
    DnBlock b[SCAN_NB];
    __half v[SCAN_TB][SCAN_ROWS];
};

__global__ void __launch_bounds__(SCAN_WARPS * 32)
dn_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
               const DnBlock* __restrict__ blocks, const __half* __restrict__ conv_out, int conv_dim,
               float* __restrict__ state, __half* __restrict__ o_out, int nk, int nv, int n) {
    pdl_prologue();
    PDL_FRESH(qn); PDL_FRESH(kn); PDL_FRESH(blocks); PDL_FRESH(conv_out); PDL_FRESH(state); PDL_FRESH(o_out);
    __shared__ __align__(16) ScanStage stage[2];
    const int per_head = PF_DK / SCAN_ROWS;                  // CTAs per value head
    const int h = blockIdx.x / per_head, part = blockIdx.x % per_head;
    const int kh = h / (nv / nk);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane & 15, mine = (lane >> 3) & 1, s8 = lane & 7;
    const int lrow = warp * 4 + (lane >> 4) * 2;             // first of this lane's two rows, in the CTA
    const int row0 = part * SCAN_ROWS + lrow;
    const int key_dim = nk * PF_DK;
    const int nb = (n + DNB - 1) / DNB;

    // Stage the operands of blocks [b0, b0 + SCAN_NB) into buffer b; blocks past the end are not read.  The
    // workspace keeps a head's rows together, so a thread's pieces lie a constant apart (with token-major
    // rows the copies' index arithmetic cost 4 %: a layer of 512 tokens 149 -> 143 us).
    constexpr int THREADS = SCAN_WARPS * 32;
    constexpr int PIECES = SCAN_TB * PF_DK / 4 / THREADS;    // 16-byte pieces of k (of q) per thread
    constexpr int BP = (int)sizeof(DnBlock) / 16, VP = SCAN_ROWS / 8;
    static_assert(SCAN_TB * PF_DK / 4 % THREADS == 0 && SCAN_TB * VP <= 32 && SCAN_NB * BP <= THREADS - 32, "one piece each");
    const float* kp = kn + (size_t)kh * nb * DNB * PF_DK + tid * 4;
    const float* qp = qn + (size_t)kh * nb * DNB * PF_DK + tid * 4;
    const __half* vp = conv_out + 2 * key_dim + h * PF_DK + part * SCAN_ROWS + (tid % VP) * 8;
    const uint8_t* bp = reinterpret_cast<const uint8_t*>(blocks + (size_t)h * nb) + (tid - 32) * 16;
    auto issue = [&](int b0, int b) {
        ScanStage& s = stage[b];
        const int nblk = min(SCAN_NB, nb - b0), t0 = b0 * DNB;
        float* ks = &s.k[0][0] + tid * 4;
        float* qs = &s.q[0][0] + tid * 4;
        const float* k0 = kp + (size_t)t0 * PF_DK;
        const float* q0 = qp + (size_t)t0 * PF_DK;
        if (nblk == SCAN_NB) {
#pragma unroll
            for (int i = 0; i < PIECES; i++) {
                cp_async_16(ks + i * THREADS * 4, k0 + i * THREADS * 4);
                cp_async_16(qs + i * THREADS * 4, q0 + i * THREADS * 4);
            }
        } else {
            for (int i = 0; i * THREADS + tid < nblk * DNB * (PF_DK / 4); i++) {
                cp_async_16(ks + i * THREADS * 4, k0 + i * THREADS * 4);
                cp_async_16(qs + i * THREADS * 4, q0 + i * THREADS * 4);
            }
        }
        if (tid < SCAN_TB * VP)                              // (tokens past the end repeat the last one)
            cp_async_16(&s.v[tid / VP][(tid % VP) * 8], vp + (size_t)min(t0 + tid / VP, n - 1) * conv_dim);
        if (tid >= 32 && tid - 32 < nblk * BP)
            cp_async_16(reinterpret_cast<uint8_t*>(&s.b[0]) + (tid - 32) * 16, bp + (size_t)b0 * sizeof(DnBlock));
        cp_async_commit();
    };

    float2 S[2][4];
    float* sp = state + ((size_t)h * PF_DK + row0) * PF_DK + sub * 4;
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float4 v = *reinterpret_cast<const float4*>(sp + (size_t)r * PF_DK + j * 64);
            S[r][2 * j] = make_float2(v.x, v.y);
            S[r][2 * j + 1] = make_float2(v.z, v.w);
        }

    const int nst = (nb + SCAN_NB - 1) / SCAN_NB;
    issue(0, 0);
    for (int st = 0; st < nst; st++) {
        const int cur = st & 1;
        if (st + 1 < nst) {
            issue((st + 1) * SCAN_NB, cur ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const ScanStage& s = stage[cur];
        const int bcount = min(SCAN_NB, nb - st * SCAN_NB);
        for (int bb = 0; bb < bcount; bb++) {
            float2 k[DNB][4];
            float dot[2][2 * DNB];                           // S k_i, then S q_i: this lane's part
#pragma unroll
            for (int i = 0; i < DNB; i++) {
                const float* ks = &s.k[bb * DNB + i][sub * 4];
                const float* qs = &s.q[bb * DNB + i][sub * 4];
                const float4 k0 = *reinterpret_cast<const float4*>(ks), k1 = *reinterpret_cast<const float4*>(ks + 64);
                const float4 q0 = *reinterpret_cast<const float4*>(qs), q1 = *reinterpret_cast<const float4*>(qs + 64);
                const float2 q[4] = {make_float2(q0.x, q0.y), make_float2(q0.z, q0.w), make_float2(q1.x, q1.y),
                                     make_float2(q1.z, q1.w)};
                k[i][0] = make_float2(k0.x, k0.y);
                k[i][1] = make_float2(k0.z, k0.w);
                k[i][2] = make_float2(k1.x, k1.y);
                k[i][3] = make_float2(k1.z, k1.w);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    float2 ak = fmul2(S[r][0], k[i][0]), aq = fmul2(S[r][0], q[0]);
#pragma unroll
                    for (int j = 1; j < 4; j++) {
                        ak = ffma2(S[r][j], k[i][j], ak);
                        aq = ffma2(S[r][j], q[j], aq);
                    }
                    dot[r][i] = ak.x + ak.y;
                    dot[r][DNB + i] = aq.x + aq.y;
                }
            }
            // lane sub ends with sum s8 of row `mine`
            float own;
            {
                float w8[8], w4[4], w2[2];
#pragma unroll
                for (int a = 0; a < 8; a++)
                    w8[a] = (mine ? dot[1][a] : dot[0][a]) + __shfl_xor_sync(0xffffffffu, mine ? dot[0][a] : dot[1][a], 8);
#pragma unroll
                for (int a = 0; a < 4; a++)
                    w4[a] = ((s8 & 4) ? w8[a + 4] : w8[a]) + __shfl_xor_sync(0xffffffffu, (s8 & 4) ? w8[a] : w8[a + 4], 4);
#pragma unroll
                for (int a = 0; a < 2; a++)
                    w2[a] = ((s8 & 2) ? w4[a + 2] : w4[a]) + __shfl_xor_sync(0xffffffffu, (s8 & 2) ? w4[a] : w4[a + 2], 2);
                own = ((s8 & 1) ? w2[1] : w2[0]) + __shfl_xor_sync(0xffffffffu, (s8 & 1) ? w2[0] : w2[1], 1);
            }
            const DnBlock& w = s.b[bb];
            const float4 gam = *reinterpret_cast<const float4*>(w.gam);
            const float4 beta = *reinterpret_cast<const float4*>(w.beta);
            const float4 tail = *reinterpret_cast<const float4*>(w.tail);
            const float4 c1 = *reinterpret_cast<const float4*>(w.c[1]);
            const float4 c2 = *reinterpret_cast<const float4*>(w.c[2]);
            const float4 c3 = *reinterpret_cast<const float4*>(w.c[3]);
            const float4 d = *reinterpret_cast<const float4*>(w.d[s8 & 3]);
            const float gq = w.gam[s8 & 3];
            const int t0 = (st * SCAN_NB + bb) * DNB;
            float p[DNB], v[DNB];
#pragma unroll
            for (int i = 0; i < DNB; i++) {
                p[i] = __shfl_sync(0xffffffffu, own, (lane & 24) + i);
                v[i] = __half2float(s.v[bb * DNB + i][lrow + mine]);
            }
            const float e0 = beta.x * (v[0] - gam.x * p[0]);
            const float e1 = beta.y * ((v[1] - gam.y * p[1]) - c1.x * e0);
            const float e2 = beta.z * (((v[2] - gam.z * p[2]) - c2.x * e0) - c2.y * e1);
            const float e3 = beta.w * ((((v[3] - gam.w * p[3]) - c3.x * e0) - c3.y * e1) - c3.z * e2);
            float f[DNB] = {e0 * tail.x, e1 * tail.y, e2 * tail.z, e3 * tail.w};
            if (t0 + DNB > n) {                              // a place past the end adds nothing, also where zero
#pragma unroll                                               // times what the block holds is not zero
                for (int i = 1; i < DNB; i++)
                    if (t0 + i >= n) f[i] = 0.0f;
            }
            float g[DNB];                                    // the other row's
#pragma unroll
            for (int i = 0; i < DNB; i++) g[i] = __shfl_xor_sync(0xffffffffu, f[i], 8);
            const float2 g2 = make_float2(gam.w, gam.w);
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float2 a = fmul2(S[r][j], g2);
#pragma unroll
                    for (int i = 0; i < DNB; i++) {
                        const float fi = mine == r ? f[i] : g[i];
                        a = ffma2(k[i][j], make_float2(fi, fi), a);
                    }
                    S[r][j] = a;
                }
            if (s8 >= 4 && t0 + (s8 & 3) < n) {              // token s8 - 4 of the block
                // a later token's delta stays out even if it is not finite
                float o = fmaf(d.x, e0, gq * own);
                if (s8 >= 5) o = fmaf(d.y, e1, o);
                if (s8 >= 6) o = fmaf(d.z, e2, o);
                if (s8 >= 7) o = fmaf(d.w, e3, o);
                o_out[((size_t)(t0 + (s8 & 3)) * nv + h) * PF_DK + row0 + mine] = __float2half(o);
            }
        }
        __syncthreads();     // everyone is done with this buffer before it is refilled
    }
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
        for (int j = 0; j < 2; j++)
            *reinterpret_cast<float4*>(sp + (size_t)r * PF_DK + j * 64) =
                make_float4(S[r][2 * j].x, S[r][2 * j].y, S[r][2 * j + 1].x, S[r][2 * j + 1].y);
}

// Unused dynamic shared memory that lets no SM take more than its share of the scan's CTAs.  They are
// launched while the kernel before still holds some SMs (programmatic dependent launch) and would
// otherwise crowd the free ones, for the whole chunk: a layer of 512 tokens 249 -> 180 us.
static size_t scan_padding(int ctas) {
    static int sms[NVFP4_MAX_DEVICES] = {0};
    static bool opted[NVFP4_MAX_DEVICES] = {false};
    constexpr int SM_BYTES = 227 * 1024, RESERVED = 1024;
    constexpr int MOST = (SM_BYTES - RESERVED - (int)(2 * sizeof(ScanStage))) & ~127;
    const int dev = current_device_index();
    if (!sms[dev] && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    // the opt-in is the same whatever this call needs: another thread's first call cannot lower it
    if (!opted[dev]) {
        if (cudaFuncSetAttribute(dn_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        opted[dev] = true;
    }
    const int per_sm = (ctas + sms[dev] - 1) / sms[dev];
    const int pad = (SM_BYTES / per_sm - RESERVED - (int)(2 * sizeof(ScanStage))) & ~127;
    return pad > 0 ? (size_t)pad : 0;
}

// gated norm per (token, value head): out = f16( f32(f16(o rsqrt(mean(o^2) + eps)) * norm_w) * silu(z) )
// A warp per (token, head), lane owns 4 of the head's 128 outputs; eight warps a CTA (one-warp
// CTAs: 27.4 -> 8.7 us for 512 tokens of 48 heads).  The kernel also stores the carried conv window (the
// last four inputs): the conv kernel, which reads the old one, has finished by then.  The grid covers
// conv_dim threads.
__global__ void __launch_bounds__(256)
dn_post_kernel(const __half* __restrict__ o_in, const __half* __restrict__ x, long long ld,
               int conv_dim, const __half* __restrict__ norm_w, __half* __restrict__ out,
               __half* __restrict__ conv_state, int nv, int n, float rms_eps) {
    pdl_prologue();
    PDL_FRESH(o_in); PDL_FRESH(x); PDL_FRESH(norm_w); PDL_FRESH(out); PDL_FRESH(conv_state);
    const int id = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int t = id / nv, h = id % nv;
    if (const int c = blockIdx.x * 256 + threadIdx.x; c < conv_dim) {
        __half old[4], nw[4];
#pragma unroll
        for (int j = 0; j < 4; j++) old[j] = conv_state[(size_t)c * 4 + j];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int tt = n - 4 + j;
            nw[j] = (tt >= 0) ? x[(size_t)tt * ld + c] : old[4 + tt];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) conv_state[(size_t)c * 4 + j] = nw[j];
    }
    if (t >= n) return;
    const uint2 ov = *reinterpret_cast<const uint2*>(o_in + ((size_t)t * nv + h) * PF_DK + lane * 4);
    const __half* oh = reinterpret_cast<const __half*>(&ov);
    float o[4], ss = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        o[j] = __half2float(oh[j]);
        ss = fmaf(o[j], o[j], ss);
    }
    ss = warp_sum(ss);
    const float inv = rsqrtf(ss / (float)PF_DK + rms_eps);
    const __half* z = x + (size_t)t * ld + conv_dim + (size_t)h * PF_DK + lane * 4;
    __half res[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const __half hw = __hmul(__float2half(o[j] * inv), norm_w[lane * 4 + j]);
        res[j] = __float2half(__half2float(hw) * silu_pf(__half2float(z[j])));
    }
    *reinterpret_cast<uint2*>(out + ((size_t)t * nv + h) * PF_DK + lane * 4) =
        *reinterpret_cast<const uint2*>(res);
}

}  // namespace nvfp4

extern "C" {

// dst[c][r] = src[r][c], r < R, c < C; dst rows ld_dst >= R long, the tail zero-filled.
int launch_transpose_f16(const void* src, long long ld_src, void* dst, long long ld_dst, int R,
                         int C, void* stream) {
    if (!src || !dst || R <= 0 || C <= 0 || ld_src < C || ld_dst < R) return -1;
    const dim3 grid((C + 63) / 64, (unsigned)((ld_dst + 63) / 64));
    return nvfp4::launch_pdl(nvfp4::transpose_f16_kernel, grid, dim3(256), 0, (cudaStream_t)stream,
                             (const __half*)src, ld_src, (__half*)dst, ld_dst, R, C) == cudaSuccess
               ? 0 : -1;
}

// h[t][c] += dT[c][t] (fp32 add, one fp16 rounding), t < n, c < C; h rows C long, dT rows ldT long.
int launch_add_transposed(void* h, const void* dT, long long ldT, int n, int C, void* stream) {
    if (!h || !dT || n <= 0 || C <= 0 || ldT < n) return -1;
    const dim3 grid((n + 63) / 64, (C + 63) / 64);
    return nvfp4::launch_pdl(nvfp4::add_transposed_kernel, grid, dim3(256), 0, (cudaStream_t)stream,
                             (__half*)h, (const __half*)dT, ldT, n, C) == cudaSuccess ? 0 : -1;
}

// out[t][0..hidden) = table[ids[t]], ids: device int64 [n].
int launch_embed_rows(const void* table, const void* ids, void* out, int n, int hidden,
                      long long vocab, void* stream) {
    if (!table || !ids || !out || n <= 0 || n > 65535 || hidden <= 0 || vocab <= 0) return -1;
    const dim3 grid((hidden + 2047) / 2048, n);
    return nvfp4::launch_pdl(nvfp4::embed_rows_kernel, grid, dim3(256), 0, (cudaStream_t)stream,
                             (const __half*)table, (const long long*)ids, (__half*)out, hidden,
                             vocab) == cudaSuccess ? 0 : -1;
}

// gu: token-minor [2 * inter][N] with gate/up rows interleaved in groups of 8; act: [inter][N].
int launch_silu_mul_rows(const void* gu, void* act, int inter, int N, void* stream) {
    if (!gu || !act || inter <= 0 || inter % 8 != 0 || inter > 65535 || N <= 0) return -1;
    const uintptr_t at = (uintptr_t)gu | (uintptr_t)act;
    // eight tokens a thread once that fills the GPU (1024 rows of 512 tokens 1.9 us with two, 2.5 with eight;
    // of 2048 5.7 and 4.2)
    const bool wide = N % 8 == 0 && (at & 15) == 0 && (long long)inter * N >= (1LL << 20);
    const bool even = N % 2 == 0 && (at & 3) == 0;
    const auto kernel = wide   ? nvfp4::silu_mul_rows_kernel<8, false>
                        : even ? nvfp4::silu_mul_rows_kernel<2, false>
                               : nvfp4::silu_mul_rows_kernel<2, true>;
    const long long groups = wide ? N / 8 : ((long long)N + 1) / 2, items = (long long)inter * groups;
    const bool flat = inter > 8 * nvfp4::device_sms(nvfp4::current_device_index()) && items < 0x7fffff00LL;
    const dim3 grid = flat ? dim3((unsigned)((items + 255) / 256)) : dim3((unsigned)((groups + 255) / 256), (unsigned)inter);
    return nvfp4::launch_pdl(kernel, grid, dim3(256), 0, (cudaStream_t)stream, (const __half*)gu, (__half*)act, inter, N,
                             flat) == cudaSuccess ? 0 : -1;
}

// gu: token-major [n][2 * inter] with gate/up columns interleaved in groups of 8; act: [n][inter].
int launch_silu_mul_tokens(const void* gu, void* act, int inter, int n, void* stream) {
    if (!gu || !act || inter <= 0 || inter % 8 != 0 || n <= 0 || (((uintptr_t)gu | (uintptr_t)act) & 15) != 0) return -1;
    const long long pieces = (long long)inter / 8 * n, blocks = (pieces + 255) / 256;
    if (blocks > 0x7fffffffLL) return -1;
    return nvfp4::launch_pdl(nvfp4::silu_mul_tokens_kernel, dim3((unsigned)blocks), dim3(256), 0, (cudaStream_t)stream,
                             (const __half*)gu, (__half*)act, pieces) == cudaSuccess ? 0 : -1;
}

// Bytes of workspace launch_dn_prefill needs for n tokens.
long long nvfp4_dn_prefill_work_bytes(int n, int nk, int nv) {
    if (n <= 0 || nk <= 0 || nv <= 0) return -1;
    const long long conv_dim = (2LL * nk + nv) * PF_DK;
    long long b = (long long)n * conv_dim * 2;            // conv output, fp16
    b = (b + 255) & ~255LL;
    const long long nb = (n + DNB - 1) / DNB;              // blocks of the recurrence
    long long blocks = 2LL * nb * DNB * nk * PF_DK * 4;    // normalised q and k, fp32
    blocks += nb * nv * (long long)sizeof(nvfp4::DnBlock); // the blocks' coefficients
    blocks = (blocks + 255) & ~255LL;
    // (never less than for fewer tokens: 64 of 64 heads go in one block of 64, 65 four at a time, which takes less)
    if (nvfp4::dn_chunk_takes(n, nv) || nvfp4::dn_chunk_takes(n / 64 * 64, nv))
        blocks = std::max(blocks, nvfp4::dn_chunk_work_bytes(n, nk, nv));
    b += blocks;
    b += (long long)n * nv * PF_DK * 2;                    // recurrence output, fp16
    return b + 256;
}

// One Gated-DeltaNet layer over a chunk of n tokens.  x: token-major in-projection output
// [n][ld], row = [mixed | z | b | a]; conv_w, conv_state fp16 [conv_dim][4]; A_log, dt_bias fp16
// [nv]; norm_w fp16 [128]; state fp32 [nv][128][128] (value-row major), updated; out token-major
// [n][nv * 128].  nv a multiple of nk.  Four launches on `stream`.  0; -1 bad arguments; -2 launch.
int launch_dn_prefill(const void* x, long long ld, const void* conv_w, void* conv_state,
                      const void* A_log, const void* dt_bias, const void* norm_w, void* state,
                      void* work, long long work_bytes, void* out, int n, int nk, int nv,
                      float rms_eps, void* stream) {
    if (!x || !conv_w || !conv_state || !A_log || !dt_bias || !norm_w || !state || !work || !out)
        return -1;
    if (n <= 0 || n > 65535 || nk <= 0 || nv <= 0 || nv % nk != 0) return -1;
    const int conv_dim = (2 * nk + nv) * PF_DK;
    if (ld < (long long)conv_dim + (long long)nv * PF_DK + 2LL * nv || (ld & 3)) return -1;
    if (work_bytes < nvfp4_dn_prefill_work_bytes(n, nk, nv) || ((uintptr_t)work & 255)) return -1;
    unsigned char* w = (unsigned char*)work;
    __half* conv_out = (__half*)w;
    long long off = ((long long)n * conv_dim * 2 + 255) & ~255LL;
    cudaStream_t st = (cudaStream_t)stream;
    const __half* xh = (const __half*)x;
    bool ok = true;
    const int conv_t = n > 128 ? 8 : 2;
    const bool wide = ((uintptr_t)x & 7) == 0;                  // (ld is a multiple of 4)
    const auto conv = conv_t == 8 ? (wide ? nvfp4::dn_conv_tokens_kernel<8, true> : nvfp4::dn_conv_tokens_kernel<8, false>)
                                  : (wide ? nvfp4::dn_conv_tokens_kernel<2, true> : nvfp4::dn_conv_tokens_kernel<2, false>);
    ok = ok && nvfp4::launch_pdl(conv, dim3((conv_dim + 511) / 512, (n + conv_t - 1) / conv_t), dim3(128), 0, st, xh, ld,
                                 (const __half*)conv_w, (const __half*)conv_state, conv_out, conv_dim,
                                 n) == cudaSuccess;
    __half* o16;
    if (nvfp4::dn_chunk_takes(n, nv)) {
        void* blocks = w + off;
        o16 = (__half*)(w + off + nvfp4::dn_chunk_work_bytes(n, nk, nv));
        ok = ok && nvfp4::dn_chunk_launch(conv_out, conv_dim, xh, ld, (const __half*)A_log, (const __half*)dt_bias,
                                          (float*)state, blocks, o16, n, nk, nv, st) == cudaSuccess;
    } else {
        float* qn = (float*)(w + off);
        const int nb = (n + DNB - 1) / DNB;
        float* kn = qn + (size_t)nb * DNB * nk * PF_DK;
        off += 2LL * nb * DNB * nk * PF_DK * 4;
        nvfp4::DnBlock* blocks = (nvfp4::DnBlock*)(w + off);
        off = (off + (long long)nb * nv * (long long)sizeof(nvfp4::DnBlock) + 255) & ~255LL;
        o16 = (__half*)(w + off);
        ok = ok && nvfp4::launch_pdl(nvfp4::dn_block_kernel, dim3((nk + 3) / 4, nb), dim3(128), 0,
                                     st, (const __half*)conv_out, conv_dim, xh, ld,
                                     (const __half*)A_log, (const __half*)dt_bias, qn, kn, blocks, nk,
                                     nv, n) == cudaSuccess;
        ok = ok && nvfp4::launch_pdl(nvfp4::dn_scan_kernel, dim3(nv * (PF_DK / SCAN_ROWS)),
                                     dim3(SCAN_WARPS * 32), nvfp4::scan_padding(nv * (PF_DK / SCAN_ROWS)), st,
                                     (const float*)qn, (const float*)kn, (const nvfp4::DnBlock*)blocks,
                                     (const __half*)conv_out, conv_dim, (float*)state, o16, nk, nv,
                                     n) == cudaSuccess;
    }
    ok = ok && nvfp4::launch_pdl(nvfp4::dn_post_kernel,
                                 dim3((unsigned)max((nv * n + 7) / 8, (conv_dim + 255) / 256)), dim3(256), 0, st,
                                 (const __half*)o16, xh, ld, conv_dim, (const __half*)norm_w,
                                 (__half*)out, (__half*)conv_state, nv, n, rms_eps) == cudaSuccess;
    return ok ? 0 : -2;
}

}  // extern "C"
