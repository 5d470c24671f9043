// What the W4A16 GEMM kernels share: dequantisation of a piece of a weight row and the output layouts.
#pragma once
#include "common.cuh"

namespace nvfp4 {

// output layouts of the W4A16 GEMM kernels
enum {
    GEMM_OUT_FM = 0,       // out[m][token]
    GEMM_OUT_TM = 1,       // out[token][m]
    GEMM_OUT_TM_ADD = 2,   // out[token][m] += result
    GEMM_OUT_TM_SILU = 3,  // out[token][m / 16 * 8 + m % 8] = silu(row m) * row m + 8, m % 16 < 8 (gemm_pair.cu only)
};

// 16 packed bytes (32 weights, two scale blocks) -> 16 words of fp16 pairs, scaled in fp16
__device__ __forceinline__ void gemm_dequant32(const uint4 p, uint32_t sc2, uint32_t (&o)[16]) {
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const __half2 s2 = __half2half2(__float2half(e8m0_to_f32((sc2 >> (8 * (j >> 1))) & 0xFFu)));
        uint32_t h[4];
        e2m1x8_to_half2x4(w[j], h[0], h[1], h[2], h[3]);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const __half2 t = __hmul2(*reinterpret_cast<const __half2*>(&h[e]), s2);
            o[4 * j + e] = *reinterpret_cast<const uint32_t*>(&t);
        }
    }
}

// Eight rows of one token to (or into) memory; `rows` of them exist, `vec`: p is 16-byte aligned.  `old`: what is
// there, if vec and all eight rows.  The caller reads it for all its pieces at once: read here, each read waited
// for the store before it (5120 x 6144 at 512 tokens added into the output 33.0 us, now 30.6; stored 29.4).
__device__ __forceinline__ void gemm_store_rows8(const uint4 val, __half* p, bool vec, int rows, bool add, const uint4 old) {
    const __half2* h2 = reinterpret_cast<const __half2*>(&val);
    if (vec && rows >= 8) {
        uint4 o = val;
        if (add) {
            const __half2* r2 = reinterpret_cast<const __half2*>(&old);
            __half2* o2 = reinterpret_cast<__half2*>(&o);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 a = __half22float2(h2[e]), b = __half22float2(r2[e]);
                o2[e] = __floats2half2_rn(a.x + b.x, a.y + b.y);
            }
        }
        *reinterpret_cast<uint4*>(p) = o;
    } else {
        const __half* h1 = reinterpret_cast<const __half*>(&val);
        for (int e = 0; e < 8 && e < rows; e++) {
            __half r = h1[e];
            if (add) r = __float2half(__half2float(r) + __half2float(p[e]));
            p[e] = r;
        }
    }
}

// Epilogue store of one 32-token block of a thread's row (v = 32 fp32 accumulator values), in the
// layout out_mode asks for.  m = this thread's row, mbase = first row of its 128-row tile,
// nb = first token of the block.  `piece` counts the token-major staging pieces of this column
// half (chalf); all four warps of a column half call this together.
__device__ __forceinline__ void gemm_store_block(const uint32_t (&v)[32], __half* out, int out_mode,
                                                 uint8_t* smem, int chalf, int& piece, int q, int lane,
                                                 int m, int mbase, int nb, int M, int N, int ld_out,
                                                 int n_out) {
    if (out_mode != GEMM_OUT_FM) {
        // Token-major: a thread holds one row's 32 tokens, memory wants one token's rows
        // together.  The four warps of this column half (128 rows) turn the 32 x 128 piece
        // over in shared memory - the operand ring is free once the accumulation has
        // retired - and then store 16 bytes (8 rows of one token) per thread.  Two staging
        // pieces alternate, so the one barrier per piece also orders a piece's writes
        // after the reads of the piece before last.  (Storing 2 bytes per lane straight
        // from the registers cost 4 us per 512-token GEMM, 23 us with the residual add.)
        __half* stg = reinterpret_cast<__half*>(smem + (chalf * 2 + (piece & 1)) * 8192);
        const int rr = q * 32 + lane;
#pragma unroll
        for (int j = 0; j < 32; j++) stg[j * 128 + rr] = __float2half(__uint_as_float(v[j]));
        asm volatile("bar.sync %0, 128;\n" ::"r"(1 + chalf) : "memory");
        const bool vec = ((ld_out & 7) == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
        uint4 old[4] = {};
        if (out_mode == GEMM_OUT_TM_ADD && vec) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int tg = nb + ((i * 128 + rr) >> 4), mg = mbase + (rr & 15) * 8;
                if (tg < n_out && mg + 8 <= M)
                    old[i] = *reinterpret_cast<const uint4*>(out + (size_t)tg * (size_t)ld_out + mg);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int pid = i * 128 + rr, tok = pid >> 4, part = pid & 15;
            const int tg = nb + tok, mg = mbase + part * 8;
            if (tg >= n_out || mg >= M) continue;
            const uint4 val = *reinterpret_cast<const uint4*>(stg + tok * 128 + part * 8);
            __half* p = out + (size_t)tg * (size_t)ld_out + mg;
            gemm_store_rows8(val, p, vec, M - mg, out_mode == GEMM_OUT_TM_ADD, old[i]);
        }
        piece++;
    } else if (m < M && nb < N) {
        __half* orow = out + (size_t)m * (size_t)N + nb;
        if (nb + 32 <= N) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
                uint4 o;
                __half2 t;
                t = __floats2half2_rn(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                o.x = *reinterpret_cast<uint32_t*>(&t);
                t = __floats2half2_rn(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                o.y = *reinterpret_cast<uint32_t*>(&t);
                t = __floats2half2_rn(__uint_as_float(v[j + 4]), __uint_as_float(v[j + 5]));
                o.z = *reinterpret_cast<uint32_t*>(&t);
                t = __floats2half2_rn(__uint_as_float(v[j + 6]), __uint_as_float(v[j + 7]));
                o.w = *reinterpret_cast<uint32_t*>(&t);
                *reinterpret_cast<uint4*>(orow + j) = o;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (nb + j < N) orow[j] = __float2half(__uint_as_float(v[j]));
        }
    }
}

}  // namespace nvfp4
