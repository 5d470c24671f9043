// Gated DeltaNet over a prompt chunk, 64 tokens at a time on the tensor cores.
//
// Token by token (a value head's state S is 128 rows of 128; e^g decay, beta update strength, q and k L2-normalised)
//   delta_t = beta_t (v_t - e^g_t S k_t),  S <- e^g_t S + delta_t k_t^T,  o_t = S q_t.
// For a block of C = 64 tokens that meets the state S, with P(j..i) = e^g_j ... e^g_i and G_i = P(0..i):
//   R_i  = beta_i (v_i - G_i S k_i)                             all products with the state that enters
//   (I + A) delta = R,        A[i][m] = beta_i P(m+1..i) k_i.k_m  (m < i)
//   delta = X R,              X = (I + A)^-1                      one 64 x 64 matrix per head and block
//   o_i  = G_i S q_i + sum_{j<=i} D[i][j] delta_j,  D[i][j] = P(j+1..i) q_i.k_j
//   S   <- G_63 S + sum_i P(i+1..63) delta_i k_i^T
// which is the same algebra with five contractions in the place of a chain of 64 steps.  X and D depend on q, k,
// beta and g only: dn_chunk_prep_kernel makes them for all heads and blocks at once, and the chain that is left
// (dn_chunk_scan_kernel) runs over n / 64 blocks.
//
// Precision: q and k are fp16 numbers times an fp32 norm, so the raw fp16 numbers are EXACT tensor-core operands and
// the norms scale the results.  The fp32 operands (S, R, delta, X, D) enter as two fp16 numbers: a row is scaled by a
// power of two that puts its largest element at 2^14..2^15, the first number is the element rounded to fp16 and the second
// 2^11 times what that leaves, with an accumulator of its own.  Together they hold 23 bits: within 2^-23 of the element
// down to 2^-28 of the row's largest, and within 2^-51 of the largest below.  (Without the 2^11 the second number goes
// subnormal from 2^-16 of the largest on: a token beside one 2^20 times as large kept 9 bits.)  fp32 has 24, so what is
// not a sum of many such products is kept out of them: X's unit diagonal and D's diagonal are applied in fp32, and delta
// times its factor meets the state as three numbers, which hold more than fp32 does.  Products of two split operands leave
// out low x low (2^-24 of the product).  Sums are fp32, and a block's update is summed on its own before it meets the
// state, so the state is rounded once per block.
// Measured against float64 from the same fp16 q, k, v (16 / 48 heads), four tokens at a time / this.  Error of the state, and
// share of the outputs that are not the correctly rounded fp16:
//   usual decays        512 tokens 6.9e-8 / 5.5e-8, 6.8e-5 / 5.2e-5       100 tokens 8.8e-8 / 6.3e-8, 7.3e-5 / 6.0e-5
//   hardly any decay    512 tokens 5.1e-6 / 3.1e-7, 7.5e-3 / 1.3e-3       100 tokens 1.4e-6 / 2.3e-7, 1.7e-3 / 9.6e-4
//   that and keys alike 512 tokens 4.4e-6 / 9.3e-7, 9.0e-3 / 3.5e-3       100 tokens 1.2e-6 / 5.3e-7, 2.1e-3 / 2.4e-3
//   large tokens first  512 tokens 7.7e-7 / 1.7e-7, 1.8e-4 / 1.0e-4       100 tokens 4.8e-7 / 1.2e-7, 1.8e-4 / 1.0e-4
// (With two numbers everywhere the first line is 1.0e-7, 1.4e-4, and without the 2^11 the last one 2.0e-5, 3.3e-2.)
#include <cstddef>

#include "common.cuh"
#include "dn_chunk.cuh"

#define DC 128              // dims of a head (keys and values)

namespace nvfp4 {

constexpr int CH = 64;                              // tokens of a block
constexpr int KLD = DC + 8, TLD = CH + 8;           // halves per row in shared memory: rows an odd multiple of 16 bytes

// what the prep kernel leaves per key head and block
struct __align__(16) DcKQ {
    __half k[CH][KLD];                              // raw fp16 keys and queries, zeros past the end of the chunk
    __half q[CH][KLD];
};
// per value head and block
struct __align__(16) DcHead {
    __half x_hi[CH][TLD], x_lo[CH][TLD];            // X below its diagonal, row i times a power of two (inverse in x_inv[i])
    __half d_hi[CH][TLD], d_lo[CH][TLD];            // D below its diagonal, the same
    float x_inv[CH], d_inv[CH];
    float beta[CH];
    float d_diag[CH];                               // D's diagonal: q_i.k_i
    float ksc[CH];                                  // G_i / |k_i|
    float qsc[CH];                                  // G_i / |q_i| / sqrt(128)
    float usc[CH], usl[CH];                         // P(i+1..63) / |k_i| and what its rounding to fp32 leaves
    float glast[4];                                 // G_63
    // for the token-by-token form (non-finite values only)
    float eg[CH], ik[CH], iq[CH];
};
static_assert(sizeof(DcKQ) % 16 == 0 && sizeof(DcHead) % 16 == 0, "copied in 16-byte pieces");
constexpr int DC_HEAD_COPY = (int)offsetof(DcHead, eg);      // bytes the scan stages
static_assert(DC_HEAD_COPY % 16 == 0, "copied in 16-byte pieces");

__device__ __forceinline__ void dc_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void dc_ldsm(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void dc_ldsm_t(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}

// Power of two that brings a row's largest magnitude to 2^14..2^15, and its inverse.  (Zero rows and rows below
// 2^-111 take the scale of 2^-111; infinite ones give NaN products, which the caller notices.)
__device__ __forceinline__ void dc_scale(float mx, float& s, float& inv) {
    const int ex = max((int)(__float_as_uint(mx) >> 23), 16);
    s = __uint_as_float((uint32_t)(268 - ex) << 23);
    inv = __uint_as_float((uint32_t)(ex - 14) << 23);
}
constexpr float DC_LO = 2048.0f, DC_LO_INV = 1.0f / 2048.0f;     // what a low half is scaled by
// Two fp32 numbers -> hi and lo fp16 pairs.
__device__ __forceinline__ void dc_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((x - f.x) * DC_LO, (y - f.y) * DC_LO);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
// The products x (u.x + ul.x) and y (u.y + ul.y), times s, as three fp16 pairs, the last on the scale of lo: what rounding
// the product to fp32 leaves goes into them as well.  (s, a power of two, only ever meets the product: it can be as large
// as that is small.)
__device__ __forceinline__ void dc_split3(float x, float y, const float2 u, const float2 ul, float s, uint32_t& hi,
                                          uint32_t& lo, uint32_t& rest) {
    const float px = x * u.x, py = y * u.y;
    const float ex = fmaf(x, ul.x, fmaf(x, u.x, -px)), ey = fmaf(y, ul.y, fmaf(y, u.y, -py));
    const __half2 h = __floats2half2_rn(px * s, py * s);
    const float2 f = __half22float2(h);
    const float rx = fmaf(ex, s, fmaf(px, s, -f.x)) * DC_LO, ry = fmaf(ey, s, fmaf(py, s, -f.y)) * DC_LO;
    const __half2 l = __floats2half2_rn(rx, ry);
    const float2 g = __half22float2(l);
    const __half2 r = __floats2half2_rn(rx - g.x, ry - g.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
    rest = *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ float dc_quad_max(float v) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
    return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
// A running sum of log decays as two fp32 numbers, and e^(a - b) with what the rounding of a - b to fp32 leaves (a
// difference as large as 10 loses 5e-7 of the result otherwise).
__device__ __forceinline__ float2 dc_two(double d) {
    const float h = (float)d;
    return make_float2(h, (float)(d - (double)h));
}
__device__ __forceinline__ float dc_exp(const float2 a, const float2 b) {
    const float x = a.x - b.x, t = x - a.x;                                 // x + r = a.x - b.x exactly
    const float r = (a.x - (x - t)) - (b.x + t), e = expf(x);
    return e == 0.0f ? 0.0f : fmaf(e, r + (a.y - b.y), e);
}
// 1 / sqrt(s): the fp32 approximation and one Newton step (where s is finite)
__device__ __forceinline__ double dc_rsqrt(double s) {
    const double y = (double)rsqrtf((float)s);
    return s < 1e38 ? fma(0.5 * y, fma(-s * y, y, 1.0), y) : y;
}

// One CTA per (value head, block): X and D with their scales, the scales of the other products, and (first value
// head of a key head) the block's keys and queries.  k.k and q.k are tensor-core products of the raw fp16 numbers.  The
// inverse of I + A (unit lower triangular) goes by blocks: 16 x 16 by substitution, a thread per column, then twice
// [X1 0; -X2 A21 X1, X2].  Sums run over the lower triangle only, so that a token with a non-finite value does
// not reach earlier ones.
struct DcPrepSmem {
    union {
        struct { __half k[CH][KLD], q[CH][KLD]; } kq;
        struct { float x[CH][CH + 4]; float y[32][36]; } inv;  // (I + A)^-1 and an intermediate: after the products
    };
    float a[CH][CH + 4];                            // k.k, then A
    float d[CH][CH + 4];                            // q.k
    double g[CH], ikd[CH], iqd[CH];                 // log G_i, the norms
    float2 g2[CH];
    float ik[CH], iq[CH], eg[CH], beta[CH];
};
static_assert(3 * (sizeof(DcPrepSmem) + 1024) <= 227 * 1024, "three CTAs an SM");

__global__ void __launch_bounds__(256, 3)
dn_chunk_prep_kernel(const __half* __restrict__ conv_out, int conv_dim, const __half* __restrict__ x, long long ld,
                     const __half* __restrict__ A_log, const __half* __restrict__ dt_bias, DcKQ* __restrict__ kq,
                     DcHead* __restrict__ heads, int nk, int nv, int n) {
    pdl_prologue();
    PDL_FRESH(conv_out); PDL_FRESH(x); PDL_FRESH(A_log); PDL_FRESH(dt_bias); PDL_FRESH(kq); PDL_FRESH(heads);
    extern __shared__ __align__(16) uint8_t dc_smem[];
    DcPrepSmem& s = *reinterpret_cast<DcPrepSmem*>(dc_smem);
    const int h = blockIdx.x, blk = blockIdx.y, nblk = gridDim.y, rep = nv / nk, kh = h / rep;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = blk * CH;
    DcHead& out = heads[(size_t)h * nblk + blk];
    DcKQ& okq = kq[(size_t)kh * nblk + blk];

    // warp 7's lanes: beta and decay of tokens 2 l and 2 l + 1 (requested first, used last)
    __half gb[2] = {}, ga[2] = {}, gl = {}, gd = {};
    if (warp == 7) {
        gl = A_log[h];
        gd = dt_bias[h];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int t = t0 + 2 * lane + e;
            if (t < n) {
                const __half* row = x + (size_t)t * ld + conv_dim + (size_t)nv * DC;
                gb[e] = row[h];
                ga[e] = row[nv + h];
            }
        }
    }
    // keys and queries: 16 lanes a row of 128
    uint4 kv[4], qv[4];
    const int c8 = (tid & 15) * 8;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int t = t0 + i * 16 + (tid >> 4);
        kv[i] = qv[i] = make_uint4(0u, 0u, 0u, 0u);
        if (t < n) {
            const __half* src = conv_out + (size_t)t * conv_dim + kh * DC + c8;
            qv[i] = *reinterpret_cast<const uint4*>(src);
            kv[i] = *reinterpret_cast<const uint4*>(src + nk * DC);
        }
    }
    double ks[4], qs[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = i * 16 + (tid >> 4);
        *reinterpret_cast<uint4*>(&s.kq.k[row][c8]) = kv[i];
        *reinterpret_cast<uint4*>(&s.kq.q[row][c8]) = qv[i];
        if (h == kh * rep) {
            *reinterpret_cast<uint4*>(&okq.k[row][c8]) = kv[i];
            *reinterpret_cast<uint4*>(&okq.q[row][c8]) = qv[i];
        }
        const uint32_t kw[4] = {kv[i].x, kv[i].y, kv[i].z, kv[i].w}, qw[4] = {qv[i].x, qv[i].y, qv[i].z, qv[i].w};
        float kp[4], qp[4];                          // sums of two squares
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&kw[e]));
            const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&qw[e]));
            kp[e] = fmaf(a.x, a.x, a.y * a.y);
            qp[e] = fmaf(b.x, b.x, b.y * b.y);
        }
        ks[i] = ((double)kp[0] + (double)kp[1]) + ((double)kp[2] + (double)kp[3]);
        qs[i] = ((double)qp[0] + (double)qp[1]) + ((double)qp[2] + (double)qp[3]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            ks[i] += __shfl_xor_sync(0xffffffffu, ks[i], o);
            qs[i] += __shfl_xor_sync(0xffffffffu, qs[i], o);
        }
    if ((tid & 15) < 4) {                            // lane i of a row's 16 finishes row i * 16 + ..
        const int i = tid & 15, row = i * 16 + (tid >> 4);
        const double k = dc_rsqrt((i == 0 ? ks[0] : i == 1 ? ks[1] : i == 2 ? ks[2] : ks[3]) + 1e-6);
        const double q = dc_rsqrt((i == 0 ? qs[0] : i == 1 ? qs[1] : i == 2 ? qs[2] : qs[3]) + 1e-6) * 0.08838834764831845;
        s.ikd[row] = k;
        s.iqd[row] = q;
        s.ik[row] = (float)k;
        s.iq[row] = (float)q;
    }
    __syncthreads();
    if (warp == 7) {                                 // (its products below are the fewest)
        const float decay = -expf(__half2float(gl)), dt = __half2float(gd);
        double g[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float gt = 0.0f, beta = 0.0f;
            if (t0 + 2 * lane + e < n) {
                beta = round_f16(1.0f / (1.0f + expf(-__half2float(gb[e]))));
                gt = decay * softplus_pf(__half2float(ga[e]) + dt);
                // e^g is 0 either way, but differences of the sums must exist and not lose the other tokens' decays
                if (gt < -200.0f) gt = -200.0f;
            }
            s.beta[2 * lane + e] = beta;
            s.eg[2 * lane + e] = expf(gt);
            g[e] = (double)gt;
        }
        double run = g[0] + g[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += up;
        }
        s.g[2 * lane] = run - g[1];
        s.g[2 * lane + 1] = run;
        s.g2[2 * lane] = dc_two(run - g[1]);
        s.g2[2 * lane + 1] = dc_two(run);
    }
    // warps 0..3: k.k, 4..7: q.k, 16 rows each, columns up to the diagonal
    {
        const int mt = warp < 4 ? warp : 7 - warp;
        const __half(*A)[KLD] = warp < 4 ? s.kq.k : s.kq.q;
        float(*C)[CH + 4] = warp < 4 ? s.a : s.d;
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.0f;
#pragma unroll 2
        for (int kk = 0; kk < DC / 16; kk++) {
            uint32_t a[4];
            dc_ldsm(a, &A[mt * 16 + (lane & 15)][kk * 16 + (lane >> 4) * 8]);
#pragma unroll
            for (int p = 0; p < 4; p++)
                if (p <= mt) {
                    uint32_t b[4];
                    dc_ldsm(b, &s.kq.k[p * 16 + (lane >> 4) * 8 + (lane & 7)][kk * 16 + ((lane >> 3) & 1) * 8]);
                    // (sixteen products at a time: the tensor core truncates the sum it adds to, the addition here rounds)
                    float c0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, c1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    dc_mma(c0, a, b[0], b[1]);
                    dc_mma(c1, a, b[2], b[3]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        acc[2 * p][e] += c0[e];
                        acc[2 * p + 1][e] += c1[e];
                    }
                }
        }
        const int r = mt * 16 + (lane >> 2), c = (lane & 3) * 2;
#pragma unroll
        for (int nt = 0; nt < 8; nt++)
            if (nt <= 2 * mt + 1) {
                *reinterpret_cast<float2*>(&C[r][nt * 8 + c]) = make_float2(acc[nt][0], acc[nt][1]);
                *reinterpret_cast<float2*>(&C[r + 8][nt * 8 + c]) = make_float2(acc[nt][2], acc[nt][3]);
            }
    }
    __syncthreads();
    // row i, columns part * 16 ..: A in place, D to global memory
    const int i = tid >> 2, part = tid & 3;
    auto store_row = [&](const float (&v)[16], __half* hi, __half* lo, float* inv_out) {
        float mx = 0.0f;
#pragma unroll
        for (int e = 0; e < 16; e++) mx = fmaxf(mx, fabsf(v[e]));
        float sc, inv;
        dc_scale(dc_quad_max(mx), sc, inv);
        uint32_t hw[8], lw[8];
#pragma unroll
        for (int e = 0; e < 8; e++) dc_split(v[2 * e] * sc, v[2 * e + 1] * sc, hw[e], lw[e]);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            reinterpret_cast<uint4*>(hi)[e] = make_uint4(hw[4 * e], hw[4 * e + 1], hw[4 * e + 2], hw[4 * e + 3]);
            reinterpret_cast<uint4*>(lo)[e] = make_uint4(lw[4 * e], lw[4 * e + 1], lw[4 * e + 2], lw[4 * e + 3]);
        }
        if (part == 0) *inv_out = inv;
    };
    {
        float dv[16];
        const float2 gi = s.g2[i];
        const float bk = s.beta[i] * s.ik[i], iqi = s.iq[i];
#pragma unroll
        for (int e4 = 0; e4 < 4; e4++) {
            const int j0 = part * 16 + e4 * 4;
            float av[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            dv[e4 * 4] = dv[e4 * 4 + 1] = dv[e4 * 4 + 2] = dv[e4 * 4 + 3] = 0.0f;
            if (j0 <= i) {
                const float4 a4 = *reinterpret_cast<const float4*>(&s.a[i][j0]);
                const float4 d4 = *reinterpret_cast<const float4*>(&s.d[i][j0]);
                const float4 k4 = *reinterpret_cast<const float4*>(&s.ik[j0]);
                const float aa[4] = {a4.x, a4.y, a4.z, a4.w}, dd[4] = {d4.x, d4.y, d4.z, d4.w}, kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int j = j0 + e;
                    const float p = dc_exp(gi, s.g2[j]) * kk[e];
                    const float d = p * (iqi * dd[e]);
                    if (j == i) out.d_diag[i] = d;
                    dv[e4 * 4 + e] = j < i ? d : 0.0f;                     // (selected, not multiplied: above the
                    av[e] = j < i ? p * (bk * aa[e]) : 0.0f;               // diagonal there is nothing to trust)
                }
            }
            *reinterpret_cast<float4*>(&s.a[i][j0]) = make_float4(av[0], av[1], av[2], av[3]);
        }
        store_row(dv, &out.d_hi[i][part * 16], &out.d_lo[i][part * 16], &out.d_inv[i]);
        if (part == 0) {
            const double gam = exp(s.g[i]), tail = exp(s.g[CH - 1] - s.g[i]);
            out.ksc[i] = (float)(gam * s.ikd[i]);
            out.qsc[i] = (float)(gam * s.iqd[i]);
            const double us = tail * s.ikd[i];
            out.usc[i] = (float)us;
            out.usl[i] = (float)(us - (double)(float)us);
            out.eg[i] = s.eg[i];
            out.beta[i] = s.beta[i];
            out.ik[i] = s.ik[i];
            out.iq[i] = iqi;
            if (i == CH - 1) out.glast[0] = out.glast[1] = out.glast[2] = out.glast[3] = (float)gam;
        }
    }
    __syncthreads();
    if (tid < CH) {                                  // 16 x 16 blocks on the diagonal: column m of block b
        const int b = tid >> 4, m = tid & 15;
        float xv[16];
#pragma unroll
        for (int r = 0; r < 16; r++) {
            float row[16];
#pragma unroll
            for (int l4 = 0; l4 < (r + 3) / 4; l4++)
                *reinterpret_cast<float4*>(&row[l4 * 4]) = *reinterpret_cast<const float4*>(&s.a[b * 16 + r][b * 16 + l4 * 4]);
            float acc = r == m ? 1.0f : 0.0f;
#pragma unroll
            for (int l = 0; l < r; l++) acc = fmaf(-row[l], xv[l], acc);
            xv[r] = r < m ? 0.0f : acc;
            s.inv.x[b * 16 + r][b * 16 + m] = xv[r];
        }
    }
    __syncthreads();
    // 32 x 32 blocks: X21 = -X22 (A21 X11), a thread has two columns of a row.  (In the second product the rows below r
    // are left out, not multiplied by zero: one of them may be a token with a value that is not finite.)
    {
        const int r0 = (tid >> 7) * 32, r = (tid & 127) >> 3, c = (tid & 7) * 2, yb = (tid >> 7) * 16;
        float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll 8
        for (int l = 0; l < 16; l++) {
            const float a = s.a[r0 + 16 + r][r0 + l];
            const float2 v = *reinterpret_cast<const float2*>(&s.inv.x[r0 + l][r0 + c]);
            acc.x = fmaf(a, v.x, acc.x);
            acc.y = fmaf(a, v.y, acc.y);
        }
        *reinterpret_cast<float2*>(&s.inv.y[yb + r][c]) = acc;
        __syncthreads();
        acc = make_float2(0.0f, 0.0f);
#pragma unroll 8
        for (int l = 0; l < 16; l++) {
            const float a = -s.inv.x[r0 + 16 + r][r0 + 16 + l];
            const float2 v = *reinterpret_cast<const float2*>(&s.inv.y[yb + l][c]);
            if (l <= r) {
                acc.x = fmaf(a, v.x, acc.x);
                acc.y = fmaf(a, v.y, acc.y);
            }
        }
        *reinterpret_cast<float2*>(&s.inv.x[r0 + 16 + r][r0 + c]) = acc;
    }
    __syncthreads();
    // the whole: 32 x 32 below the diagonal, a thread has four columns of a row
    {
        const int r = tid >> 3, c = (tid & 7) * 4;
        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
        for (int l = 0; l < 32; l++) {
            const float a = s.a[32 + r][l];
            const float4 v = *reinterpret_cast<const float4*>(&s.inv.x[l][c]);
            if (l >= (c & 16)) {                      // (above the 16 x 16 blocks on the diagonal nothing is written)
                acc.x = fmaf(a, v.x, acc.x); acc.y = fmaf(a, v.y, acc.y);
                acc.z = fmaf(a, v.z, acc.z); acc.w = fmaf(a, v.w, acc.w);
            }
        }
        *reinterpret_cast<float4*>(&s.inv.y[r][c]) = acc;
        __syncthreads();
        acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
        for (int l = 0; l < 32; l++) {
            const float a = -s.inv.x[32 + r][32 + l];
            const float4 v = *reinterpret_cast<const float4*>(&s.inv.y[l][c]);
            if (l <= r) {
                acc.x = fmaf(a, v.x, acc.x); acc.y = fmaf(a, v.y, acc.y);
                acc.z = fmaf(a, v.z, acc.z); acc.w = fmaf(a, v.w, acc.w);
            }
        }
        *reinterpret_cast<float4*>(&s.inv.x[32 + r][c]) = acc;
    }
    __syncthreads();
    {
        float xv[16];
#pragma unroll
        for (int e4 = 0; e4 < 4; e4++) {
            const int m0 = part * 16 + e4 * 4;
            const float4 x4 = *reinterpret_cast<const float4*>(&s.inv.x[i][m0]);
            const float xx[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
            for (int e = 0; e < 4; e++) xv[e4 * 4 + e] = m0 + e < i ? xx[e] : 0.0f;
        }
        store_row(xv, &out.x_hi[i][part * 16], &out.x_lo[i][part * 16], &out.x_inv[i]);
    }
}

// The tokens of one block for a warp's 16 rows, one after the other: for blocks in which something is not finite,
// where a product with a zero of X or D would spread it to earlier tokens.  The state rows are in global memory.
__device__ __noinline__ void dn_chunk_plain(float* state, const DcHead* head, const DcKQ* kq, const __half* v,
                                            int conv_dim, __half* o, int ldo, int count, int lane) {
    for (int r = 0; r < 16; r++) {
        float4 S = *reinterpret_cast<const float4*>(state + (size_t)r * DC + lane * 4);
        for (int t = 0; t < count; t++) {
            const __half2* kp = reinterpret_cast<const __half2*>(&kq->k[t][lane * 4]);
            const __half2* qp = reinterpret_cast<const __half2*>(&kq->q[t][lane * 4]);
            const float2 k0 = __half22float2(kp[0]), k1 = __half22float2(kp[1]);
            const float2 q0 = __half22float2(qp[0]), q1 = __half22float2(qp[1]);
            const float ik = head->ik[t], iq = head->iq[t], eg = head->eg[t];
            S.x *= eg; S.y *= eg; S.z *= eg; S.w *= eg;
            const float dot = warp_sum(S.x * (k0.x * ik) + S.y * (k0.y * ik) + S.z * (k1.x * ik) + S.w * (k1.y * ik));
            const float delta = head->beta[t] * (__half2float(v[(size_t)t * conv_dim + r]) - dot);
            S.x = fmaf(k0.x * ik, delta, S.x); S.y = fmaf(k0.y * ik, delta, S.y);
            S.z = fmaf(k1.x * ik, delta, S.z); S.w = fmaf(k1.y * ik, delta, S.w);
            const float out = warp_sum(S.x * (q0.x * iq) + S.y * (q0.y * iq) + S.z * (q1.x * iq) + S.w * (q1.y * iq));
            if (lane == 0) o[(size_t)t * ldo + r] = __float2half(out);
        }
        *reinterpret_cast<float4*>(state + (size_t)r * DC + lane * 4) = S;
    }
}

// The chain.  A pair of warps owns 16 rows of a head's state.  The first one, the chain warp, holds them as the
// accumulators of sixteen m16n8 tiles (dims 8 j .. 8 j + 7 in tile j) and goes from block to block: R, delta, next state.
// The second one, the output warp, makes o from the operands the first one leaves in shared memory (the split state that
// enters the block, delta), and requests the next block's k, q, X, D and v.  Two accumulator tiles packed
// to fp16 are the A operand of the next product, so what all rows share is all that has to pass through shared memory.
// The products of the small halves have accumulators of their own: the tensor core truncates the sum it adds to,
// and those of the large halves are then 8 (S k, S q) or up to 4 (the others) additions long.
template <int W>
struct DcScanSmem {
    static constexpr int VLD = W * 16 + 8;          // halves per token row: an odd multiple of 16 bytes
    struct Stage {
        DcKQ kq;
        uint8_t head[DC_HEAD_COPY];
        __half v[CH][VLD];
    } stage[2];
    uint4 s_hi[W][8][32], s_lo[W][8][32];           // A operands: the state that enters the block, 16 dims each
    float4 delta[W][8][32];                         // delta, 8 tokens each
    float2 s_inv[W][32];                            // what the rows g and g + 8 were scaled by
    int plain[W];
};

__device__ __forceinline__ void dc_pair_sync(int id) { asm volatile("bar.sync %0, 64;\n" ::"r"(id) : "memory"); }

// the A operands of rows g, g + 8 and 16 columns: accumulator tiles x, y times the rows' scales
__device__ __forceinline__ void dc_operand(const float (&x)[4], const float (&y)[4], float s0, float s1, uint32_t (&hi)[4],
                                           uint32_t (&lo)[4]) {
    dc_split(x[0] * s0, x[1] * s0, hi[0], lo[0]);
    dc_split(x[2] * s1, x[3] * s1, hi[1], lo[1]);
    dc_split(y[0] * s0, y[1] * s0, hi[2], lo[2]);
    dc_split(y[2] * s1, y[3] * s1, hi[3], lo[3]);
}
__device__ __forceinline__ uint4 dc_u4(const uint32_t (&r)[4]) { return make_uint4(r[0], r[1], r[2], r[3]); }
__device__ __forceinline__ void dc_from(const uint4 v, uint32_t (&r)[4]) { r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w; }
template <int N>
__device__ __forceinline__ void dc_zero(float (&a)[N][4]) {
#pragma unroll
    for (int i = 0; i < N; i++) a[i][0] = a[i][1] = a[i][2] = a[i][3] = 0.0f;
}
// largest magnitudes of rows g and g + 8 -> scales and inverses
template <int N>
__device__ __forceinline__ void dc_row_scales(const float (&a)[N][4], float& s0, float& s1, float& i0, float& i1) {
    float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
    for (int j = 0; j < N; j++) {
        m0 = fmaxf(m0, fmaxf(fabsf(a[j][0]), fabsf(a[j][1])));
        m1 = fmaxf(m1, fmaxf(fabsf(a[j][2]), fabsf(a[j][3])));
    }
    dc_scale(dc_quad_max(m0), s0, i0);
    dc_scale(dc_quad_max(m1), s1, i1);
}
// out[row][i] += sum over tokens 16 m .. 16 m + 15 of in[row][.] X[i][.] for i >= 16 m, X split in fp16 like the operand
__device__ __forceinline__ void dc_triangle(float (&oh)[8][4], float (&ol)[8][4], const uint32_t (&hi)[4],
                                            const uint32_t (&lo)[4], int m, const __half (*xh)[TLD], const __half (*xl)[TLD],
                                            int lr, int lc) {
#pragma unroll
    for (int p = 0; p < 4; p++)
        if (p >= m) {
            uint32_t bh[4], bl[4];
            dc_ldsm(bh, &xh[p * 16 + lr][m * 16 + lc]);
            dc_ldsm(bl, &xl[p * 16 + lr][m * 16 + lc]);
            dc_mma(oh[2 * p], hi, bh[0], bh[1]);
            dc_mma(oh[2 * p + 1], hi, bh[2], bh[3]);
            dc_mma(ol[2 * p], lo, bh[0], bh[1]);
            dc_mma(ol[2 * p + 1], lo, bh[2], bh[3]);
            dc_mma(ol[2 * p], hi, bl[0], bl[1]);
            dc_mma(ol[2 * p + 1], hi, bl[2], bl[3]);
        }
}

template <int W>
__global__ void __launch_bounds__(W * 64)
dn_chunk_scan_kernel(const DcKQ* __restrict__ kq, const DcHead* __restrict__ heads, const __half* __restrict__ conv_out,
                     int conv_dim, float* __restrict__ state, __half* __restrict__ o_out, int nk, int nv, int n) {
    pdl_prologue();
    PDL_FRESH(kq); PDL_FRESH(heads); PDL_FRESH(conv_out); PDL_FRESH(state); PDL_FRESH(o_out);
    extern __shared__ __align__(16) uint8_t dc_smem[];
    DcScanSmem<W>& sm = *reinterpret_cast<DcScanSmem<W>*>(dc_smem);
    constexpr int PER_HEAD = (DC / 16 + W - 1) / W;
    const int h = blockIdx.x / PER_HEAD, part = blockIdx.x % PER_HEAD, kh = h / (nv / nk);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = warp < W ? warp : warp - W;
    const int g = lane >> 2, t4 = lane & 3;
    const int row0 = (part * W + w) * 16;                    // this pair's first row of the head
    const bool active = row0 < DC;
    const int nblk = (n + CH - 1) / CH;
    const DcKQ* kqp = kq + (size_t)kh * nblk;
    const DcHead* hp = heads + (size_t)h * nblk;
    const __half* vbase = conv_out + 2 * nk * DC + h * DC;
    // addresses of this lane in the four 8 x 8 matrices of an ldmatrix: (row half, column half) = (bit 4, bit 3) for a B
    // operand stored [n][k]; the same matrices transposed serve a B operand stored [k][n] with the halves exchanged
    const int lr = (lane >> 4) * 8 + (lane & 7), lc = ((lane >> 3) & 1) * 8;
    const int tr = ((lane >> 3) & 1) * 8 + (lane & 7), tc = (lane >> 4) * 8;

    // (the output warps' threads)
    auto issue = [&](int c) {
        typename DcScanSmem<W>::Stage& s = sm.stage[c & 1];
        const int tid = threadIdx.x - W * 32;
        constexpr int T = W * 32;
        const uint8_t* a = reinterpret_cast<const uint8_t*>(kqp + c);
        const uint8_t* d = reinterpret_cast<const uint8_t*>(hp + c);
        uint8_t* sa = reinterpret_cast<uint8_t*>(&s.kq);
#pragma unroll 4
        for (int i = tid; i < (int)sizeof(DcKQ) / 16; i += T) cp_async_16(sa + i * 16, a + i * 16);
#pragma unroll 4
        for (int i = tid; i < DC_HEAD_COPY / 16; i += T) cp_async_16(s.head + i * 16, d + i * 16);
        // values: pieces of 8 rows per token; rows past the head's end and tokens past the chunk's end are not there
        const int rows = min(W * 16, DC - part * W * 16);
        for (int i = tid; i < CH * W * 2; i += T) {
            const int t = i / (W * 2), p = i - t * (W * 2);
            if (p * 8 >= rows) continue;
            __half* dst = &s.v[t][p * 8];
            if (c * CH + t < n) cp_async_16(dst, vbase + (size_t)(c * CH + t) * conv_dim + part * W * 16 + p * 8);
            else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    if (warp >= W) {
        // ---------------- output warps ----------------
        issue(0);
        for (int c = 0; c < nblk; c++) {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();                                 // block c's operands and the state that enters it are there
            if (c + 1 < nblk) issue(c + 1);                  // (block c - 1 is done with that buffer)
            if (!active) continue;
            const typename DcScanSmem<W>::Stage& s = sm.stage[c & 1];
            const DcHead& hd = *reinterpret_cast<const DcHead*>(s.head);
            const int count = min(CH, n - c * CH);
            float qh[8][4], ql[8][4];
            dc_zero(qh);
            dc_zero(ql);
#pragma unroll
            for (int kk = 0; kk < 8; kk++) {
                uint32_t hi[4], lo[4];
                dc_from(sm.s_hi[w][kk][lane], hi);
                dc_from(sm.s_lo[w][kk][lane], lo);
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    uint32_t q[4];
                    dc_ldsm(q, &s.kq.q[p * 16 + lr][kk * 16 + lc]);
                    dc_mma(qh[2 * p], hi, q[0], q[1]);
                    dc_mma(qh[2 * p + 1], hi, q[2], q[3]);
                    dc_mma(ql[2 * p], lo, q[0], q[1]);
                    dc_mma(ql[2 * p + 1], lo, q[2], q[3]);
                }
            }
            const float2 si = sm.s_inv[w][lane];
#pragma unroll
            for (int nt = 0; nt < 8; nt++) {
                const float2 qs = *reinterpret_cast<const float2*>(&hd.qsc[nt * 8 + t4 * 2]);
                qh[nt][0] = fmaf(ql[nt][0], DC_LO_INV, qh[nt][0]) * si.x * qs.x;
                qh[nt][1] = fmaf(ql[nt][1], DC_LO_INV, qh[nt][1]) * si.x * qs.y;
                qh[nt][2] = fmaf(ql[nt][2], DC_LO_INV, qh[nt][2]) * si.y * qs.x;
                qh[nt][3] = fmaf(ql[nt][3], DC_LO_INV, qh[nt][3]) * si.y * qs.y;
            }
            dc_pair_sync(1 + w);                             // delta is there; the entering state has been read
            if (sm.plain[w]) continue;                       // (the chain warp writes this block's outputs)
            float oh[8][4], ol[8][4], dl[8][4], s0, s1, i0, i1;
#pragma unroll
            for (int nt = 0; nt < 8; nt++) {
                const float4 d4 = sm.delta[w][nt][lane];
                const float2 dd = *reinterpret_cast<const float2*>(&hd.d_diag[nt * 8 + t4 * 2]);
                dl[nt][0] = d4.x; dl[nt][1] = d4.y; dl[nt][2] = d4.z; dl[nt][3] = d4.w;
                qh[nt][0] = fmaf(d4.x, dd.x, qh[nt][0]);
                qh[nt][1] = fmaf(d4.y, dd.y, qh[nt][1]);
                qh[nt][2] = fmaf(d4.z, dd.x, qh[nt][2]);
                qh[nt][3] = fmaf(d4.w, dd.y, qh[nt][3]);
            }
            dc_row_scales(dl, s0, s1, i0, i1);
            dc_zero(oh);
            dc_zero(ol);
#pragma unroll
            for (int m = 0; m < 4; m++) {
                uint32_t hi[4], lo[4];
                dc_operand(dl[2 * m], dl[2 * m + 1], s0, s1, hi, lo);
                dc_triangle(oh, ol, hi, lo, m, hd.d_hi, hd.d_lo, lr, lc);
            }
            __half* op = o_out + ((size_t)(c * CH + t4 * 2) * nv + h) * DC + row0 + g;
#pragma unroll
            for (int nt = 0; nt < 8; nt++) {
                const float2 di = *reinterpret_cast<const float2*>(&hd.d_inv[nt * 8 + t4 * 2]);
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (nt * 8 + t4 * 2 + u < count) {
                        const float dt = u ? di.y : di.x;
                        __half* o = op + (size_t)(nt * 8 + u) * nv * DC;
                        o[0] = __float2half(fmaf(fmaf(ol[nt][u], DC_LO_INV, oh[nt][u]) * i0, dt, qh[nt][u]));
                        o[8] = __float2half(fmaf(fmaf(ol[nt][2 + u], DC_LO_INV, oh[nt][2 + u]) * i1, dt, qh[nt][2 + u]));
                    }
            }
        }
        return;
    }

    // ---------------- chain warps ----------------
    float S[16][4];
    float* sp = state + ((size_t)h * DC + row0 + g) * DC + t4 * 2;
    auto load_state = [&]() {
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const float2 a = *reinterpret_cast<const float2*>(sp + j * 8);
            const float2 b = *reinterpret_cast<const float2*>(sp + 8 * DC + j * 8);
            S[j][0] = a.x; S[j][1] = a.y; S[j][2] = b.x; S[j][3] = b.y;
        }
    };
    auto store_state = [&]() {
#pragma unroll
        for (int j = 0; j < 16; j++) {
            *reinterpret_cast<float2*>(sp + j * 8) = make_float2(S[j][0], S[j][1]);
            *reinterpret_cast<float2*>(sp + 8 * DC + j * 8) = make_float2(S[j][2], S[j][3]);
        }
    };
    float s0, s1, inv0 = 0.0f, inv1 = 0.0f;
    auto leave_state = [&]() {                               // the operands of both warps' products with it
        dc_row_scales(S, s0, s1, inv0, inv1);
        sm.s_inv[w][lane] = make_float2(inv0, inv1);
#pragma unroll
        for (int kk = 0; kk < 8; kk++) {
            uint32_t hi[4], lo[4];
            dc_operand(S[2 * kk], S[2 * kk + 1], s0, s1, hi, lo);
            sm.s_hi[w][kk][lane] = dc_u4(hi);
            sm.s_lo[w][kk][lane] = dc_u4(lo);
        }
    };
    if (active) {
        load_state();
        leave_state();
    }
    for (int c = 0; c < nblk; c++) {
        __syncthreads();
        if (!active) continue;
        const typename DcScanSmem<W>::Stage& s = sm.stage[c & 1];
        const DcHead& hd = *reinterpret_cast<const DcHead*>(s.head);
        // ---- S k, raw; R = beta (v - G S k) ----
        float r[8][4], rl[8][4];
        dc_zero(r);
        dc_zero(rl);
#pragma unroll
        for (int kk = 0; kk < 8; kk++) {
            uint32_t hi[4], lo[4];
            dc_from(sm.s_hi[w][kk][lane], hi);
            dc_from(sm.s_lo[w][kk][lane], lo);
#pragma unroll
            for (int p = 0; p < 4; p++) {
                uint32_t b[4];
                dc_ldsm(b, &s.kq.k[p * 16 + lr][kk * 16 + lc]);
                dc_mma(r[2 * p], hi, b[0], b[1]);
                dc_mma(r[2 * p + 1], hi, b[2], b[3]);
                dc_mma(rl[2 * p], lo, b[0], b[1]);
                dc_mma(rl[2 * p + 1], lo, b[2], b[3]);
            }
        }
#pragma unroll
        for (int p = 0; p < 4; p++) {
            uint32_t v[4];
            dc_ldsm_t(v, &s.v[p * 16 + lr][w * 16 + lc]);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int nt = 2 * p + u;
                const float2 v0 = __half22float2(*reinterpret_cast<const __half2*>(&v[2 * u]));
                const float2 v1 = __half22float2(*reinterpret_cast<const __half2*>(&v[2 * u + 1]));
                const float2 ks = *reinterpret_cast<const float2*>(&hd.ksc[nt * 8 + t4 * 2]);
                const float2 bt = *reinterpret_cast<const float2*>(&hd.beta[nt * 8 + t4 * 2]);
                r[nt][0] = fmaf(-fmaf(rl[nt][0], DC_LO_INV, r[nt][0]) * inv0, ks.x, v0.x) * bt.x;
                r[nt][1] = fmaf(-fmaf(rl[nt][1], DC_LO_INV, r[nt][1]) * inv0, ks.y, v0.y) * bt.y;
                r[nt][2] = fmaf(-fmaf(rl[nt][2], DC_LO_INV, r[nt][2]) * inv1, ks.x, v1.x) * bt.x;
                r[nt][3] = fmaf(-fmaf(rl[nt][3], DC_LO_INV, r[nt][3]) * inv1, ks.y, v1.y) * bt.y;
            }
        }
        // ---- delta = X R ----
        float i0, i1, dh[8][4], dl[8][4];
        dc_row_scales(r, s0, s1, i0, i1);
        dc_zero(dh);
        dc_zero(dl);
#pragma unroll
        for (int m = 0; m < 4; m++) {
            uint32_t hi[4], lo[4];
            dc_operand(r[2 * m], r[2 * m + 1], s0, s1, hi, lo);
            dc_triangle(dh, dl, hi, lo, m, hd.x_hi, hd.x_lo, lr, lc);
        }
        float bad = 0.0f;
#pragma unroll
        for (int nt = 0; nt < 8; nt++) {
            const float2 xi = *reinterpret_cast<const float2*>(&hd.x_inv[nt * 8 + t4 * 2]);
            dh[nt][0] = fmaf(fmaf(dl[nt][0], DC_LO_INV, dh[nt][0]) * i0, xi.x, r[nt][0]);
            dh[nt][1] = fmaf(fmaf(dl[nt][1], DC_LO_INV, dh[nt][1]) * i0, xi.y, r[nt][1]);
            dh[nt][2] = fmaf(fmaf(dl[nt][2], DC_LO_INV, dh[nt][2]) * i1, xi.x, r[nt][2]);
            dh[nt][3] = fmaf(fmaf(dl[nt][3], DC_LO_INV, dh[nt][3]) * i1, xi.y, r[nt][3]);
#pragma unroll
            for (int e = 0; e < 4; e++) bad = fmaf(dh[nt][e], 0.0f, bad);       // NaN if one of them is not finite
        }
        const bool plain = __any_sync(0xffffffffu, bad != 0.0f);                // (NaN != 0)
        if (!plain) {
#pragma unroll
            for (int nt = 0; nt < 8; nt++) sm.delta[w][nt][lane] = make_float4(dh[nt][0], dh[nt][1], dh[nt][2], dh[nt][3]);
        }
        if (lane == 0) sm.plain[w] = plain;
        dc_pair_sync(1 + w);
        if (plain) {
            // the block again, token by token, from the state that enters it
            store_state();
            __syncwarp();
            dn_chunk_plain(state + ((size_t)h * DC + row0) * DC, hp + c, kqp + c, vbase + (size_t)c * CH * conv_dim + row0,
                           conv_dim, o_out + ((size_t)c * CH * nv + h) * DC + row0, nv * DC, min(CH, n - c * CH), lane);
            __syncwarp();
            load_state();
        } else {
            // ---- S <- G_63 S + sum_i P(i+1..63) delta_i k_i^T ----
            {
                float u[8][4];
#pragma unroll
                for (int nt = 0; nt < 8; nt++) {
                    const float2 us = *reinterpret_cast<const float2*>(&hd.usc[nt * 8 + t4 * 2]);
                    u[nt][0] = dh[nt][0] * us.x; u[nt][1] = dh[nt][1] * us.y;
                    u[nt][2] = dh[nt][2] * us.x; u[nt][3] = dh[nt][3] * us.y;
                }
                dc_row_scales(u, s0, s1, i0, i1);
            }
            uint32_t hi[4][4], lo[4][4], rest[4][4];
#pragma unroll
            for (int m = 0; m < 4; m++)
#pragma unroll
                for (int e = 0; e < 4; e++) {        // (dc_operand's order)
                    const int nt = 2 * m + (e >> 1);
                    dc_split3(dh[nt][(e & 1) * 2], dh[nt][(e & 1) * 2 + 1],
                              *reinterpret_cast<const float2*>(&hd.usc[nt * 8 + t4 * 2]),
                              *reinterpret_cast<const float2*>(&hd.usl[nt * 8 + t4 * 2]), (e & 1) ? s1 : s0, hi[m][e],
                              lo[m][e], rest[m][e]);
                }
            const float gl = hd.glast[0];
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                float uh[4][4], ul[4][4];
                dc_zero(uh);
                dc_zero(ul);
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    uint32_t b0[4], b1[4];
                    dc_ldsm_t(b0, &s.kq.k[m * 16 + tr][jj * 32 + tc]);
                    dc_ldsm_t(b1, &s.kq.k[m * 16 + tr][jj * 32 + 16 + tc]);
                    dc_mma(uh[0], hi[m], b0[0], b0[1]);
                    dc_mma(uh[1], hi[m], b0[2], b0[3]);
                    dc_mma(uh[2], hi[m], b1[0], b1[1]);
                    dc_mma(uh[3], hi[m], b1[2], b1[3]);
                    dc_mma(ul[0], lo[m], b0[0], b0[1]);
                    dc_mma(ul[1], lo[m], b0[2], b0[3]);
                    dc_mma(ul[2], lo[m], b1[0], b1[1]);
                    dc_mma(ul[3], lo[m], b1[2], b1[3]);
                    dc_mma(ul[0], rest[m], b0[0], b0[1]);
                    dc_mma(ul[1], rest[m], b0[2], b0[3]);
                    dc_mma(ul[2], rest[m], b1[0], b1[1]);
                    dc_mma(ul[3], rest[m], b1[2], b1[3]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int j = jj * 4 + i;
                    S[j][0] = fmaf(S[j][0], gl, fmaf(ul[i][0], DC_LO_INV, uh[i][0]) * i0);
                    S[j][1] = fmaf(S[j][1], gl, fmaf(ul[i][1], DC_LO_INV, uh[i][1]) * i0);
                    S[j][2] = fmaf(S[j][2], gl, fmaf(ul[i][2], DC_LO_INV, uh[i][2]) * i1);
                    S[j][3] = fmaf(S[j][3], gl, fmaf(ul[i][3], DC_LO_INV, uh[i][3]) * i1);
                }
            }
        }
        if (c + 1 < nblk) leave_state();
    }
    if (active) store_state();
}

// us of a layer, four tokens at a time / blocks of 64 (conv, gated norm and launches included):
//   64 value heads: 64 tokens 31.6 / 29.6, 72: 34.8 / 37.4, 512: 178 / 90     56: 64 tokens 31.4 / 29.3, 80: 36.7 / 37.2
//   48: 100 tokens 37.4 / 37.3, 128: 45.5 / 38.2, 512: 142 / 76, 1024: 279 / 146       40: 100 tokens 36.0 / 36.9, 112: 38.9 / 36.6
//   24: 160 tokens 43.7 / 44.4, 176: 46.4 / 45.0, 512: 109 / 69               20: 160 tokens 42.5 / 40.5
//   18: 256 tokens 47.5 / 51.0    12: 256 tokens 48.5 / 49.7, 288: 52.7 / 54.5, 320: 56.9 / 54.5, 512: 83 / 70
//   1: 256 tokens 44.4 / 36.5
// The one takes a time per token, more with more heads; the other one per block, the last block's empty places included.
// Both lines in ns, as fitted to the above; chunks shorter than those were not tried.
bool dn_chunk_takes(int n, int nv) {
    if (n < (nv < 20 ? 256 : 64)) return false;
    const int blocks = (n + CH - 1) / CH;
    const long long four = 10500 + (long long)n * (nv < 20 ? 140 : 130 + 3LL * nv);
    const long long b64 = nv >= 56   ? 22000 + 7500LL * blocks
                          : nv >= 40 ? 25000 + 6300LL * blocks
                          : nv >= 20 ? 25500 + 1000LL * (nv < 24 ? nv - 20 : 4) + 5000LL * blocks
                                     : 17000 + 1000LL * (nv < 13 ? nv : 13) + 5000LL * blocks;
    return b64 < four;
}

long long dn_chunk_work_bytes(int n, int nk, int nv) {
    const long long nblk = (n + CH - 1) / CH;
    return (nblk * (nk * (long long)sizeof(DcKQ) + nv * (long long)sizeof(DcHead)) + 255) & ~255LL;
}

template <int W>
static cudaError_t launch_scan(const DcKQ* kq, const DcHead* heads, const __half* conv_out, int conv_dim, float* state,
                               __half* o_out, int n, int nk, int nv, cudaStream_t st) {
    constexpr int SMEM = (int)sizeof(DcScanSmem<W>);
    static_assert(SMEM <= 227 * 1024, "shared memory");
    static bool opted[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index();
    if (!opted[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(dn_chunk_scan_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return e;
        opted[dev] = true;
    }
    constexpr int PER_HEAD = (DC / 16 + W - 1) / W;
    return launch_pdl(dn_chunk_scan_kernel<W>, dim3(nv * PER_HEAD), dim3(W * 64), SMEM, st, kq, heads, conv_out, conv_dim,
                      state, o_out, nk, nv, n);
}

cudaError_t dn_chunk_launch(const __half* conv_out, int conv_dim, const __half* x, long long ld, const __half* A_log,
                            const __half* dt_bias, float* state, void* work, __half* o_out, int n, int nk, int nv,
                            cudaStream_t st) {
    static bool opted[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index(), sms = device_sms(dev);
    if (!opted[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(dn_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)sizeof(DcPrepSmem));
        if (e != cudaSuccess) return e;
        opted[dev] = true;
    }
    const int nblk = (n + CH - 1) / CH;
    DcKQ* kq = static_cast<DcKQ*>(work);
    DcHead* heads = reinterpret_cast<DcHead*>(kq + (size_t)nk * nblk);
    cudaError_t e = launch_pdl(dn_chunk_prep_kernel, dim3(nv, nblk), dim3(256), sizeof(DcPrepSmem), st, conv_out, conv_dim,
                               x, ld, A_log, dt_bias, kq, heads, nk, nv, n);
    if (e != cudaSuccess) return e;
    // a CTA fills an SM's shared memory: as few pairs of warps in it as leave every CTA an SM
    const DcHead* hd = heads;
    const DcKQ* kp = kq;
    if (nv * 8 <= sms) return launch_scan<1>(kp, hd, conv_out, conv_dim, state, o_out, n, nk, nv, st);
    if (nv * 4 <= sms) return launch_scan<2>(kp, hd, conv_out, conv_dim, state, o_out, n, nk, nv, st);
    if (nv * 3 <= sms) return launch_scan<3>(kp, hd, conv_out, conv_dim, state, o_out, n, nk, nv, st);
    return launch_scan<4>(kp, hd, conv_out, conv_dim, state, o_out, n, nk, nv, st);
}

}  // namespace nvfp4
