// What the tensor-core GEMVs share (gemv_tc.cu: one activation; gemv_tc2.cu: two): the stage, the block-scaled FP4 MMA and
// the exact base-4 digits of an fp16 activation.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace nvfp4 {

constexpr int TC_BM = 128;                      // weight rows of a tile
constexpr int TC_BK = 256;                      // K elements of a stage
constexpr int TC_A_BYTES = TC_BM * 128;         // packed weights of a stage
constexpr int TC_S_BYTES = TC_BM * 16;          // weight scale bytes of a stage

__device__ __forceinline__ void tc_mma(uint32_t taddr, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, e;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "@e tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n}\n" ::
            "r"(taddr), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
}
__device__ __forceinline__ void tc_st_x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
        "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
        "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ uint32_t tc_prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;\n" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// Digit planes of 8 consecutive activations (one 16-byte vector; lane o of a warp holds elements
// 8o .. 8o+7 of a 256-element stage) -> 16 words, one per plane row of the B tile, and the block's
// exponent byte.  All by bit operations on whole words: a transpose of the eight 32-bit fractions by nibbles puts
// two digits of every element into one word, and a digit with bits h, l is the E2M1 code (h, l & ~h, h & l).  (A table of
// codes per byte in shared memory took 32 scattered reads a lane, which the SM's other CTA waited for as well.)
// A block with a value that is not finite has no digits: its exponent byte is 255, a NaN scale, so that every sum it
// enters is NaN and the rows are formed by tc_plain_row instead.
__device__ __forceinline__ void tc_digit_planes(const uint4 xv, uint8_t* btile, uint8_t* lbytes, int lane) {
    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
    uint32_t hmax = 0;
#pragma unroll
    for (int w = 0; w < 4; w++) {
        hmax = max(hmax, xw[w] & 0x7FFFu);
        hmax = max(hmax, (xw[w] >> 16) & 0x7FFFu);
    }
    hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, 1));   // lanes 2b, 2b+1 share block b
    const uint32_t em = hmax >> 10;
    const uint32_t m11 = em ? ((hmax & 0x3FFu) | 0x400u) : (hmax & 0x3FFu);
    const int bits = 32 - __clz(m11);
    const int L = bits + (int)(em ? em : 1u) - 25;
    // the fraction |x| / 2^L: significand m (|x| = m 2^(e - 25), e at least 1) with the block's largest at bit 31
    const uint32_t left = em ? 21u : (uint32_t)min(32 - bits, 31);
    const int right = em ? (int)em : 1;
    uint32_t u[8], sgn = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t h = (xw[k >> 1] >> (16 * (k & 1))) & 0x7FFFu;
        const uint32_t e = max(h >> 10, 1u);
        u[k] = __funnelshift_rc((h + 1024u - e * 1024u) << left, 0u, (uint32_t)(right - (int)e));   // (32 and more: 0)
    }
#pragma unroll
    for (int w = 0; w < 4; w++) sgn |= (((xw[w] >> 12) & 0x8u) | ((xw[w] >> 24) & 0x80u)) << (8 * w);
    // nibbles of elements 2 i and 2 i + 1 side by side: byte k of ev[i] = their nibbles 2 k, of od[i] = 2 k + 1
    uint32_t ev[4], od[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t a = u[2 * i], c = u[2 * i + 1];
        ev[i] = (a & 0x0F0F0F0Fu) | ((c << 4) & 0xF0F0F0F0u);
        od[i] = ((a >> 4) & 0x0F0F0F0Fu) | (c & 0xF0F0F0F0u);
    }
    // 4 x 4 byte transposes: word n = nibble n of all eight elements
    auto transpose = [](const uint32_t (&v)[4], uint32_t (&o)[4]) {
        const uint32_t t0 = tc_prmt(v[0], v[1], 0x5140u), t1 = tc_prmt(v[2], v[3], 0x5140u);
        const uint32_t t2 = tc_prmt(v[0], v[1], 0x7362u), t3 = tc_prmt(v[2], v[3], 0x7362u);
        o[0] = tc_prmt(t0, t1, 0x5410u);
        o[1] = tc_prmt(t0, t1, 0x7632u);
        o[2] = tc_prmt(t2, t3, 0x5410u);
        o[3] = tc_prmt(t2, t3, 0x7632u);
    };
    uint32_t te[4], to[4];
    transpose(ev, te);
    transpose(od, to);
    auto put = [&](int row, uint32_t word) {
        const int chunk = (lane >> 2) ^ (row & 7);              // 128-byte swizzle
        *reinterpret_cast<uint32_t*>(btile + row * 128 + chunk * 16 + (lane & 3) * 4) = word | sgn;
    };
#pragma unroll
    for (int n = 0; n < 8; n++) {                              // nibble 7 - n: planes 2 n and 2 n + 1
        const uint32_t t = ((7 - n) & 1) ? to[(7 - n) >> 1] : te[(7 - n) >> 1];
        put(2 * n, ((t >> 1) & 0x44444444u) | ((t >> 1) & ~(t >> 2) & 0x22222222u) | ((t >> 3) & (t >> 2) & 0x11111111u));
        put(2 * n + 1, ((t << 1) & 0x44444444u) | ((t << 1) & ~t & 0x22222222u) | ((t >> 1) & t & 0x11111111u));
    }
    if ((lane & 1) == 0) lbytes[lane >> 1] = (uint8_t)(em == 31u ? 255 : L + 125);
}

// Whether a row has to be formed by tc_plain_row.  An infinity too: a digit column's part of a sum can overflow where the
// sum does not (scale bytes near 254).
__device__ __forceinline__ bool tc_not_finite(float sum) { return !(fabsf(sum) <= 3.402823466e38f); }
// A row's sum in plain fp32, block by block, as the register-streaming kernels form it: for sums that are not finite (an
// activation that is not; a scale byte of 255, which is infinity here and NaN to the tensor core).  load(k): the
// activations k .. k + 7.
template <typename LOAD>
__device__ __forceinline__ float tc_plain_row(const uint8_t* packed, const uint8_t* scales, const LOAD load, int row, int K) {
    const uint8_t* w = packed + (size_t)row * (K / 2);
    const uint8_t* sc = scales + (size_t)row * (K / 16);
    float sum = 0.0f;
#pragma unroll 1
    for (int b = 0; b < K / 16; b++) {
        const uint2 p = *reinterpret_cast<const uint2*>(w + b * 8);
        float acc = 0.0f;
#pragma unroll 1
        for (int half = 0; half < 2; half++) {
            uint32_t h[4];
            e2m1x8_to_half2x4(half ? p.y : p.x, h[0], h[1], h[2], h[3]);
            const uint4 xv = load(b * 16 + half * 8);
            const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
            for (int e = 0; e < 4; e++) {
                const float2 wf = __half22float2(*reinterpret_cast<const __half2*>(&h[e]));
                const float2 xf = __half22float2(*reinterpret_cast<const __half2*>(&xw[e]));
                acc = fmaf(wf.x, xf.x, acc);
                acc = fmaf(wf.y, xf.y, acc);
            }
        }
        sum = fmaf(acc, e8m0_to_f32(sc[b]), sum);
    }
    return sum;
}

}  // namespace nvfp4
