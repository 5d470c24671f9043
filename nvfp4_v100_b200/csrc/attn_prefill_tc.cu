// Causal attention of a prefill chunk on the tensor cores (head dim 256, grouped query heads).
//
// attn_prefill_group_kernel (fused_ops.cu) keeps the decode kernel's arithmetic: a warp forms one
// score at a time with a shuffle reduction, so a chunk costs about 30 instructions per (query, key)
// pair and lane and the scores of four queries in shared memory.  Here both products are matrix
// products on tcgen05, the scores stay in tensor memory and the softmax is the running form.
//
// One CTA (384 threads) = the query heads of one KV head x as many tokens as fit in 128 rows (row =
// token * heads + head: every K and V tile is read once for all heads that share it), 128 keys a step:
//   warp 0       TMA producer: Q once (four boxes of 64 dims), then a ring of four 32 KB pieces in the
//                order of use: K(0), K(1), V(0), K(2), V(1), ... (a K piece = 128 keys x 128 dims, a
//                V piece = 64 keys x 256 dims)
//   warp 1       MMA issuer: S(i+1) = Q . K(i+1)^T (M 128, N 128) while the softmax of S(i) runs, then
//                O += P(i) . V(i) (M 128, N 256, P from tensor memory)
//   warps 4..11  softmax: a thread owns 64 of the 128 scores of its row
// Tensor memory: two S/P buffers of 128 columns and the 256 columns of O.  P takes the place of its
// own scores and is carried as p = hi + lo, two fp16 numbers whose sum is within 2^-23 of p's power of two
// (the kernel before held it in fp32: 2^-24) and, p being scaled by 2^12, within 2^-37 for small weights;
// O accumulates hi . V and lo . V.
// O is rescaled only when a row's maximum has grown by more than 2 since the last time (so p stays
// below 2^15); otherwise the old reference point stays and nothing waits on the MMAs.
// Few tokens leave SMs idle: then the keys are split over the CTAs of a cluster, whose (max, sum, O)
// meet in distributed shared memory.
// A row whose result is not finite is recomputed with plain fp32 arithmetic by the warp that was
// about to write it: a masked weight is an exact zero, but zero times an infinite or NaN value of
// a later token is not, and hi . inf + lo . inf need not be inf.
// Every wait is bounded and reported through nvfp4_gemm_status.
//
// Measured, 24 query / 4 KV heads, us (in brackets attn_prefill_group_kernel), tokens after context:
//   512 after 0      27.7 (395)     512 after 3488  127 (3598)     26 after 511   16.4 (59.3)
//   512 after 512    40.8 (859)     512 after 9000  300 (8681)    100 after 0    18.0 (46.0)
// i.e. some 20 us fixed and 28 us per 1024 keys of 512 tokens: 3072 cycles of MMAs per step and tile.
// Relative error against float64 as before (3.5e-4, the fp16 rounding of the output; see ATC_CHAIN).  Of the
// outputs 0.2 to 0.8 % are not the correctly rounded ones, against 0.1 % before.
#include <cuda.h>

#include "attn_prefill_tc.cuh"
#include "common.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nvfp4 {

constexpr int ATC_THREADS = 384;
constexpr int ATC_D = 256;
constexpr int ATC_ROWS = 128;                       // query rows of a CTA
constexpr int ATC_KEYS = 128;                       // keys of a step
constexpr int ATC_SLOTS = 4;                        // ring pieces
constexpr int ATC_PIECE = 32768;
constexpr int ATC_Q_GROUP = ATC_ROWS * 128;         // bytes of 64 dims of all rows
constexpr int ATC_SMEM = 4 * ATC_Q_GROUP + ATC_SLOTS * ATC_PIECE + 1024;
constexpr int ATC_LD = ATC_D + 4;                   // floats per row of the output tile in shared memory
constexpr int ATC_MAX_SPLIT = 8;
// Key steps of one CTA's accumulation.  An MMA truncates the fp32 sum that it adds to (a bias towards
// zero, twice per 16 keys), where the kernel before rounded to nearest: with all 32 steps of 4000 keys in
// one CTA the outputs' relative error against float64 was 3.1e-4 of itself above that kernel's (24 seeds,
// standard error 4e-5), with 16 steps 9e-5, with 8 steps 2e-5, which is none.  The partial results of a
// cluster are added by ordinary fp32 instructions.
constexpr int ATC_CHAIN = 8;
constexpr float ATC_P_SCALE = 4096.0f;
constexpr float ATC_RESCALE = 2.0f;                 // e^2 * 4096 < 65504
constexpr float ATC_NO_MAX = -3.4e38f;
constexpr uint32_t ATC_SPIN_LIMIT = 100000;
static_assert(ATC_ROWS * ATC_LD * 4 <= ATC_SMEM - 1024, "the output tile takes the place of Q and the ring");

__device__ int g_atc_status = 0;

// Bounded wait (about 2 s), parked by the hardware.  One that runs out is noted for the host and the CTA.
__device__ __forceinline__ bool atc_wait(uint32_t bar, uint32_t parity, int id, volatile int& ran_out) {
    for (uint32_t i = 0; i < ATC_SPIN_LIMIT; i++)
        if (mbar_try_wait_hint(bar, parity, 20000)) return true;
    atomicExch(&g_atc_status, 1 + id);
    ran_out = 1;
    return false;
}
__device__ __forceinline__ float atc_ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 atc_ld_cluster4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}
__device__ __forceinline__ void atc_unpack8(const uint4 u, float (&f)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
        f[2 * j] = v.x;
        f[2 * j + 1] = v.y;
    }
}

// One query row by one warp in fp32, the chain of attn_one_query: only keys below L are read.
__device__ __noinline__ void atc_row_plain(const __half* q, const __half* kbase, const __half* vbase, int L,
                                           float scale, const __half* gate, __half* out) {
    const int lane = threadIdx.x & 31;
    float qf[8];
    atc_unpack8(*reinterpret_cast<const uint4*>(q + lane * 8), qf);
    auto score = [&](int i) {
        float kf[8], acc = 0.0f;
        atc_unpack8(*reinterpret_cast<const uint4*>(kbase + (size_t)i * ATC_D + lane * 8), kf);
#pragma unroll
        for (int j = 0; j < 8; j++) acc = fmaf(qf[j], kf[j], acc);
        return warp_sum(acc) * scale;
    };
    float m = ATC_NO_MAX, l = 0.0f, o[8];
    for (int i = 0; i < L; i++) m = fmaxf(m, score(i));
    for (int i = 0; i < L; i++) l += expf(score(i) - m);
    const float inv = 1.0f / l;
#pragma unroll
    for (int j = 0; j < 8; j++) o[j] = 0.0f;
    for (int i = 0; i < L; i++) {
        const float p = expf(score(i) - m) * inv;
        float vf[8];
        atc_unpack8(*reinterpret_cast<const uint4*>(vbase + (size_t)i * ATC_D + lane * 8), vf);
#pragma unroll
        for (int j = 0; j < 8; j++) o[j] = fmaf(p, vf[j], o[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float sg = round_f16(1.0f / (1.0f + expf(-__half2float(gate[lane * 8 + j]))));
        out[lane * 8 + j] = __float2half(round_f16(o[j]) * sg);
    }
}

__global__ void __launch_bounds__(ATC_THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                       const __grid_constant__ CUtensorMap v_map, const __half* q, const __half* keys,
                       const __half* values, int len0, int n_tokens, const __half* gate, __half* out,
                       int max_len, int hq, int gqa, float scale, int split) {
    extern __shared__ __align__(1024) uint8_t atc_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(atc_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_ring = smem + 4 * ATC_Q_GROUP;
    __shared__ __align__(8) uint64_t bar_q;
    __shared__ __align__(8) uint64_t bar_full[ATC_SLOTS];    // piece landed
    __shared__ __align__(8) uint64_t bar_empty[ATC_SLOTS];   // its MMAs retired
    __shared__ __align__(8) uint64_t bar_s[2];               // scores of a step ready
    __shared__ __align__(8) uint64_t bar_p[2];               // weights of a step ready
    __shared__ __align__(8) uint64_t bar_o[2];               // O holds a step
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_ran_out;                       // a wait of this CTA has
    __shared__ int s_next[2];                                // the ring slot after the last piece, and its lap
    __shared__ float s_mx[2][2][ATC_ROWS];                   // step parity, key half, row
    __shared__ float s_m[ATC_ROWS], s_l[2][ATC_ROWS];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % split;                // = rank in the cluster
    const int tiles = (int)gridDim.x / split;
    const int bt = ATC_ROWS / gqa;                           // tokens of a CTA
    const int t0 = (tiles - 1 - (int)blockIdx.x / split) * bt;   // the longest rows are started first
    const int kv = blockIdx.y;
    const int l_max = len0 + min(t0 + bt, n_tokens) - 1;     // keys the last token sees
    const int steps_all = (l_max + ATC_KEYS - 1) / ATC_KEYS;
    const int step0 = steps_all * rank / split, steps = steps_all * (rank + 1) / split - step0;

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&q_map) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&k_map) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&v_map) : "memory");
        mbar_init(smem_u32(&bar_q), 1);
        for (int s = 0; s < ATC_SLOTS; s++) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&bar_s[b]), 1);
            mbar_init(smem_u32(&bar_p[b]), 8);
            mbar_init(smem_u32(&bar_o[b]), 1);
        }
        s_ran_out = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tcgen05_alloc(smem_u32(&s_tmem), 512);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = s_tmem, tmem_o = tmem + 256;
    // only now: a CTA of the next kernel must not take tensor memory before this one has all of it
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    PDL_FRESH(q); PDL_FRESH(keys); PDL_FRESH(values); PDL_FRESH(gate); PDL_FRESH(out);

    if (warp == 0) {
        if (lane == 0 && steps > 0) {
            mbar_arrive_expect_tx(smem_u32(&bar_q), (uint32_t)(4 * gqa * bt * 128));
            for (int g = 0; g < 4; g++)
                tma_load_3d(smem_u32(smem + g * ATC_Q_GROUP), &q_map, g * 64, kv * gqa, t0, smem_u32(&bar_q));
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            auto slot = [&]() {                              // the next free piece of the ring
                if (ok) ok = atc_wait(smem_u32(&bar_empty[s]), ph ^ 1u, 0, s_ran_out);
                return ok;
            };
            auto next = [&]() { if (++s == ATC_SLOTS) { s = 0; ph ^= 1u; } };
            auto load_k = [&](int i) {
                for (int h = 0; h < 2 && slot(); h++) {
                    const uint32_t bar = smem_u32(&bar_full[s]), dst = smem_u32(smem_ring + s * ATC_PIECE);
                    mbar_arrive_expect_tx(bar, ATC_PIECE);
                    for (int g = 0; g < 2; g++)
                        tma_load_3d(dst + g * 16384, &k_map, (2 * h + g) * 64, (step0 + i) * ATC_KEYS, kv, bar);
                    next();
                }
            };
            auto load_v = [&](int i) {
                for (int h = 0; h < 2 && slot(); h++) {
                    const uint32_t bar = smem_u32(&bar_full[s]), dst = smem_u32(smem_ring + s * ATC_PIECE);
                    mbar_arrive_expect_tx(bar, ATC_PIECE);
                    for (int g = 0; g < 4; g++)
                        tma_load_3d(dst + g * 8192, &v_map, g * 64, (step0 + i) * ATC_KEYS + h * 64, kv, bar);
                    next();
                }
            };
            load_k(0);
            for (int i = 0; i < steps && ok; i++) {
                if (i + 1 < steps) load_k(i + 1);
                load_v(i);
            }
            s_next[0] = s;
            s_next[1] = (int)ph;
        }
    } else if (warp == 1) {
        if (steps > 0) {
            // D fp32, A and B fp16, M = 128; S: B K-major, N = 128; O: B MN-major, N = 256
            const uint32_t idesc_s = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
            const uint32_t idesc_o = (1u << 4) | (1u << 16) | ((256u >> 3) << 17) | ((128u >> 4) << 24);
            int s = 0;
            uint32_t ph = 0;
            bool ok = atc_wait(smem_u32(&bar_q), 0, 1, s_ran_out);
            auto piece = [&]() {
                if (ok) ok = atc_wait(smem_u32(&bar_full[s]), ph, 2, s_ran_out);
                tcgen05_fence_after();
            };
            auto done = [&]() {
                tcgen05_commit(smem_u32(&bar_empty[s]));
                if (++s == ATC_SLOTS) { s = 0; ph ^= 1u; }
            };
            auto scores = [&](int i) {
                const uint32_t d = tmem + (uint32_t)((i & 1) * 128);
                for (int h = 0; h < 2; h++) {
                    piece();
                    const uint32_t a = smem_u32(smem + 2 * h * ATC_Q_GROUP), b = smem_u32(smem_ring + s * ATC_PIECE);
#pragma unroll
                    for (int kk = 0; kk < 8; kk++)           // 128 dims, 16 at a time
                        tcgen05_mma_f16(d, make_desc_sw128(a + (kk >> 2) * ATC_Q_GROUP + (kk & 3) * 32, 16, 1024),
                                        make_desc_sw128(b + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024), idesc_s,
                                        (h | kk) != 0 ? 1u : 0u);
                    done();
                }
                tcgen05_commit(smem_u32(&bar_s[i & 1]));
            };
            scores(0);
            for (int i = 0; i < steps; i++) {
                if (i + 1 < steps) scores(i + 1);
                if (ok) ok = atc_wait(smem_u32(&bar_p[i & 1]), (uint32_t)(i >> 1) & 1u, 3, s_ran_out);
                tcgen05_fence_after();
                for (int h = 0; h < 2; h++) {
                    piece();
                    const uint32_t a = tmem + (uint32_t)((i & 1) * 128 + h * 64), b = smem_u32(smem_ring + s * ATC_PIECE);
#pragma unroll
                    for (int kk = 0; kk < 8; kk++)           // four 16-key steps of hi, then of lo
                        tcgen05_mma_f16_ta(tmem_o, a + (uint32_t)(kk * 8),
                                           make_desc_sw128(b + (kk & 3) * 2048, 8192, 1024), idesc_o,
                                           (i | h | kk) != 0 ? 1u : 0u);
                    done();
                }
                tcgen05_commit(smem_u32(&bar_o[i & 1]));
            }
        }
    } else if (warp >= 4) {
        const int qd = warp & 3, half = (warp - 4) >> 2;     // lane quarter, half of the keys
        const uint32_t lane_base = (uint32_t)(qd * 32) << 16;
        const int r = qd * 32 + lane;
        const int tok = t0 + r / gqa;
        const int L = (r < bt * gqa && tok < n_tokens) ? len0 + tok : 0;
        float m = ATC_NO_MAX, l = 0.0f;
        bool ok = true;
        for (int i = 0; i < steps; i++) {
            const int b = i & 1;
            if (ok) ok = atc_wait(smem_u32(&bar_s[b]), (uint32_t)(i >> 1) & 1u, 4, s_ran_out);
            __syncwarp();                                    // the accesses below are .aligned
            tcgen05_fence_after();
            const uint32_t at = tmem + lane_base + (uint32_t)(b * 128 + half * 64);
            uint32_t sv[2][32];
            tcgen05_ld_32x32b_x32(at, sv[0]);
            tcgen05_ld_32x32b_x32(at + 32, sv[1]);
            tcgen05_wait_ld();
            const int seen = L - ((step0 + i) * ATC_KEYS + half * 64);   // keys of this half the row sees
            float mt = ATC_NO_MAX;
            if (__all_sync(0xffffffffu, seen >= 64)) {
#pragma unroll
                for (int j = 0; j < 64; j++) {
                    const float x = __uint_as_float(sv[j >> 5][j & 31]) * scale;
                    sv[j >> 5][j & 31] = __float_as_uint(x);
                    mt = fmaxf(mt, x);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 64; j++) {
                    const float x = (j < seen) ? __uint_as_float(sv[j >> 5][j & 31]) * scale : -INFINITY;
                    sv[j >> 5][j & 31] = __float_as_uint(x);
                    mt = fmaxf(mt, x);
                }
            }
            // the row's other half belongs to the warp that shares this quarter
            s_mx[b][half][r] = mt;
            asm volatile("bar.sync %0, 64;\n" ::"r"(1 + qd) : "memory");
            mt = fmaxf(mt, s_mx[b][half ^ 1][r]);
            if (i == 0) {
                m = mt;
            } else if (__any_sync(0xffffffffu, mt > m + ATC_RESCALE)) {      // the same in both warps
                const float f = (mt > m + ATC_RESCALE) ? expf(m - mt) : 1.0f;
                if (mt > m + ATC_RESCALE) m = mt;
                l *= f;
                if (ok) ok = atc_wait(smem_u32(&bar_o[b ^ 1]), (uint32_t)((i - 1) >> 1) & 1u, 5, s_ran_out);
                __syncwarp();
                tcgen05_fence_after();
#pragma unroll 1
                for (int c = 0; c < 128; c += 16) {
                    const uint32_t oc = tmem_o + lane_base + (uint32_t)(half * 128 + c);
                    uint32_t v[16];
                    tcgen05_ld_32x32b_x16(oc, v);
                    tcgen05_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) * f);
                    tcgen05_st_32x32b_x16(oc, v);
                }
            }
#pragma unroll
            for (int c = 0; c < 2; c++) {                    // 32 keys: 16 columns of hi, 16 of lo
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float p0 = expf(__uint_as_float(sv[c][2 * j]) - m);
                    const float p1 = expf(__uint_as_float(sv[c][2 * j + 1]) - m);
                    l += p0;
                    l += p1;
                    const float a0 = p0 * ATC_P_SCALE, a1 = p1 * ATC_P_SCALE;
                    const __half2 h = __floats2half2_rn(a0, a1);
                    const float2 back = __half22float2(h);
                    const __half2 e = __floats2half2_rn(a0 - back.x, a1 - back.y);
                    hi[j] = *reinterpret_cast<const uint32_t*>(&h);
                    lo[j] = *reinterpret_cast<const uint32_t*>(&e);
                }
                tcgen05_st_32x32b_x16(at + (uint32_t)(c * 16), hi);
                tcgen05_st_32x32b_x16(at + (uint32_t)(32 + c * 16), lo);
            }
            tcgen05_wait_st();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_p[b]));
        }
        if (half == 0) s_m[r] = m;
        s_l[half][r] = l;
        // O -> shared memory (Q and the ring are idle: the last MMA has retired, every copy was consumed)
        float* tile = reinterpret_cast<float*>(smem);
        if (steps > 0) {
            atc_wait(smem_u32(&bar_o[(steps - 1) & 1]), (uint32_t)((steps - 1) >> 1) & 1u, 6, s_ran_out);
            __syncwarp();
            tcgen05_fence_after();
        }
#pragma unroll
        for (int c = 0; c < 128; c += 32) {
            uint32_t v[32];
            if (steps > 0) {
                tcgen05_ld_32x32b_x32(tmem_o + lane_base + (uint32_t)(half * 128 + c), v);
                tcgen05_wait_ld();
            } else {
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<uint4*>(&tile[r * ATC_LD + half * 128 + c + j]) =
                    make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    // No copy may be in flight when the CTA leaves.  Where no wait has run out, all have been consumed by now
    // (waiting for them all the same costs 0.6 to 1 us); a slot that was never filled answers at once.
    if (threadIdx.x == 0 && s_ran_out) {
        if (steps > 0) atc_wait(smem_u32(&bar_q), 0, 7, s_ran_out);
        for (int j = 0; j < ATC_SLOTS && steps > 0; j++)
            atc_wait(smem_u32(&bar_full[j]), (uint32_t)s_next[1] ^ (j < s_next[0] ? 0u : 1u), 7, s_ran_out);
    }
    if (split > 1) cluster_sync_all();

    // ---- weighted sum over the cluster, gate, output: a warp takes a row, a lane 4 + 4 dims ----
    // The gates of OUT_ROWS rows are requested together: with one row at a time a warp waited for
    // memory eleven times in a row (64 tokens 21.4 -> 17.6 us, 512 tokens 30.9 -> 27.1).
    constexpr int OUT_ROWS = 4;
    const int stride = split * (ATC_THREADS / 32);
    for (int r0 = rank + split * warp; r0 < bt * gqa; r0 += OUT_ROWS * stride) {
        uint2 gw[OUT_ROWS][2];
#pragma unroll
        for (int u = 0; u < OUT_ROWS; u++) {
            const int r = r0 + u * stride, tok = t0 + r / gqa;
            const bool row = r < bt * gqa && tok < n_tokens;
            const size_t at = ((size_t)tok * hq + kv * gqa + r % gqa) * ATC_D;
#pragma unroll
            for (int g = 0; g < 2; g++)
                gw[u][g] = row ? *reinterpret_cast<const uint2*>(gate + at + g * 128 + lane * 4) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < OUT_ROWS; u++) {
            const int r = r0 + u * stride, tok = t0 + r / gqa, h = kv * gqa + r % gqa;
            if (r >= bt * gqa || tok >= n_tokens) continue;
            float o[8], l;
            if (split == 1) {
                const float* t = reinterpret_cast<const float*>(smem) + r * ATC_LD + lane * 4;
                const float4 x = *reinterpret_cast<const float4*>(t), y = *reinterpret_cast<const float4*>(t + 128);
                o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w;
                o[4] = y.x; o[5] = y.y; o[6] = y.z; o[7] = y.w;
                l = s_l[0][r] + s_l[1][r];
            } else {
                const uint32_t am = smem_u32(&s_m[r]), al = smem_u32(&s_l[0][r]), ah = smem_u32(&s_l[1][r]);
                const uint32_t ao = smem_u32(smem) + (uint32_t)(r * ATC_LD + lane * 4) * 4u;
                float mc[ATC_MAX_SPLIT], mm = ATC_NO_MAX;
#pragma unroll
                for (int c = 0; c < ATC_MAX_SPLIT; c++) {
                    mc[c] = c < split ? atc_ld_cluster(cluster_map_shared(am, (uint32_t)c)) : ATC_NO_MAX;
                    mm = fmaxf(mm, mc[c]);
                }
                l = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; j++) o[j] = 0.0f;
#pragma unroll
                for (int c = 0; c < ATC_MAX_SPLIT; c++)
                    if (c < split) {
                        const float w = expf(mc[c] - mm);
                        l = fmaf(w, atc_ld_cluster(cluster_map_shared(al, (uint32_t)c)) +
                                        atc_ld_cluster(cluster_map_shared(ah, (uint32_t)c)), l);
                        const float4 x = atc_ld_cluster4(cluster_map_shared(ao, (uint32_t)c));
                        const float4 y = atc_ld_cluster4(cluster_map_shared(ao + 512u, (uint32_t)c));
                        o[0] = fmaf(w, x.x, o[0]); o[1] = fmaf(w, x.y, o[1]);
                        o[2] = fmaf(w, x.z, o[2]); o[3] = fmaf(w, x.w, o[3]);
                        o[4] = fmaf(w, y.x, o[4]); o[5] = fmaf(w, y.y, o[5]);
                        o[6] = fmaf(w, y.z, o[6]); o[7] = fmaf(w, y.w, o[7]);
                    }
            }
            const float inv = 1.0f / l;
            bool finite = true;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                o[j] = o[j] * (1.0f / ATC_P_SCALE) * inv;
                finite = finite && (fabsf(o[j]) <= 3.4e38f);
            }
            const size_t at = ((size_t)tok * hq + h) * ATC_D;
            if (!__all_sync(0xffffffffu, finite)) {
                const size_t base = (size_t)kv * (size_t)max_len * ATC_D;
                atc_row_plain(q + at, keys + base, values + base, len0 + tok, scale, gate + at, out + at);
                continue;
            }
#pragma unroll
            for (int g = 0; g < 2; g++) {
                const float2 g0 = __half22float2(*reinterpret_cast<const __half2*>(&gw[u][g].x));
                const float2 g1 = __half22float2(*reinterpret_cast<const __half2*>(&gw[u][g].y));
                const float gt[4] = {g0.x, g0.y, g1.x, g1.y};
                float f[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    f[j] = round_f16(o[4 * g + j]) * round_f16(1.0f / (1.0f + expf(-gt[j])));
                const __half2 w0 = __floats2half2_rn(f[0], f[1]), w1 = __floats2half2_rn(f[2], f[3]);
                uint2 w;
                w.x = *reinterpret_cast<const uint32_t*>(&w0);
                w.y = *reinterpret_cast<const uint32_t*>(&w1);
                *reinterpret_cast<uint2*>(out + at + g * 128 + lane * 4) = w;
            }
        }
    }
    if (split > 1) cluster_sync_all();       // nobody leaves while a peer still reads its shared memory
    if (warp == 1) tcgen05_dealloc(tmem, 512);
}

static void atc_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&at)[2], dim3 grid, int split) {
    cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(ATC_THREADS);
    cfg.dynamicSmemBytes = ATC_SMEM;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)split;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
}

// How many clusters of `split` CTAs (one per SM) run at once; 0 if the driver does not say.
static int atc_clusters(int dev, int split) {
    static int cached[NVFP4_MAX_DEVICES][ATC_MAX_SPLIT + 1] = {};
    int& c = cached[dev][split];
    if (c == 0) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        atc_config(cfg, at, dim3((unsigned)split), split);
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, attn_prefill_tc_kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        c = n > 0 ? n : -1;
    }
    return c > 0 ? c : 0;
}

bool attn_prefill_tc_takes(const void* q, const void* keys, const void* values, const void* gate, const void* out,
                           int len0, int n_tokens, int hq, int hkv) {
    if (hq / hkv > ATC_ROWS) return false;
    if (((uintptr_t)q | (uintptr_t)keys | (uintptr_t)values | (uintptr_t)gate | (uintptr_t)out) & 15) return false;
    const int L = len0 + n_tokens - 1, gqa = hq / hkv;
    if ((long long)n_tokens * L < ATTN_TC_MIN_PAIRS) return false;
    // Few heads: while the other kernel's CTAs (a head's eight tokens) fit on half of the SMs they all run
    // at once and take a time that only the keys decide; this kernel's first 256 keys cost by its rows.  In
    // ns, measured for 1 to 32 heads, e.g. 64 tokens of 6 heads 9.7 us against 18.3, 32 of 12 heads after 98
    // 13.9 against 19.1, 24 of 24 heads after 150 15.6 against 19.2; 16 of 24 heads after 242 19.6 against 15.1.
    if (2LL * hq * ((n_tokens + 7) / 8) <= device_sms(current_device_index()))
        return 6700 + 48LL * L >= 9500 + 75 * gqa * min(n_tokens, ATC_ROWS / gqa);
    return true;
}

int attn_prefill_tc_launch(const __half* q, const __half* keys, const __half* values, int len0, int n_tokens,
                           const __half* gate, __half* out, int max_len, int hq, int hkv, float scale,
                           cudaStream_t st) {
    static bool opted[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index();
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return -3;
    if (!opted[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   ATC_SMEM);
        if (e != cudaSuccess) return (int)e;
        opted[dev] = true;
    }
    const int gqa = hq / hkv, bt = ATC_ROWS / gqa, lcap = len0 + n_tokens - 1;
    CUtensorMap qm, km, vm;
    const cuuint32_t estr[3] = {1, 1, 1};
    auto encode = [&](CUtensorMap& m, const __half* p, cuuint64_t d1, cuuint64_t d2, cuuint64_t s2, cuuint32_t b1,
                      cuuint32_t b2) {
        const cuuint64_t dims[3] = {ATC_D, d1, d2};
        const cuuint64_t strides[2] = {ATC_D * sizeof(__half), s2};
        const cuuint32_t box[3] = {64, b1, b2};
        return enc(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(p), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    const cuuint64_t head = (cuuint64_t)max_len * ATC_D * sizeof(__half);
    // rows past the chunk's last key read as zeros: whatever the cache holds there stays out
    if (!encode(qm, q, (cuuint64_t)hq, (cuuint64_t)n_tokens, (cuuint64_t)hq * ATC_D * sizeof(__half), (cuuint32_t)gqa,
                (cuuint32_t)bt) ||
        !encode(km, keys, (cuuint64_t)lcap, (cuuint64_t)hkv, head, ATC_KEYS, 1) ||
        !encode(vm, values, (cuuint64_t)lcap, (cuuint64_t)hkv, head, 64, 1))
        return -3;
    const int tiles = (n_tokens + bt - 1) / bt, steps = (lcap + ATC_KEYS - 1) / ATC_KEYS;
    // key split: the fewest steps per CTA among the splits whose clusters all run at once, and more where
    // the accumulation would get too long (512 tokens after 3488: 115 -> 125 us, after 2048 79 -> 95)
    int split = 1;
    for (int s = 2; s <= ATC_MAX_SPLIT && s <= steps; s++)
        if (tiles * hkv <= atc_clusters(dev, s) && (steps + s - 1) / s < (steps + split - 1) / split) split = s;
    split = max(split, min(ATC_MAX_SPLIT, (steps + ATC_CHAIN - 1) / ATC_CHAIN));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    atc_config(cfg, at, dim3((unsigned)(tiles * split), (unsigned)hkv), split);
    cfg.stream = st;
    return (int)cudaLaunchKernelEx(&cfg, attn_prefill_tc_kernel, qm, km, vm, q, keys, values, len0, n_tokens, gate,
                                   out, max_len, hq, gqa, scale, split);
}

int attn_prefill_tc_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_atc_status, sizeof(int)) != cudaSuccess) return -1;
    if (reset) {
        const int z = 0;
        cudaMemcpyToSymbol(g_atc_status, &z, sizeof(int));
    }
    return v;
}

}  // namespace nvfp4
