// W4A4 GEMM on the block-scaled FP4 tensor-core path:
//   out[M, ld_out] (fp16) = dequant(W)[M, K] . dequant(A)[n_tokens, K]^T
// Both operands stay in the container's format all the way into the tensor core: E2M1 nibbles, two
// per byte (low nibble = even element), one E8M0 scale byte per 16 elements along K
// (codec/nvfp4_codec.py:13-19 layout, :60-86 decode rule).  No fp16 copy of either operand is made;
// tcgen05.mma kind::mxf4nvf4 with 16-element scale blocks multiplies the nibbles, applies both block
// scales and accumulates in fp32 in tensor memory.  This is the FP4 path the reference names as its
// aim for tensor cores that have it (README.md "W4A4", kernels/nvfp4_cuda_v5.cu:1-20 keeps W4A16
// because its target GPU has none).
//
// One CTA (192 threads) computes a 128-row x BN-token tile, K in stages of 256 elements:
//   warp 0      TMA producer: per stage one box of weight bytes (128 rows x 128 B) and one box of
//               activation bytes (BN tokens x 128 B), both K-major with the 128-byte swizzle, and the
//               two boxes of their scale bytes (rows x 16 B), into an ST-stage shared-memory ring;
//               completion by transaction bytes on an mbarrier.
//   warp 1      MMA issuer: 4 tcgen05.mma (K = 64 each) per stage, one elected thread;
//               tcgen05.commit hands the stage back.
//   warps 2..5  scale-factor writers, then the epilogue.  The tensor core reads the scale bytes from
//               tensor memory: for an operand row r (weight row or token) of the tile, lane r % 32,
//               32-bit column r / 32 holds the row's 4 scale bytes of one 64-element K block, the
//               same in all four 32-lane quarters.  Each of the 4 warps owns one quarter: a lane
//               reads 16 scale bytes (one stage) of each of its rows from the ring and writes
//               them with tcgen05.st.  Per stage 16 columns for the weights and max(BN / 8, 16) for the tokens.
// Tensor memory: BN accumulator columns + ST x (16 + max(BN/8, 16)) scale columns.
//
// Every wait is bounded (status word, see nvfp4_gemm_fp4_status); a CTA always runs to its end and
// frees its tensor memory.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nvfp4 {

constexpr int F4_BM = 128;
constexpr int F4_BK = 256;                 // elements of K per stage = 128 bytes per row
constexpr int F4_THREADS = 192;
constexpr int F4_PAIR_THREADS = 352;       // the CTA-pair kernel
constexpr uint32_t F4_SPIN_LIMIT = 1u << 24;

__device__ int g_fp4_status = 0;           // 0 ok; otherwise 1 + id of the wait that ran out

__device__ __forceinline__ bool f4_wait(uint32_t bar, uint32_t parity, int id) {
    for (uint32_t i = 0; i < F4_SPIN_LIMIT; i++)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(&g_fp4_status, 1 + id);
    return false;
}

__device__ __forceinline__ void tcgen05_mma_fp4_block16(uint32_t taddr, uint64_t adesc, uint64_t bdesc,
                                                        uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                                        uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, e;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "@e tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n}\n" ::
            "r"(taddr), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
}
// tcgen05.st, shape 32x32b: lane l of the warp writes NR consecutive 32-bit columns of its own lane
template <int NR>
__device__ __forceinline__ void tcgen05_st_32x32b(uint32_t taddr, const uint32_t* r) {
    static_assert(NR == 1 || NR == 2 || NR == 4 || NR == 8, "column count");
    if constexpr (NR == 1)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};\n" ::"r"(taddr), "r"(r[0]) : "memory");
    else if constexpr (NR == 2)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};\n" ::"r"(taddr), "r"(r[0]),
                     "r"(r[1]) : "memory");
    else if constexpr (NR == 4)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(taddr), "r"(r[0]),
                     "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
    else
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr),
                     "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                     : "memory");
}

__host__ __device__ constexpr int f4_tmem_cols(int need) { return need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512; }

template <int BN, int ST>
__global__ void __launch_bounds__(F4_THREADS)
gemm_fp4_block_scaled_kernel(const __grid_constant__ CUtensorMap w_map,
                             const __grid_constant__ CUtensorMap a_map,
                             const __grid_constant__ CUtensorMap ws_map,
                             const __grid_constant__ CUtensorMap as_map,
                             __half* __restrict__ out, int M, int n_tokens, int K, int ld_out,
                             float* __restrict__ part, unsigned int* __restrict__ counters, int kper) {
    constexpr int A_BYTES = F4_BM * 128;             // weight tile of a stage
    constexpr int B_BYTES = BN * 128;                // token tile of a stage
    constexpr int NB = BN / 32;                      // token rows per lane
    // one MMA's scale bytes start on a 4-column boundary of tensor memory (an address between
    // boundaries raised "misaligned address"), so narrow token tiles leave columns unused
    constexpr int NBC = NB < 4 ? 4 : NB;             // token-scale columns reserved per MMA
    constexpr int SFA_COLS = 16, SFB_COLS = 4 * NBC, SF_COLS = SFA_COLS + SFB_COLS;
    constexpr int TCOLS = f4_tmem_cols(BN + ST * SF_COLS);
    static_assert(BN + ST * SF_COLS <= 512, "tensor memory");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~(uintptr_t)1023);
    constexpr int SA_BYTES = F4_BM * 16;             // weight scale bytes of a stage
    constexpr int SB_BYTES = BN * 16;                // token scale bytes of a stage
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem + ST * A_BYTES;
    uint8_t* smem_sa = smem_b + ST * B_BYTES;
    uint8_t* smem_sb = smem_sa + ST * SA_BYTES;
    __shared__ __align__(8) uint64_t bar_full[ST];    // TMA bytes landed
    __shared__ __align__(8) uint64_t bar_sf[ST];      // scale bytes written to tensor memory
    __shared__ __align__(8) uint64_t bar_empty[ST];   // the stage's MMAs retired
    __shared__ __align__(8) uint64_t bar_accum;       // a tile's accumulation retired
    __shared__ __align__(8) uint64_t bar_acc_free;    // the epilogue has read the accumulator
    __shared__ uint32_t s_tmem;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // A CTA walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ... (row tile fastest): barriers,
    // tensor memory and the tensor maps are set up once, and the copies of the next tile's first
    // stages run under this tile's epilogue.  With a K split (gridDim.z > 1) the grid has one
    // CTA per tile and split.
    const int tiles_m = (M + F4_BM - 1) / F4_BM;
    const int ntiles = tiles_m * ((n_tokens + BN - 1) / BN);
    // K split (gridDim.z > 1; few CTA tiles, e.g. 32 tokens x 5120 rows): this CTA takes the stages
    // [k_first, k_first + ksteps) and the tile's CTAs meet in the epilogue
    const int k_first = (int)blockIdx.z * kper;
    const int ksteps = min(kper, K / F4_BK - k_first);
    __shared__ int s_last;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_sf[s]), 128);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_accum), 1);
        mbar_init(smem_u32(&bar_acc_free), 128);
        fence_barrier_init();
    }
    if (warp == 0) {
        tcgen05_alloc(smem_u32(&s_tmem), TCOLS);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t tmem_sf = tmem + BN;               // scale columns follow the accumulator

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
                const int m0 = (tile % tiles_m) * F4_BM, n0 = (tile / tiles_m) * BN;
                for (int it = 0; it < ksteps; it++) {
                    if (!f4_wait(smem_u32(&bar_empty[s]), ph ^ 1u, 0)) { ok = false; break; }
                    const uint32_t bar = smem_u32(&bar_full[s]);
                    mbar_arrive_expect_tx(bar, A_BYTES + B_BYTES + SA_BYTES + SB_BYTES);
                    // coordinates: x = byte along K (a multiple of 128 / of 16), y = row; rows past
                    // the end of either matrix are filled with zero bytes by the copy engine
                    const int kt = k_first + it;
                    tma_load_2d(smem_u32(smem_a + s * A_BYTES), &w_map, kt * 128, m0, bar);
                    tma_load_2d(smem_u32(smem_b + s * B_BYTES), &a_map, kt * 128, n0, bar);
                    tma_load_2d(smem_u32(smem_sa + s * SA_BYTES), &ws_map, kt * 16, m0, bar);
                    tma_load_2d(smem_u32(smem_sb + s * SB_BYTES), &as_map, kt * 16, n0, bar);
                    if (++s == ST) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // block-scaled instruction descriptor: A and B E2M1 (code 1) K-major, N = BN, scale
        // type E8M0, M = 128, scale-factor ids 0 (a block-16 MMA consumes all four bytes of a
        // column), K = 64
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (1u << 23) |
                               ((uint32_t)(F4_BM >> 4) << 24);
        int s = 0, ti = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ti++) {
            // the epilogue of the tile before must have read the accumulator
            if (ok && ti > 0) ok = f4_wait(smem_u32(&bar_acc_free), (uint32_t)(ti - 1) & 1u, 5);
            tcgen05_fence_after();
            for (int it = 0; it < ksteps; it++) {
                // (the scale writers arrive only after they saw the stage's copies land)
                if (ok) ok = f4_wait(smem_u32(&bar_sf[s]), ph, 1);
                tcgen05_fence_after();
                const uint32_t a_base = smem_u32(smem_a + s * A_BYTES);
                const uint32_t b_base = smem_u32(smem_b + s * B_BYTES);
                const uint32_t sf = tmem_sf + (uint32_t)(s * SF_COLS);
#pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    // 64 elements of K = 32 bytes further along the swizzled 128-byte row
                    const uint64_t adesc = make_desc_sw128(a_base + kk * 32, 16, 1024);
                    const uint64_t bdesc = make_desc_sw128(b_base + kk * 32, 16, 1024);
                    tcgen05_mma_fp4_block16(tmem, adesc, bdesc, idesc, sf + (uint32_t)(kk * 4),
                                            sf + (uint32_t)(SFA_COLS + kk * NBC), (it | kk) != 0 ? 1u : 0u);
                }
                tcgen05_commit(smem_u32(&bar_empty[s]));
                if (++s == ST) { s = 0; ph ^= 1u; }
            }
            tcgen05_commit(smem_u32(&bar_accum));
        }
    } else {
        // ---------------- scale-factor writers ----------------
        const int q = warp & 3;                            // this warp's 32-lane quarter
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        bool ok = true;
        int s = 0, ti = 0;
        uint32_t ph = 0;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ti++) {
        const int m0 = (tile % tiles_m) * F4_BM, n0 = (tile / tiles_m) * BN;
        for (int it = 0; it < ksteps; it++) {
            // The scale bytes travel with the stage (two more TMA boxes: 128 x 16 B and BN x 16 B),
            // so they are requested ST stages ahead like the operands.  (Loaded by the lanes
            // from global memory one stage ahead, they queued behind the operand requests in the
            // SM's request path.)  The stage's landing also means that the MMAs which read this
            // slot's tensor-memory columns a ring round ago have retired.
            if (ok) ok = f4_wait(smem_u32(&bar_full[s]), ph, 3);
            tcgen05_fence_after();
            const uint8_t* sa = smem_sa + s * SA_BYTES;
            const uint8_t* sb = smem_sb + s * SB_BYTES;
            uint4 wv[4], av[NB];
#pragma unroll
            for (int c = 0; c < 4; c++) wv[c] = *reinterpret_cast<const uint4*>(sa + (c * 32 + lane) * 16);
#pragma unroll
            for (int c = 0; c < NB; c++) av[c] = *reinterpret_cast<const uint4*>(sb + (c * 32 + lane) * 16);
            // column 4 kk + c (weights) / kk NBC + c (tokens) = word kk of row c's 16 bytes
            uint32_t wa[4][4], wb[4][NB];
#pragma unroll
            for (int c = 0; c < 4; c++) { wa[0][c] = wv[c].x; wa[1][c] = wv[c].y; wa[2][c] = wv[c].z; wa[3][c] = wv[c].w; }
#pragma unroll
            for (int c = 0; c < NB; c++) { wb[0][c] = av[c].x; wb[1][c] = av[c].y; wb[2][c] = av[c].z; wb[3][c] = av[c].w; }
            const uint32_t sf = tmem_sf + (uint32_t)(s * SF_COLS) + lane_base;
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                tcgen05_st_32x32b<4>(sf + (uint32_t)(kk * 4), wa[kk]);
                tcgen05_st_32x32b<NB>(sf + (uint32_t)(SFA_COLS + kk * NBC), wb[kk]);
            }
            tcgen05_wait_st();
            tcgen05_fence_before();
            mbar_arrive(smem_u32(&bar_sf[s]));
            if (++s == ST) { s = 0; ph ^= 1u; }
        }

        // ---------------- epilogue: tensor memory -> fp16 out[m][token] ----------------
        if (ok) ok = f4_wait(smem_u32(&bar_accum), (uint32_t)ti & 1u, 4);
        tcgen05_fence_after();
        const int m = m0 + q * 32 + lane;
        const int Z = (int)gridDim.z;
        bool reduce = false;
        if (Z > 1) {
            // Every CTA of the tile stores its fp32 partial tile; the one that finds the others'
            // already counted adds them in split order (the same sum whichever CTA comes last) and
            // writes the fp16 result.  Nobody waits for anybody.
            float* mine = part + (((size_t)tile * Z + blockIdx.z) * F4_BM + (q * 32 + lane)) * BN;
#pragma unroll 1
            for (int cb = 0; cb < BN / 32; cb++) {
                uint32_t v[32];
                tcgen05_ld_32x32b_x32(tmem + lane_base + (uint32_t)(cb * 32), v);
                tcgen05_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    __stcg(reinterpret_cast<uint4*>(mine + cb * 32 + j), make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]));
            }
            tcgen05_fence_before();
            mbar_arrive(smem_u32(&bar_acc_free));
            __threadfence();
            asm volatile("bar.sync 1, 128;\n" ::: "memory");
            if (threadIdx.x == 64) {
                const unsigned seen = atomicAdd(counters + tile, 1u);
                s_last = (seen == (unsigned)(Z - 1));
                if (s_last) counters[tile] = 0u;                 // ready for the next launch
            }
            asm volatile("bar.sync 1, 128;\n" ::: "memory");
            reduce = s_last != 0;
            if (reduce) __threadfence();
        }
        if (Z == 1 || reduce) {
#pragma unroll 1
            for (int cb = 0; cb < BN / 32; cb++) {
                uint32_t v[32];
                if (Z == 1) {
                    tcgen05_ld_32x32b_x32(tmem + lane_base + (uint32_t)(cb * 32), v);
                    tcgen05_wait_ld();
                } else {
                    const float* p0 = part + (((size_t)tile * Z) * F4_BM + (q * 32 + lane)) * BN + cb * 32;
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 a = __ldcg(reinterpret_cast<const float4*>(p0 + j));
                        v[j] = __float_as_uint(a.x); v[j + 1] = __float_as_uint(a.y);
                        v[j + 2] = __float_as_uint(a.z); v[j + 3] = __float_as_uint(a.w);
                    }
                    for (int z = 1; z < Z; z++) {
                        const float* pz = p0 + (size_t)z * F4_BM * BN;
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 a = __ldcg(reinterpret_cast<const float4*>(pz + j));
                            v[j] = __float_as_uint(__uint_as_float(v[j]) + a.x);
                            v[j + 1] = __float_as_uint(__uint_as_float(v[j + 1]) + a.y);
                            v[j + 2] = __float_as_uint(__uint_as_float(v[j + 2]) + a.z);
                            v[j + 3] = __float_as_uint(__uint_as_float(v[j + 3]) + a.w);
                        }
                    }
                }
                const int nb = n0 + cb * 32;
                if (m < M && nb < n_tokens) {
                    __half* orow = out + (size_t)m * (size_t)ld_out + nb;
                    if (nb + 32 <= n_tokens && (ld_out & 7) == 0) {
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
                            if (nb + j < n_tokens) orow[j] = __float2half(__uint_as_float(v[j]));
                    }
                }
            }
        }
        if (Z == 1) {     // this thread's part of the accumulator is read: the next tile may overwrite it
            tcgen05_fence_before();
            mbar_arrive(smem_u32(&bar_acc_free));
        }
        }   // tiles
    }

    tcgen05_fence_before();
    __syncthreads();
    if (warp == 0) tcgen05_dealloc(tmem, TCOLS);
}

// ---------------------------------------------------------------------------------------------
// CTA-pair kernel (cluster of two, tcgen05 cta_group::2): a pair walks tiles of 256 weight rows x BN = 192 or 256
// tokens.  Each CTA loads its own 128 weight rows, HALF of the token tile, its rows' scale bytes and the
// scale bytes of all BN tokens (every tensor core needs them); the pair's first CTA issues M = 256 MMAs for both SMs.
//
// What bounds it is the warp that issues the MMAs: a wait takes it 170 cycles, an MMA 60, a copy of scale bytes 20, and a
// stage's MMAs run 440.  So there is one barrier a stage, which the copies of the operands complete themselves, and it is
// asked a stage ahead.  The scale bytes go their own way ahead of the operands: copied 64 bytes a row (four stages) at a
// time, rearranged by four warps into a ring as deep as the operands', and moved to tensor memory by tcgen05.cp,
// issued with the MMAs that read them.  (Warps that store them there have to wait for the MMAs of two stages before.)
// That copy wants a K block's bytes as 32 pieces of 16, piece l = 4 bytes of each of rows l, l + 32, l + 64, l + 96.
// 192 tokens leave room in tensor memory for two accumulators, so that a tile's epilogue (four warps of its own, through
// shared memory and TMA stores) runs under the next tile's MMAs; 256 tokens have one, and 10 % more work per stage.  128
// tokens (few deep tiles only) have two and room for a third: K in parts of kseg stages, which the epilogue warps add up.
// 17408 x 5120 at 8192 tokens 383 -> 338 us (4.3 PFLOP/s; with the K loop's copies alone 233, its MMAs alone 292).
//
// Roles per CTA (352 threads): warp 0 operand copies, warp 1 MMAs (first CTA), warps 2..5 scale bytes, every fourth
// stage each, warps 6..9 epilogue, warp 10 scale copies.
// Barriers (same offsets in both CTAs): full[s] in the first CTA (both CTAs' operands of a stage landed, both CTAs' scale
// bytes rearranged), sfull[u] local (scale bytes of four stages landed), sempty[u] local (rearranged), empty[s] and
// acc_full[a] committed to in each CTA, acc_free[a] in the first CTA (the epilogue warps of both have read the
// accumulator).
// ---------------------------------------------------------------------------------------------
constexpr int F4P_SK = 4;                            // stages per box of scale bytes
constexpr int F4P_SF = 3 * 2048;                     // rearranged scale bytes of a stage: weights, two groups of 128 tokens
constexpr int F4P_OUT = 32 * 64;                     // an epilogue warp's 32 rows x 32 tokens of fp16
template <int BN>
struct F4Pair {
    static constexpr int ACCS = BN == 256 ? 1 : 2;                       // accumulators
    static constexpr bool SEGS = BN == 128;                              // K in segments, whose sums go to a third one
    static constexpr int ST = BN == 256 ? 4 : BN == 192 ? 5 : 6;         // ring of stages
    static constexpr int A = F4_BM * 128, B = BN / 2 * 128;              // operand bytes of a stage
    static constexpr int SA = F4_BM * 16 * F4P_SK, SB = BN * 16 * F4P_SK;    // scale bytes of a box
    static constexpr int SMEM = ST * (A + B + F4P_SF) + 2 * (SA + SB) + 4 * F4P_OUT + 1024;
};

// called by a whole converged warp; one elected lane issues (see tcgen05_mma_f16)
__device__ __forceinline__ void f4p_mma(uint32_t taddr, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sfa,
                                        uint32_t sfb, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, e;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "@e tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n}\n" ::
            "r"(taddr), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
}
// 512 bytes of shared memory (32 pieces of 16) -> 4 columns of tensor memory, all four lane quarters, in both CTAs
__device__ __forceinline__ void f4p_copy(uint32_t taddr, uint64_t desc) {
    asm volatile(
        "{\n.reg .pred e;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "@e tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;\n}\n" ::"r"(taddr), "l"(desc)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs once the MMAs issued so far have retired
__device__ __forceinline__ void f4p_commit(uint32_t bar) {
    asm volatile(
        "{\n.reg .pred e;\n.reg .b16 m;\n"
        "mov.b16 m, 3;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n}\n" ::"r"(bar)
        : "memory");
}
__device__ __forceinline__ void f4p_store(const CUtensorMap* map, uint32_t src, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];\n" ::"l"(map), "r"(src),
                 "r"(c0), "r"(c1)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t f4p_half2(uint32_t a, uint32_t b) {
    const __half2 t = __floats2half2_rn(__uint_as_float(a), __uint_as_float(b));
    return *reinterpret_cast<const uint32_t*>(&t);
}

// o_map: the output as boxes of 32 rows x 32 tokens; only used where `tma_out` (16-byte row pitch)
template <int BN>
__global__ void __launch_bounds__(F4_PAIR_THREADS, 1)
gemm_fp4_pair_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map,
                     const __grid_constant__ CUtensorMap ws_map, const __grid_constant__ CUtensorMap as_map,
                     const __grid_constant__ CUtensorMap o_map, int tma_out, __half* __restrict__ out, int M,
                     int n_tokens, int K, int ld_out, int kseg_) {
    using T = F4Pair<BN>;
    constexpr int HALF = BN / 2, ST = T::ST, SK = F4P_SK, ACCS = T::ACCS;
    constexpr bool SEGS = T::SEGS;
    constexpr int PARTS = BN > 128 ? 3 : 2;          // rearranged scale bytes: weights, groups of 128 tokens
    constexpr int NB = BN / 32;                      // groups of 32 tokens
    constexpr int SFB = 8;                           // token-scale columns per MMA (a multiple of 4)
    constexpr int SF_STRIDE = 64;                    // columns of a stage (two take turns): 16 for the weights, 4 x SFB
    static_assert(NB <= SFB && (ACCS + (SEGS ? 1 : 0)) * BN + 2 * SF_STRIDE <= 512 && 16 + 4 * SFB <= SF_STRIDE, "tensor memory");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~(uintptr_t)1023);
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem_a + ST * T::A;
    uint8_t* smem_sa = smem_b + ST * T::B;
    uint8_t* smem_sb = smem_sa + 2 * T::SA;
    uint8_t* smem_sf = smem_sb + 2 * T::SB;
    uint8_t* smem_o = smem_sf + ST * F4P_SF;
    __shared__ __align__(8) uint64_t bar_full[ST], bar_empty[ST];
    __shared__ __align__(8) uint64_t bar_sfull[2], bar_sempty[2];
    __shared__ __align__(8) uint64_t bar_acc_full[2], bar_acc_free[2];
    __shared__ uint32_t s_tmem;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    // a pair walks the pair tiles pair, pair + pairs, ... (row pair fastest)
    const int pairs = (int)(gridDim.x >> 1), pair0 = (int)(blockIdx.x >> 1);
    const int tiles_m = (M + 2 * F4_BM - 1) / (2 * F4_BM);
    const int ntiles = tiles_m * ((n_tokens + BN - 1) / BN);
    const int ksteps = K / F4_BK, kseg = SEGS ? kseg_ : ksteps;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) {
            mbar_init(smem_u32(&bar_full[s]), 4);        // a copy-issuing thread and a scale warp of each CTA
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int u = 0; u < 2; u++) {
            mbar_init(smem_u32(&bar_sfull[u]), 1);
            mbar_init(smem_u32(&bar_sempty[u]), 4);      // the scale warps of this CTA
            mbar_init(smem_u32(&bar_acc_full[u]), 1);
            mbar_init(smem_u32(&bar_acc_free[u]), 8);    // four epilogue warps of each CTA
        }
        fence_barrier_init();
    }
    if (warp == 0) {
        tcgen05_alloc_pair(smem_u32(&s_tmem), 512);
        tcgen05_relinquish_pair();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();
    tcgen05_fence_after();
    const uint32_t tmem = s_tmem;
    const uint32_t tmem_sum = tmem + ACCS * BN, tmem_sf = tmem + (ACCS + (SEGS ? 1 : 0)) * BN;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0, issued = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int tile = pair0; tile < ntiles && ok; tile += pairs) {
                const int m0 = ((tile % tiles_m) * 2 + (int)rank) * F4_BM, nh = (tile / tiles_m) * BN + (int)rank * HALF;
                for (int it = 0; it < ksteps; it++, issued++) {
                    ok = f4_wait(smem_u32(&bar_empty[s]), ph ^ 1u, 0);
                    if (!ok) break;
                    const uint32_t bar = cluster_map_shared(smem_u32(&bar_full[s]), 0);
                    mbar_arrive_expect_tx_cluster(bar, T::A + T::B);
                    tma_load_2d_pair(smem_u32(smem_a + s * T::A), &w_map, it * 128, m0, bar);
                    tma_load_2d_pair(smem_u32(smem_b + s * T::B), &a_map, it * 128, nh, bar);
                    if (++s == ST) { s = 0; ph ^= 1u; }
                }
            }
            // No copy may be in flight when the CTA leaves, also where a wait has run out.  (full is the first CTA's and
            // counts both CTAs' copies; the second stays until the first has synced.)
            if (rank == 0)
                for (int i = max(issued - ST, 0); i < issued; i++)
                    f4_wait(smem_u32(&bar_full[i % ST]), (uint32_t)(i / ST) & 1u, 7);
        }
    } else if (warp == 10) {
        if (lane == 0) {
            int boxes = 0;
            bool ok = true;
            for (int tile = pair0; tile < ntiles && ok; tile += pairs) {
                const int m0 = ((tile % tiles_m) * 2 + (int)rank) * F4_BM, n0 = (tile / tiles_m) * BN;
                for (int it = 0; it < ksteps; it += SK, boxes++) {
                    const int u = boxes & 1;
                    ok = f4_wait(smem_u32(&bar_sempty[u]), ((uint32_t)(boxes >> 1) & 1u) ^ 1u, 6);
                    if (!ok) break;
                    const uint32_t bar = smem_u32(&bar_sfull[u]);
                    mbar_arrive_expect_tx(bar, T::SA + T::SB);
                    // x = byte along K / 16 (a multiple of 64); what lies past the end of a row or of the matrix is
                    // filled with zero bytes
                    tma_load_2d(smem_u32(smem_sa + u * T::SA), &ws_map, it * 16, m0, bar);
                    tma_load_2d(smem_u32(smem_sb + u * T::SB), &as_map, it * 16, n0, bar);
                }
            }
            for (int i = max(boxes - 2, 0); i < boxes; i++)
                f4_wait(smem_u32(&bar_sfull[i & 1]), (uint32_t)(i >> 1) & 1u, 7);
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (1u << 23) |
                                   ((uint32_t)((2 * F4_BM) >> 4) << 24);
            // descriptors: +1 in the low word = 16 bytes further in shared memory
            const uint64_t a_desc = make_desc_sw128(smem_u32(smem_a), 16, 1024);
            const uint64_t b_desc = make_desc_sw128(smem_u32(smem_b), 16, 1024);
            // scale bytes: 32 rows of 16 bytes, 128 bytes from one eight to the next, no swizzle
            const uint64_t s_desc = (uint64_t)((smem_u32(smem_sf) >> 4) & 0x3FFF) | ((uint64_t)8 << 32) | ((uint64_t)1 << 46);
            int s = 0, set = 0, acc = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true, ready = false;
            for (int tile = pair0; tile < ntiles; tile += pairs) {
                int k0 = 0;
                do {
                    const int k1 = SEGS ? min(k0 + kseg, ksteps) : ksteps;
                    // both CTAs' epilogues must have read what this accumulator held
                    if (ok) ok = f4_wait(smem_u32(&bar_acc_free[acc]), aph ^ 1u, 5);
                    const uint32_t d = tmem + (uint32_t)(acc * BN);
                    for (int it = k0; it < k1; it++) {
                        if (ok && !ready) ok = f4_wait(smem_u32(&bar_full[s]), ph, 1);
                        __syncwarp();
                        tcgen05_fence_after();
                        // the next stage's barrier is asked before this stage's instructions are issued, which hide the
                        // answer's 170 cycles (16 instructions a stage are what this warp can issue in time)
                        const bool wrap = s + 1 == ST;
                        const bool next = mbar_test_wait_cluster(smem_u32(&bar_full[wrap ? 0 : s + 1]), wrap ? ph ^ 1u : ph);
                        const uint64_t ad = a_desc + (uint64_t)(s * (T::A >> 4)), bd = b_desc + (uint64_t)(s * (T::B >> 4));
                        const uint64_t sd = s_desc + (uint64_t)(s * (F4P_SF >> 4));
                        const uint32_t sf = tmem_sf + (uint32_t)(set * SF_STRIDE);
#pragma unroll
                        for (int kk = 0; kk < 4; kk++) {
                            f4p_copy(sf + (uint32_t)(kk * 4), sd + 32 * kk);
                            f4p_copy(sf + (uint32_t)(16 + kk * SFB), sd + 128 + 32 * kk);
                            if (PARTS == 3) f4p_copy(sf + (uint32_t)(16 + kk * SFB + 4), sd + 256 + 32 * kk);
                        }
#pragma unroll
                        for (int kk = 0; kk < 4; kk++)   // 64 elements of K = 32 bytes further along the swizzled row
                            f4p_mma(d, ad + 2 * kk, bd + 2 * kk, idesc, sf + (uint32_t)(kk * 4), sf + (uint32_t)(16 + kk * SFB),
                                    ((SEGS ? it - k0 : it) | kk) != 0 ? 1u : 0u);
                        f4p_commit(smem_u32(&bar_empty[s]));
                        ready = __all_sync(0xffffffffu, next);
                        set ^= 1;
                        if (++s == ST) { s = 0; ph ^= 1u; }
                    }
                    f4p_commit(smem_u32(&bar_acc_full[acc]));
                    if (++acc == ACCS) acc = 0;
                    if (acc == 0) aph ^= 1u;
                    k0 = k1;
                } while (SEGS && k0 < ksteps);
            }
        }
    } else if (warp < 6) {
        // ---------------- scale bytes, rows -> pieces ----------------
        // Every warp goes through every box, in order, and arrives for it, with or without a stage of its own in it: a
        // barrier's parity tells a phase only from the one before, so nobody may be two boxes of a slot ahead or behind.
        const int mine = warp - 2;                         // of the stages i: those with i % 4 == mine
        bool ok = true;
        int g = 0, box = 0;                                // stages and boxes before this tile
        for (int tile = pair0; tile < ntiles; tile += pairs) {
            for (int it0 = 0; it0 < ksteps; it0 += SK, box++) {
                const int u = box & 1, j = (mine - g - it0) & 3;       // own stage of this box: it0 + j
                if (ok) ok = f4_wait(smem_u32(&bar_sfull[u]), (uint32_t)(box >> 1) & 1u, 3);
                __syncwarp();
                if (j < SK && it0 + j < ksteps) {
                    // the slot's pieces have been read: the MMAs of stage i - ST have retired
                    const int i = g + it0 + j, s = i % ST;
                    if (ok) ok = f4_wait(smem_u32(&bar_empty[s]), ((uint32_t)(i / ST) & 1u) ^ 1u, 9);
                    __syncwarp();
                    // 16 bytes of a row: piece j of its 64, in the 64-byte swizzle
                    const int c16 = lane * 64 + (j ^ ((lane >> 1) & 3)) * 16;
                    uint8_t* dst = smem_sf + s * F4P_SF + lane * 16;
#pragma unroll
                    for (int part = 0; part < PARTS; part++) { // weights, tokens 0..127, the others
                        const uint8_t* src = part == 0 ? smem_sa + u * T::SA + c16
                                                       : smem_sb + u * T::SB + (part - 1) * 8192 + c16;
                        uint4 v[4];
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            v[c] = c < 2 || part < 2 || BN == 256 ? *reinterpret_cast<const uint4*>(src + c * 2048) : make_uint4(0u, 0u, 0u, 0u);
                        *reinterpret_cast<uint4*>(dst + part * 2048) = make_uint4(v[0].x, v[1].x, v[2].x, v[3].x);
                        *reinterpret_cast<uint4*>(dst + part * 2048 + 512) = make_uint4(v[0].y, v[1].y, v[2].y, v[3].y);
                        *reinterpret_cast<uint4*>(dst + part * 2048 + 1024) = make_uint4(v[0].z, v[1].z, v[2].z, v[3].z);
                        *reinterpret_cast<uint4*>(dst + part * 2048 + 1536) = make_uint4(v[0].w, v[1].w, v[2].w, v[3].w);
                    }
                    fence_proxy_async_smem();              // the tensor core reads them (async proxy)
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(cluster_map_shared(smem_u32(&bar_full[s]), 0));
                }
                if (lane == 0) mbar_arrive(smem_u32(&bar_sempty[u]));
            }
            g += ksteps;
        }
    } else {
        // ---------------- epilogue: this CTA's 128 rows x BN tokens ----------------
        const int q = warp & 3;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        uint8_t* o = smem_o + (warp - 6) * F4P_OUT;
        bool ok = true;
        int acc = 0;
        uint32_t aph = 0;
        for (int tile = pair0; tile < ntiles; tile += pairs) {
            const int m0 = ((tile % tiles_m) * 2 + (int)rank) * F4_BM + q * 32, n0 = (tile / tiles_m) * BN;
            if (SEGS) {
                // the segments before the last: their sum, in order, beside the accumulators
                for (int k0 = kseg; k0 < ksteps; k0 += kseg) {
                    if (ok) ok = f4_wait(smem_u32(&bar_acc_full[acc]), aph, 4);
                    __syncwarp();
                    tcgen05_fence_after();
#pragma unroll 1
                    for (int cb = 0; cb < BN / 32; cb++) {
                        uint32_t v[32];
                        tcgen05_ld_32x32b_x32(tmem + lane_base + (uint32_t)(acc * BN + cb * 32), v);
                        if (k0 != kseg) {
                            uint32_t p[32];
                            tcgen05_ld_32x32b_x32(tmem_sum + lane_base + (uint32_t)(cb * 32), p);
                            tcgen05_wait_ld();
#pragma unroll
                            for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(p[j]) + __uint_as_float(v[j]));
                        } else {
                            tcgen05_wait_ld();
                        }
#pragma unroll
                        for (int j = 0; j < 32; j += 8)
                            tcgen05_st_32x32b<8>(tmem_sum + lane_base + (uint32_t)(cb * 32 + j), v + j);
                    }
                    tcgen05_wait_st();
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(cluster_map_shared(smem_u32(&bar_acc_free[acc]), 0));
                    if (++acc == ACCS) acc = 0;
                    if (acc == 0) aph ^= 1u;
                }
            }
            if (ok) ok = f4_wait(smem_u32(&bar_acc_full[acc]), aph, 4);
            __syncwarp();
            tcgen05_fence_after();
#pragma unroll 1
            for (int cb = 0; cb < BN / 32; cb++) {
                uint32_t v[32];
                tcgen05_ld_32x32b_x32(tmem + lane_base + (uint32_t)(acc * BN + cb * 32), v);
                if (SEGS && kseg < ksteps) {
                    uint32_t p[32];
                    tcgen05_ld_32x32b_x32(tmem_sum + lane_base + (uint32_t)(cb * 32), p);
                    tcgen05_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(p[j]) + __uint_as_float(v[j]));
                } else {
                    tcgen05_wait_ld();
                }
                if (cb == BN / 32 - 1) {       // the accumulator is read: the MMAs of the tile after the next may start
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(cluster_map_shared(smem_u32(&bar_acc_free[acc]), 0));
                }
                const int nb = n0 + cb * 32;
                if (nb >= n_tokens || m0 >= M) continue;
                // (a TMA store that ends inside 16 bytes writes them all: the last tokens of a ragged count go by hand)
                if (tma_out && (nb + 32 <= n_tokens || (n_tokens & 7) == 0)) {
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint32_t* x = &v[c * 8];
                        *reinterpret_cast<uint4*>(o + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) =
                            make_uint4(f4p_half2(x[0], x[1]), f4p_half2(x[2], x[3]), f4p_half2(x[4], x[5]), f4p_half2(x[6], x[7]));
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) f4p_store(&o_map, smem_u32(o), nb, m0);
                } else if (m0 + lane < M) {
                    __half* orow = out + (size_t)(m0 + lane) * (size_t)ld_out + nb;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const uint32_t* x = &v[c * 8];
                        if (tma_out && nb + c * 8 + 8 <= n_tokens) {
                            *reinterpret_cast<uint4*>(orow + c * 8) =
                                make_uint4(f4p_half2(x[0], x[1]), f4p_half2(x[2], x[3]), f4p_half2(x[4], x[5]), f4p_half2(x[6], x[7]));
                        } else if (nb + c * 8 < n_tokens) {
#pragma unroll
                            for (int j = 0; j < 8; j++)
                                if (nb + c * 8 + j < n_tokens) orow[c * 8 + j] = __float2half(__uint_as_float(x[j]));
                        }
                    }
                }
                __syncwarp();
            }
            if (++acc == ACCS) acc = 0;
            if (acc == 0) aph ^= 1u;
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }

    __syncwarp();
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 0) tcgen05_dealloc_pair(tmem, 512);
}

// Workspace of the K split, one per device: fp32 partial tiles (at most F4_SPLIT_CTAS CTAs of 128 x
// 256 values) and one arrival counter per output tile (zero between launches).  Launches that split
// K share it: they must follow one another in stream order on a device.
constexpr int F4_SPLIT_CTAS = 160;
struct F4Workspace { float* part; unsigned int* counters; };
static F4Workspace g_f4_ws[NVFP4_MAX_DEVICES] = {};
static int g_f4_split = 1;          // 0: never split K
static int g_f4_persistent = 1;     // 0: one CTA per output tile
static int f4_sm_count(int dev) {
    static int sms[NVFP4_MAX_DEVICES] = {0};
    if (!sms[dev] && (cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
                      sms[dev] <= 0))
        sms[dev] = 148;
    return sms[dev];
}

// K split of few deep tiles: stages per part; all of them where it does not pay.  When the output tiles leave more than
// half of the SMs idle AND K is deep (32 tokens x 5120 rows x K 17408 is 40 tiles of 68 stages: 25.2 us unsplit, 16.3 us in
// three parts).  Meeting in the epilogue costs about 4 us, more than a 20-stage tile saves (K = 5120: 10.0 us unsplit, 11.0
// us split), hence the floor of 40 stages; parts keep >= 8 stages each.
static int f4_split_stages(int tiles, int total, int sms) {
    if (!g_f4_split || tiles * 2 > sms || total < 40) return total;
    const int Z = std::max(1, std::min(std::min(sms / tiles, total / 8), F4_SPLIT_CTAS / tiles));
    return (total + Z - 1) / Z;
}

static bool f4_workspace(int dev, cudaStream_t st, F4Workspace* out) {
    F4Workspace& w = g_f4_ws[dev];
    if (!w.part) {
        // (an allocation is not allowed while the stream is being captured: such a launch runs unsplit)
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return false;
        float* p = nullptr;
        unsigned int* c = nullptr;
        if (cudaMalloc(&p, (size_t)F4_SPLIT_CTAS * F4_BM * 256 * sizeof(float)) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (cudaMalloc(&c, F4_SPLIT_CTAS * sizeof(unsigned int)) != cudaSuccess ||
            cudaMemset(c, 0, F4_SPLIT_CTAS * sizeof(unsigned int)) != cudaSuccess) {
            cudaGetLastError();
            cudaFree(p);
            if (c) cudaFree(c);
            return false;
        }
        w.part = p;
        w.counters = c;
    }
    *out = w;
    return true;
}

template <int BN, int ST>
static cudaError_t launch_fp4(const CUtensorMap& wm, const CUtensorMap& am, const CUtensorMap& ws,
                              const CUtensorMap& as, __half* out, int M, int n, int K, int ld,
                              cudaStream_t st) {
    constexpr int SMEM = ST * (F4_BM * 128 + BN * 128 + F4_BM * 16 + BN * 16) + 1024;
    static bool attr[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index();
    if (!attr[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_fp4_block_scaled_kernel<BN, ST>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return e;
        attr[dev] = true;
    }
    const int ntiles = ((M + F4_BM - 1) / F4_BM) * ((n + BN - 1) / BN);
    dim3 grid((unsigned)ntiles, 1, 1);
    const int tiles = ntiles, total = K / F4_BK, sms = f4_sm_count(dev);
    int Z = 1, kper = f4_split_stages(tiles, total, sms);
    F4Workspace w = {nullptr, nullptr};
    if (kper < total && f4_workspace(dev, st, &w)) Z = (total + kper - 1) / kper;      // no split without stages
    else kper = total;
    grid.z = (unsigned)Z;
    // without a K split a CTA per SM walks the tiles (see the kernel); with one, a CTA per tile and split
    if (Z == 1 && g_f4_persistent) grid.x = (unsigned)std::min(ntiles, sms);
    gemm_fp4_block_scaled_kernel<BN, ST><<<grid, F4_THREADS, SMEM, st>>>(wm, am, ws, as, out, M, n, K, ld,
                                                                        w.part, w.counters, kper);
    return cudaGetLastError();
}

static int g_f4_pairs_override = 0;  // pairs of the tile-walking pair kernel (0: one per two SMs)
static int g_f4_pair_bn = 0;        // token tile of the CTA-pair kernel: 192, 256, or 0 = by fp4_pair_tokens
static int g_f4_pair = 1;           // the CTA-pair kernel: 1 = where fp4_pair_tokens says so, 2 = more than 128 tokens, 0 = never

// Token tile of the CTA-pair kernel for this problem, 0 where the single-CTA kernel takes it.  GEMM alone, us, single-CTA
// kernel (as it was chosen before) / pairs of 192 / pairs of 256 tokens:
//   17408 x 5120: 192 tokens 18.2 / 16.5 / 17.4, 256 tokens 17.6 / 23.4 / 18.0, 1000: 57 / 56 / 51, 2048: 106 / 95 / 92,
//   8192: 438 / 373 / 376 (a long run; 383 / 338 apart); 6144 x 5120, 8192: 143 / 121 / 117; 5120 x 17408, 8192: 326 /
//   336 / 306; 4096 x 1024, 8192: 42 / 30 / 34, but 129 tokens 10.6 / 11.4 / 11.8, 800: 12.5 / 13.4 / 13.0.
// Few deep tiles are split over K by the single-CTA kernel, whose CTAs meet in memory: the partial tiles of 128 and more
// tokens are what that waits for.  From 65 tokens on pairs of 128 tokens add the same parts in the same order (*kseg stages
// each), one after the other and in tensor memory, so the bits are the same.  A single accumulation over all of K would do
// as well for speed, but the tensor core truncates the sum it adds to: with scale bytes over 12 binades 1.1e-2 of the
// results of 5120 x 17408 are not the correctly rounded ones then, 3.8e-3 in three parts; of 1024 x 17408 1.1e-2 and, in
// eight, 1.5e-3.  us, single CTAs that meet / pairs of 192 in one accumulation / this: 5120 x 17408, 65 tokens 32.6 /
// 29.4 / 27.3, 129: 57.5 / 30.5 / 28.5; 1024 x 17408, 65: 50.8 / 29.4 / 28.8, 129: 108 / 29.9 / 29.0; 5120 x 10240, 256:
// 55.6 / 21.5 / 19.5.  At 64 tokens the single CTAs take 21.4.
// Both widths run in rounds of pairs, a round costs a part per stage and a fixed part (ns, fitted to the above).
static int fp4_pair_tokens(int M, int n, int K, int* kseg) {
    const int st = K / F4_BK, sms = f4_sm_count(current_device_index());
    const int tiles1 = ((M + F4_BM - 1) / F4_BM) * ((n + 255) / 256);
    *kseg = st;
    if (g_f4_pair == 0) return 0;
    if (g_f4_pair == 1) {
        const int part = f4_split_stages(tiles1, st, sms);
        if (part < st) {
            if (n <= 64) return 0;
            if (g_f4_pair_bn) return g_f4_pair_bn;
            *kseg = part;
            return 128;
        }
        if (n <= 128 || M <= F4_BM) return 0;
        if (st <= 4 && tiles1 <= sms) return 0;
    } else if (n <= 128) {
        return 0;
    }
    if (g_f4_pair_bn) return g_f4_pair_bn;
    const long long rows = (M + 255) / 256, pairs = std::max(1, sms / 2);
    const long long r192 = (rows * ((n + 191) / 192) + pairs - 1) / pairs, r256 = (rows * ((n + 255) / 256) + pairs - 1) / pairs;
    const int bn = r256 * (454LL * st + 2900) < r192 * (407LL * st + 1100) ? 256 : 192;
    // one round of single CTAs on the whole GPU is as fast as one of 256-token pairs, and is there sooner
    return g_f4_pair == 1 && bn == 256 && tiles1 <= sms && st < 40 ? 0 : bn;
}

template <int BN>
static cudaError_t launch_fp4_pair(const CUtensorMap& wm, const CUtensorMap& am, const CUtensorMap& ws,
                                   const CUtensorMap& as, const CUtensorMap& om, bool tma_out, __half* out, int M, int n,
                                   int K, int ld, int kseg, cudaStream_t st) {
    static bool attr[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index();
    if (!attr[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_fp4_pair_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   F4Pair<BN>::SMEM);
        if (e != cudaSuccess) return e;
        attr[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    // a pair of CTAs per pair of SMs walks the 256 x BN tiles (one pair per tile with bit 3 of the config)
    const int ptiles = ((M + 255) / 256) * ((n + BN - 1) / BN);
    const int pairs = g_f4_persistent ? std::min(ptiles, g_f4_pairs_override > 0 ? g_f4_pairs_override
                                                                               : f4_sm_count(dev) / 2)
                                      : ptiles;
    cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
    cfg.blockDim = dim3(F4_PAIR_THREADS, 1, 1);
    cfg.dynamicSmemBytes = F4Pair<BN>::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, gemm_fp4_pair_kernel<BN>, wm, am, ws, as, om, tma_out ? 1 : 0, out, M, n, K, ld, kseg);
}

// scale bytes [rows][K/16]: boxes of 16 bytes (one 256-element stage, unswizzled) or 64 bytes (four of them, 64-byte
// swizzle) x box_rows rows
static bool scale_matrix_map(EncodeTiledFn enc, CUtensorMap* map, const void* base, int rows, int K,
                             int box_rows, int box_bytes) {
    if (box_bytes == 16) return scales_map(enc, map, base, rows, K, box_rows);
    return tile_map(enc, map, CU_TENSOR_MAP_DATA_TYPE_UINT8, base, K / 16, rows, K / 16, box_bytes, box_rows,
                    CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE);
}

}  // namespace nvfp4

extern "C" {

// out[m][t] (fp16, row pitch ld_out elements) = sum_k dequant(W)[m][k] * dequant(A)[t][k], both
// operands NVFP4 (packed [rows][K/2] + E8M0 scales [rows][K/16]).  K % 256 == 0; all five
// pointers 16-byte aligned; ld_out >= n_tokens.  0; -2 for a shape or pointer this kernel does not
// take (callers then use the W4A16 route); -3 when the driver offers no tensor-map encoder; or the
// cudaError_t of the launch.
int launch_nvfp4_gemm_fp4(const uint8_t* w_packed, const uint8_t* w_scales, const uint8_t* a_packed,
                          const uint8_t* a_scales, void* out, int M, int n_tokens, int K, int ld_out,
                          void* stream) {
    using namespace nvfp4;
    if (M <= 0 || n_tokens <= 0 || K <= 0 || K % F4_BK != 0 || ld_out < n_tokens) return NVFP4_ERR_SHAPE;
    if (!w_packed || !w_scales || !a_packed || !a_scales || !out) return NVFP4_ERR_SHAPE;
    if ((((uintptr_t)w_packed | (uintptr_t)w_scales | (uintptr_t)a_packed | (uintptr_t)a_scales |
          (uintptr_t)out) & 15) != 0)
        return NVFP4_ERR_SHAPE;
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return -3;
    const int BN = n_tokens > 128 ? 256 : n_tokens > 64 ? 128 : n_tokens > 32 ? 64 : 32;
    int kseg = 0;
    const int pbn = fp4_pair_tokens(M, n_tokens, K, &kseg);
    const bool pair = pbn != 0;
    CUtensorMap wm, am, wsm, asm_, om;
    const bool tma_out = pair && (ld_out & 7) == 0;
    if (!packed_map(enc, &wm, w_packed, M, K, F4_BM, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
        !packed_map(enc, &am, a_packed, n_tokens, K, pair ? pbn / 2 : BN, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
        !scale_matrix_map(enc, &wsm, w_scales, M, K, F4_BM, pair ? 64 : 16) ||
        !scale_matrix_map(enc, &asm_, a_scales, n_tokens, K, pair ? pbn : BN, pair ? 64 : 16) ||
        // the output [M][ld] as boxes of 32 rows x 32 tokens (what lies past row M or token n is not written)
        (tma_out && !tile_map(enc, &om, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, out, n_tokens, M, ld_out * (long long)sizeof(__half),
                              32, 32, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE)))
        return -3;
    if (!tma_out) om = am;                           // not used by the kernel
    cudaStream_t st = (cudaStream_t)stream;
    __half* o = static_cast<__half*>(out);
    const cudaError_t e =
        pbn == 256 ? launch_fp4_pair<256>(wm, am, wsm, asm_, om, tma_out, o, M, n_tokens, K, ld_out, kseg, st)
      : pbn == 192 ? launch_fp4_pair<192>(wm, am, wsm, asm_, om, tma_out, o, M, n_tokens, K, ld_out, kseg, st)
      : pbn == 128 ? launch_fp4_pair<128>(wm, am, wsm, asm_, om, tma_out, o, M, n_tokens, K, ld_out, kseg, st)
      : BN == 256 ? launch_fp4<256, 4>(wm, am, wsm, asm_, o, M, n_tokens, K, ld_out, st)
      : BN == 128 ? launch_fp4<128, 6>(wm, am, wsm, asm_, o, M, n_tokens, K, ld_out, st)
      : BN == 64  ? launch_fp4<64, 6>(wm, am, wsm, asm_, o, M, n_tokens, K, ld_out, st)
                  : launch_fp4<32, 6>(wm, am, wsm, asm_, o, M, n_tokens, K, ld_out, st);
    return (e == cudaSuccess) ? 0 : (int)e;
}

// 0 if no bounded wait inside the FP4 GEMM has run out since the library was loaded (or since the
// last call with reset != 0); otherwise 1 + the id of the wait.  Synchronises the device.
int nvfp4_gemm_fp4_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, nvfp4::g_fp4_status, sizeof(int)) != cudaSuccess) return -1;
    if (reset) {
        const int z = 0;
        cudaMemcpyToSymbol(nvfp4::g_fp4_status, &z, sizeof(int));
        // a launch that gave up may have left arrival counters of the K split behind
        const nvfp4::F4Workspace& w = nvfp4::g_f4_ws[nvfp4::current_device_index()];
        if (v != 0 && w.counters) cudaMemset(w.counters, 0, nvfp4::F4_SPLIT_CTAS * sizeof(unsigned int));
    }
    return v;
}

// Bit 0: K split of the FP4 GEMM for shapes with few output tiles.  Bit 1: the CTA-pair kernel where it is
// faster.  Bit 2: the CTA-pair kernel for more than 128 tokens.  Bit 3: one CTA (pair) per output tile instead of one
// per SM (two SMs) walking the tiles.  Bits 4, 5: its token tile always 256, always 192.  Bits 8..15: number of pairs of the
// walking pair kernel (0 = half the SM count).  Default 3.
void nvfp4_b200_gemm_fp4_config(int flags) {
    nvfp4::g_f4_split = (flags & 1) ? 1 : 0;
    nvfp4::g_f4_pair = (flags & 4) ? 2 : (flags & 2) ? 1 : 0;
    nvfp4::g_f4_pair_bn = (flags & 16) ? 256 : (flags & 32) ? 192 : 0;
    nvfp4::g_f4_persistent = (flags & 8) ? 0 : 1;
    nvfp4::g_f4_pairs_override = (flags >> 8) & 0xFF;     // bits 8..15: CTA pairs of the tile-walking pair kernel
}

}  // extern "C"
