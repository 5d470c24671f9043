// Dense W4A16 GEMM for more than 128 tokens on CTA pairs: out = dequant(W)[M, K] . act, the arithmetic of
// gemm.cu (weight x block scale in fp16, fp16 products, fp32 accumulation; the same MMAs in the same
// order, so the same bits).
//
// The pair kernel of gemm.cu passes both operands through shared memory: per 64 elements of K an SM
// writes 32 KB there and its tensor core reads 48 KB back, 640 cycles at 128 bytes a clock against 514
// cycles of MMAs.  Here the dequantised weights never enter shared memory: they go to TENSOR MEMORY
// and are the A operand from there, which leaves 16 KB written and 32 KB read; and the weight bytes
// come by TMA instead of through the dequantising warps' registers.
// A cluster of two CTAs = 256 weight rows x bn tokens (128 to 256); each CTA dequantises its own 128 rows and loads
// half of the token tile; one tcgen05.mma.cta_group::2 (M 256, N bn, K 16) runs on both SMs.  Roles, in both
// CTAs unless said otherwise:
//   warp 0       TMA producer of the weight ring (stages of 256 k: 128 rows x 128 packed bytes and
//                128 x 16 scale bytes)
//   warp 1       first CTA only: MMA issuer, units of 128 k = 8 MMAs
//   warp 2       TMA producer of the activation units (bn / 2 tokens x 128 k)
//   warps 4..11  dequantisation: a group of four warps takes every other unit, a warp one 32-row
//                quarter, a lane one row
//   warps 12..19 output
// ready[u] lives in the first CTA and collects four warps and one copy from each CTA; free[u] and accum are
// committed to in both; drain lives in the first CTA.  Tensor memory: 256 accumulator columns and four units of
// 64 columns of A, all 512.
// Where there are more tiles than pairs the launch is one pair per two SMs that goes from tile to tile: loads and
// dequantisation run on into the next tile while the last MMAs of this one retire, and the output warps take the
// accumulator into registers (as the fp16 numbers to be stored) and release it, so that the stores run under the
// next tile's MMAs.  As one cluster per tile, each tile of a pair's turn cost some 7 us beside its MMAs (set-up,
// first bytes, epilogue).  Where every pair has one tile (ONE) nothing follows: the dequantising warps write the
// output themselves (with eight more warps a launch was 1.5 to 2 us longer).
// Every wait is bounded and reported through nvfp4_gemm_status.
//
// Measured, us (in brackets: one cluster per tile, 192 or 256 tokens), 136 / 512 / 800 / 2048 tokens:
//    5120 x 6144    24.0 (26.4) /  28.5 (28.4) /  54 (55)   /  86 (89)
//    5120 x 17408   56.4 (64.2) /  69.7 (69.6) / 135 (134)  / 237 (233)
//   16480 x 5120    27.2 (29.7) /  61 (65)     / 101 (121)  / 227 (255)
//   34816 x 5120    51   (54)   / 116 (133)    / 199 (254)  / 433 (516)
// i.e. 1.5 to 1.7 PFLOP/s at 2048 tokens.
#include <cuda.h>

#include "common.cuh"
#include "gemm_pair.cuh"
#include "gemm_tile.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nvfp4 {

constexpr int GP_THREADS = 640, GP_THREADS_ONE = 384;
constexpr int GP_BM = 128;                         // rows of a CTA
constexpr int GP_BK = 256;                         // K elements of a weight stage
constexpr int GP_UK = 128;                         // K elements of an MMA unit
constexpr int GP_W_BYTES = GP_BM * 128;
constexpr int GP_S_BYTES = GP_BM * 16;
constexpr int GP_NS = 4, GP_NU = 4;
constexpr int GP_B_HALF = 16384;                   // room for 128 tokens x 64 k
constexpr int GP_B_BYTES = 2 * GP_B_HALF;
constexpr int GP_E_BYTES = 16 * GP_BM * 2;         // staging of an output piece: 16 tokens x 128 rows
constexpr int GP_SMEM = GP_NU * GP_B_BYTES + GP_NS * (GP_W_BYTES + GP_S_BYTES) + 1024;
constexpr int GP_COLS = 8;                         // column tiles that take turns over the same weight rows
constexpr uint32_t GP_SPIN_LIMIT = 1u << 24;
constexpr uint32_t GP_PARKED_LIMIT = 100000;       // x 20 us

__device__ int g_pair_status = 0;

__device__ __forceinline__ bool gp_wait(uint32_t bar, uint32_t parity, int id) {
    for (uint32_t i = 0; i < GP_SPIN_LIMIT; i++)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(&g_pair_status, 1 + id);
    return false;
}
// The same for a wait as long as a tile: the hardware parks the thread, which leaves the issue slots to the
// dequantising warps (192-token tiles: 3 % of the launch).
__device__ __forceinline__ bool gp_wait_parked(uint32_t bar, uint32_t parity, int id) {
    for (uint32_t i = 0; i < GP_PARKED_LIMIT; i++)
        if (mbar_try_wait_hint(bar, parity, 20000)) return true;
    atomicExch(&g_pair_status, 1 + id);
    return false;
}
// A operand in each CTA's tensor memory; called by a whole converged warp (see tcgen05_mma_f16)
__device__ __forceinline__ void gp_mma(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p, e;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(bdesc),
        "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void gp_commit(uint32_t bar_cluster) {
    asm volatile(
        "{\n.reg .pred e;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar_cluster)
        : "memory");
}

// Tile t of a launch: column tiles in groups of GP_COLS; in a group the tiles of the same rows follow one another,
// so that pairs running side by side share weights as well as activations in L2.
__device__ __forceinline__ void gp_tile(int t, int rows, int cols, int& row, int& col) {
    const int g = t / (rows * GP_COLS), c0 = g * GP_COLS, nc = min(GP_COLS, cols - c0), i = t - c0 * rows;
    row = i / nc;
    col = c0 + i - row * nc;
}

// 16 accumulator columns of this lane's row as fp16 pairs
__device__ __forceinline__ void gp_load_piece(uint32_t taddr, uint32_t (&h)[8]) {
    uint32_t v[16];
    tcgen05_ld_32x32b_x16(taddr, v);
    tcgen05_wait_ld();
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const __half2 w = __floats2half2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
        h[j] = *reinterpret_cast<const uint32_t*>(&w);
    }
}
// 16 tokens of a thread's row -> memory; the four warps of an output group call this together.
__device__ __forceinline__ void gp_store_piece(const uint32_t (&h)[8], __half* out, int out_mode, __half* stg, int bar,
                                               int rr, int m0, int nb, int M, int N, int ld_out, int n_out) {
    if (out_mode == GEMM_OUT_FM) {
        if (m0 + rr >= M) return;
        __half* o = out + (size_t)(m0 + rr) * (size_t)N + nb;
        if (nb + 16 <= N) {
            *reinterpret_cast<uint4*>(o) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(o + 8) = make_uint4(h[4], h[5], h[6], h[7]);
        } else {
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (nb + j < N) o[j] = __ushort_as_half((unsigned short)(h[j >> 1] >> (16 * (j & 1))));
        }
        return;
    }
    if (out_mode == GEMM_OUT_TM_SILU) {
        // Rows in groups of eight gate rows and their eight up rows: the lane with a gate row takes the even pairs
        // of tokens and the one eight lanes on the odd ones.  The fp16 values and roundings are those of a pass of
        // its own (silu_mul_tokens_kernel), which took 13 us for 34816 rows of 512 tokens; here they run under
        // the next tile's MMAs.  64 results a token, in rows of 72 halves (no bank conflicts).
        const int up = (rr >> 3) & 1, row = rr / 16 * 8 + (rr & 7);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? h[2 * j] : h[2 * j + 1], 8);
            const uint32_t gw = up ? got : h[2 * j], uw = up ? h[2 * j + 1] : got;
            const float2 gf = __half22float2(*reinterpret_cast<const __half2*>(&gw));
            const float2 uf = __half22float2(*reinterpret_cast<const __half2*>(&uw));
            __half* o = stg + (2 * (2 * j + up)) * 72 + row;
            o[0] = __float2half(round_f16(silu_pf(gf.x)) * uf.x);
            o[72] = __float2half(round_f16(silu_pf(gf.y)) * uf.y);
        }
        asm volatile("bar.sync %0, 128;\n" ::"r"(bar) : "memory");
        const int tg = nb + (rr >> 3), mg = m0 / 2 + (rr & 7) * 8;
        if (tg < n_out && mg < M / 2)
            *reinterpret_cast<uint4*>(out + (size_t)tg * (size_t)ld_out + mg) =
                *reinterpret_cast<const uint4*>(stg + (rr >> 3) * 72 + (rr & 7) * 8);
        return;
    }
    // A thread holds one row's tokens, memory wants one token's rows together: turned over in shared memory.  Two
    // pieces alternate, so the one barrier per piece also orders its writes after the reads of the last but one.
#pragma unroll
    for (int j = 0; j < 16; j++) stg[j * GP_BM + rr] = __ushort_as_half((unsigned short)(h[j >> 1] >> (16 * (j & 1))));
    asm volatile("bar.sync %0, 128;\n" ::"r"(bar) : "memory");
    const bool vec = ((ld_out & 7) == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
    uint4 old[2] = {};
    if (out_mode == GEMM_OUT_TM_ADD && vec) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int tg = nb + ((i * 128 + rr) >> 4), mg = m0 + (rr & 15) * 8;
            if (tg < n_out && mg + 8 <= M)
                old[i] = *reinterpret_cast<const uint4*>(out + (size_t)tg * (size_t)ld_out + mg);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int pid = i * 128 + rr, tok = pid >> 4, part = pid & 15;
        const int tg = nb + tok, mg = m0 + part * 8;
        if (tg < n_out && mg < M)
            gemm_store_rows8(*reinterpret_cast<const uint4*>(stg + tok * GP_BM + part * 8),
                             out + (size_t)tg * (size_t)ld_out + mg, vec, M - mg, out_mode == GEMM_OUT_TM_ADD, old[i]);
    }
}

template <bool IN_TM, bool ONE>
__global__ void __launch_bounds__(ONE ? GP_THREADS_ONE : GP_THREADS, 1)
gemm_w4a16_pair_tm_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap s_map,
                          const __grid_constant__ CUtensorMap act_map, __half* out, int M, int N, int K, int ld_out,
                          int out_mode, int n_out, int bn, int rows, int cols) {
    extern __shared__ __align__(1024) uint8_t gp_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gp_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_w = smem + GP_NU * GP_B_BYTES;
    uint8_t* smem_s = smem_w + GP_NS * GP_W_BYTES;
    __shared__ __align__(16) uint8_t smem_e[ONE ? 16 : 4 * GP_E_BYTES];
    __shared__ __align__(8) uint64_t bar_full[GP_NS];    // weight stage landed
    __shared__ __align__(8) uint64_t bar_empty[GP_NS];   // all 8 dequantising warps have read it
    __shared__ __align__(8) uint64_t bar_ready[GP_NU];   // first CTA: both CTAs' A in tensor memory, both halves of B
    __shared__ __align__(8) uint64_t bar_free[GP_NU];    // unit's MMAs retired
    __shared__ __align__(8) uint64_t bar_accum;          // tile's MMAs retired
    __shared__ __align__(8) uint64_t bar_drain;          // first CTA: both CTAs' accumulators have been read
    __shared__ uint32_t s_tmem;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();            // 0 = the CTA that issues the MMAs
    const int half = bn / 2;                             // tokens of this CTA's half of a tile
    const int nst = K / GP_BK, nun = 2 * nst;
    const int tile0 = (int)blockIdx.x >> 1, tiles = ONE ? tile0 + 1 : rows * cols;
    const int stride = (int)gridDim.x >> 1;

    auto request = [&](int m0, int i, int s) {           // weight stage i of the tile at row m0 into slot s
        const uint32_t bar = smem_u32(&bar_full[s]);
        mbar_arrive_expect_tx(bar, GP_W_BYTES + GP_S_BYTES);
        tma_load_2d(smem_u32(smem_w + s * GP_W_BYTES), &w_map, i * 128, m0, bar);
        tma_load_2d(smem_u32(smem_s + s * GP_S_BYTES), &s_map, i * 16, m0, bar);
    };
    // (ONE, at most a hundred tiles or so: by a reciprocal.  gp_tile's divisions ahead of the first copies made 10240 x 5120
    // at 256 tokens 32.3 us instead of 31.8.  Not as a grid of rows x columns, whose clusters land elsewhere: 5120 x 17408
    // at 300 tokens 56.9 us instead of 54.2)
    auto place = [&](int t, int& row, int& col) {
        if (ONE) {
            row = (int)__fdividef((float)t + 0.5f, (float)cols);
            col = t - row * cols;
        } else {
            gp_tile(t, rows, cols, row, col);
        }
    };
    auto rows_of = [&](int t) {                          // first row of this CTA's half of tile t
        int row, col;
        place(t, row, col);
        return (2 * row + (int)rank) * GP_BM;
    };
    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&w_map) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&s_map) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&act_map) : "memory");
        for (int s = 0; s < GP_NS; s++) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 8);
        }
        for (int u = 0; u < GP_NU; u++) {
            mbar_init(smem_u32(&bar_ready[u]), 10);      // four warps and one copy from each CTA
            mbar_init(smem_u32(&bar_free[u]), 1);
        }
        mbar_init(smem_u32(&bar_accum), 1);
        mbar_init(smem_u32(&bar_drain), 16);             // eight warps of each CTA
        fence_barrier_init();
        // weights too wait for the previous kernel: it may be the one that writes them
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        for (int i = 0; i < GP_NS && i < nst; i++) request(rows_of(tile0), i, i);
    }
    if (warp == 1) {
        tcgen05_alloc_pair(smem_u32(&s_tmem), 512);
        tcgen05_relinquish_pair();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();      // the peer's barriers are initialised before anything arrives on them
    tcgen05_fence_after();
    const uint32_t tmem = s_tmem, tmem_a = tmem + 256;
    // The next kernel starts only now: its CTAs must not take tensor memory before this one has all of it,
    // and it may read weights ahead of its own wait (the GEMVs do) that a kernel in front of this one writes.
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            int i = min(GP_NS, nst), issued = i, s = i % GP_NS;
            uint32_t ph = (uint32_t)(i / GP_NS);
            bool ok = true;
            for (int t = tile0; t < tiles && ok; t += stride) {
                const int m0 = rows_of(t);
                for (; i < nst; i++, issued++) {
                    ok = gp_wait(smem_u32(&bar_empty[s]), ph ^ 1u, 0);
                    if (!ok) break;
                    request(m0, i, s);
                    if (++s == GP_NS) { s = 0; ph ^= 1u; }
                }
                i = 0;
            }
            // no copy may be in flight when the CTA leaves, also where a wait has run out
            for (int j = max(issued - GP_NS, 0); j < issued; j++)
                gp_wait(smem_u32(&bar_full[j % GP_NS]), (uint32_t)(j / GP_NS) & 1u, 6);
        }
    } else if (warp == 2) {
        if (lane == 0) {
            const int boxes = (half + 63) / 64;              // token-minor boxes (64 tokens wide) of a half
            const uint32_t tx = (uint32_t)(IN_TM ? 2 * half * 128 : 2 * boxes * 8192);
            int u = 0, issued = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = tile0; t < tiles && ok; t += stride) {
                int row, col;
                place(t, row, col);
                const int nh = col * bn + (int)rank * half;
                for (int i = 0; i < nun; i++, issued++) {
                    ok = gp_wait(smem_u32(&bar_free[u]), ph ^ 1u, 1);
                    if (!ok) break;
                    const uint32_t bar = cluster_map_shared(smem_u32(&bar_ready[u]), 0);
                    mbar_arrive_expect_tx_cluster(bar, tx);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint32_t dst = smem_u32(smem + u * GP_B_BYTES + h * GP_B_HALF);
                        const int k = i * GP_UK + h * 64;
                        if constexpr (IN_TM) {               // half token rows x 64 k
                            tma_load_2d_pair(dst, &act_map, k, nh, bar);
                        } else {                             // boxes of 64 k rows x 64 tokens
                            for (int b = 0; b < boxes; b++)
                                tma_load_2d_pair(dst + b * 8192, &act_map, nh + b * 64, k, bar);
                        }
                    }
                    if (++u == GP_NU) { u = 0; ph ^= 1u; }
                }
            }
            // (ready is the first CTA's and counts both CTAs' copies; the second stays until the first has synced)
            if (rank == 0)
                for (int j = max(issued - GP_NU, 0); j < issued; j++)
                    gp_wait(smem_u32(&bar_ready[j % GP_NU]), (uint32_t)(j / GP_NU) & 1u, 7);
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // D fp32, A fp16 (tensor memory), B fp16 (K-major, or MN-major if token-minor), N = bn, M = 256
            const uint32_t idesc = (1u << 4) | (IN_TM ? 0u : (1u << 16)) | ((uint32_t)(bn >> 3) << 17) |
                                   ((uint32_t)((2 * GP_BM) >> 4) << 24);
            int u = 0;
            uint32_t ph = 0, drained = 1;                    // (nothing to wait for ahead of the first tile)
            bool ok = true;
            for (int t = tile0; t < tiles; t += stride) {
                if (ok) ok = gp_wait(smem_u32(&bar_drain), drained, 8);
                drained ^= 1u;
                for (int i = 0; i < nun; i++) {
                    if (ok) ok = gp_wait(smem_u32(&bar_ready[u]), ph, 2);
                    tcgen05_fence_after();
                    const uint32_t b = smem_u32(smem + u * GP_B_BYTES), a = tmem_a + (uint32_t)(u * 64);
#pragma unroll
                    for (int kk = 0; kk < 8; kk++) {
                        const uint32_t bb = b + (kk >> 2) * GP_B_HALF;
                        const uint64_t bdesc = IN_TM ? make_desc_sw128(bb + (kk & 3) * 32, 16, 1024)
                                                     : make_desc_sw128(bb + (kk & 3) * 2048, 8192, 1024);
                        gp_mma(tmem, a + (uint32_t)(kk * 8), bdesc, idesc, (i | kk) != 0 ? 1u : 0u);
                    }
                    // the unit is free in both CTAs once these MMAs have retired
                    const uint32_t bf = smem_u32(&bar_free[u]);
                    gp_commit(cluster_map_shared(bf, 0));
                    gp_commit(cluster_map_shared(bf, 1));
                    if (++u == GP_NU) { u = 0; ph ^= 1u; }
                }
                const uint32_t ba = smem_u32(&bar_accum);
                gp_commit(cluster_map_shared(ba, 0));
                gp_commit(cluster_map_shared(ba, 1));
            }
        }
    } else if (!ONE && warp >= 12) {
        const int q = warp & 3, grp = (warp - 12) >> 2;        // lane quarter; which pieces of 16 tokens
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16);
        const int rr = q * 32 + lane, pieces = bn / 16;
        int piece = 0;                                         // (goes on through the tiles: staging alternates)
        uint32_t ph = 0;
        bool ok = true;
        for (int t = tile0; t < tiles; t += stride) {
            int row, col;
            place(t, row, col);
            const int m0 = (2 * row + (int)rank) * GP_BM, n0 = col * bn;
            if (ok) ok = gp_wait_parked(smem_u32(&bar_accum), ph, 5);
            ph ^= 1u;
            __syncwarp();
            tcgen05_fence_after();
            // the whole accumulator into registers, as the fp16 numbers that will be stored: the next tile's MMAs
            // wait for this and not for the stores
            uint32_t h[8][8];
#pragma unroll
            for (int p = 0; p < 8; p++) {
                if (2 * p + grp >= pieces) break;
                gp_load_piece(at + (uint32_t)((2 * p + grp) * 16), h[p]);
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_map_shared(smem_u32(&bar_drain), 0));
            // (a loop with the registers moving up: unrolled, its code takes 2 us more to fetch)
#pragma unroll 1
            for (int p = grp; p < pieces; p += 2, piece++) {
                __half* stg = reinterpret_cast<__half*>(smem_e + (2 * grp + (piece & 1)) * GP_E_BYTES);
                gp_store_piece(h[0], out, out_mode, stg, 1 + grp, rr, m0, n0 + p * 16, M, N, ld_out, n_out);
#pragma unroll
                for (int j = 0; j < 56; j++) h[j >> 3][j & 7] = h[(j >> 3) + 1][j & 7];
            }
        }
    } else if (warp >= 4) {
        const int q = warp & 3, grp = (warp - 4) >> 2;         // lane quarter; which units of a stage
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const int r = q * 32 + lane;
        const int stages = nst * ((tiles - tile0 + stride - 1) / stride);   // of all this pair's tiles
        int s = 0, u = grp;                                    // unit i = 2 * stage + grp
        uint32_t sph = 0, uph = 0;
        bool ok = true;
        for (int i = 0; i < stages; i++) {
            if (ok) ok = gp_wait(smem_u32(&bar_full[s]), sph, 3);
            const uint8_t* row = smem_w + s * GP_W_BYTES + r * 128;
            uint4 p[4];
#pragma unroll
            for (int c = 0; c < 4; c++)
                p[c] = *reinterpret_cast<const uint4*>(row + (((grp * 4 + c) ^ (r & 7)) << 4));
            const uint2 sc = *reinterpret_cast<const uint2*>(smem_s + s * GP_S_BYTES + r * 16 + grp * 8);
            if (ok) ok = gp_wait(smem_u32(&bar_free[u]), uph ^ 1u, 4);
            __syncwarp();                                      // every lane's reads of the stage are done, and the
            if (lane == 0) mbar_arrive(smem_u32(&bar_empty[s]));   // stores below are .aligned
            tcgen05_fence_after();
            const uint32_t a = tmem_a + lane_base + (uint32_t)(u * 64);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t o[16];
                gemm_dequant32(p[c], (c < 2 ? sc.x : sc.y) >> (16 * (c & 1)), o);
                tcgen05_st_32x32b_x16(a + (uint32_t)(c * 16), o);
            }
            tcgen05_wait_st();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_map_shared(smem_u32(&bar_ready[u]), 0));
            if (++s == GP_NS) { s = 0; sph ^= 1u; }
            u += 2;
            if (u >= GP_NU) { u -= GP_NU; uph ^= 1u; }
        }
        if constexpr (ONE) {                                   // no next tile to work on: these warps write the output
            int row, col, piece = 0;
            place(tile0, row, col);
            const int m0 = (2 * row + (int)rank) * GP_BM, n0 = col * bn;
            gp_wait(smem_u32(&bar_accum), 0, 5);
            __syncwarp();
            tcgen05_fence_after();
#pragma unroll 1
            for (int b = grp; b < bn / 32; b += 2) {
                uint32_t v[32];
                tcgen05_ld_32x32b_x32(tmem + lane_base + (uint32_t)(b * 32), v);
                tcgen05_wait_ld();
                gemm_store_block(v, out, out_mode, smem, grp, piece, q, lane, m0 + r, m0, n0 + b * 32, M, N, ld_out,
                                 n_out);
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();      // neither CTA leaves (or frees tensor memory) while the other may still use it
    if (warp == 1) tcgen05_dealloc_pair(tmem, 512);
}

// Token tile: a pair does tiles one after the other, so the launch is as long as the most tiles that fall to one pair,
// each of them the MMAs of bn tokens plus the dequantisation's share, some 96 tokens' worth (34816 x 5120, us per
// tile: 19.9 / 20.8 / 23.3 / 24.9 / 28.9 at 128 / 160 / 192 / 224 / 256 tokens).  5120 rows at 512 tokens: 40 tiles
// of 256 on 74 pairs, or 60 of 192 (37 and 28.5 us for K = 6144).  cta_group::2 wants multiples of 32.
static int gp_slots(int dev) {
    static int cached[NVFP4_MAX_DEVICES] = {};
    int& c = cached[dev];
    if (c == 0) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 2) sms = 2;
        c = sms / 2;
    }
    return c;
}
static int gp_tile_tokens(int dev, int M, int N) {
    const long long rows = (M + 2 * GP_BM - 1) / (2 * GP_BM);
    const int slots = gp_slots(dev);
    int best = 256;
    long long least = 0;
    for (int bn = 256; bn >= 128; bn -= 32) {
        const long long cost = ((rows * ((N + bn - 1) / bn) + slots - 1) / slots) * ((bn < 144 ? 144 : bn) + 96);
        if (least == 0 || cost < least) { best = bn; least = cost; }
    }
    return best;
}

// Against the 256-row tiles of gemm.cu (one CTA per 256 rows x 256 tokens, in rounds of as many CTAs as the GPU has
// SMs, each with its own set-up and epilogue; in ns): a pair goes from tile to tile, the stores of one under the
// MMAs of the next, so what is left for the tiles is K so short that the stores take longer than the MMAs and
// there are too few tiles a pair to spread them.  4096 x K at 2048 tokens, token-major / added into the output /
// feature-major, us:
//   K =  256   tiles 14.6 / 15.9 / 12.2, pairs 15.0 / 21.3 / 13.1
//   K = 1024   tiles 23.4 / 24.3 / 20.6, pairs 20.9 / 26.7 / 19.6
//   K = 2048   tiles 34.6 / 36.1 / 32.7, pairs 30.1 / 33.6 / 29.2
bool gemm_pair_beats_tiles(int M, int N, int K, int out_mode) {
    const int dev = current_device_index();
    const long long slots = gp_slots(dev), rows = (M + 255) / 256, bn = gp_tile_tokens(dev, M, N);
    static const int tile_fixed[3] = {9500, 11800, 13000}, store[3] = {3900, 4800, 8500};   // by out_mode; 256 tokens
    const long long tile_rounds = (rows * ((N + 255) / 256) + 2 * slots - 1) / (2 * slots);
    const long long per_pair = (rows * ((N + bn - 1) / bn) + slots - 1) / slots;
    const long long mma = 5LL * K * bn / 256, out = store[out_mode] * bn / 256;
    const long long tiles = tile_rounds * (tile_fixed[out_mode] + 21LL * K / 2);
    const long long pairs = 4500 + mma + (per_pair - 1) * (mma > out ? mma : out) + out;
    return pairs < tiles;
}

template <bool IN_TM, bool ONE>
static cudaError_t gp_launch(const CUtensorMap& wm, const CUtensorMap& sm, const CUtensorMap& am, __half* out, int M,
                             int N, int K, int ld_out, int out_mode, int n_out, int bn, int pairs, cudaStream_t st) {
    static bool opted[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index();
    if (!opted[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_w4a16_pair_tm_kernel<IN_TM, ONE>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM);
        if (e != cudaSuccess) return e;
        opted[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    const int rows = (M + 2 * GP_BM - 1) / (2 * GP_BM), cols = (N + bn - 1) / bn;
    cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
    cfg.blockDim = dim3(ONE ? GP_THREADS_ONE : GP_THREADS, 1, 1);
    cfg.dynamicSmemBytes = GP_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, gemm_w4a16_pair_tm_kernel<IN_TM, ONE>, wm, sm, am, out, M, N, K, ld_out, out_mode,
                              n_out, bn, rows, cols);
}

// The activation in the epilogue makes a tile's stores longer (9.5 us per 256 tokens against 3.9), which costs nothing
// while they run under the next tile's MMAs and pays for itself against a pass of its own.  34816 x K, GEMM and pass /
// fused, us: K = 5120 at 136 / 512 / 2048 tokens 53 / 126 / 475 and 53 / 117 / 427; K = 1024 at 512 42 and 45.
bool gemm_pair_fuses_silu(int M, int N, int K) {
    const int dev = current_device_index();
    const long long bn = gp_tile_tokens(dev, M, N), tiles = (long long)((M + 255) / 256) * ((N + bn - 1) / bn);
    const long long per_pair = (tiles + gp_slots(dev) - 1) / gp_slots(dev);
    if (per_pair < 2) return false;                          // (no output warps)
    const long long mma = 5LL * K * bn / 256, plain = 3900 * bn / 256, silu = 9500 * bn / 256;   // ns
    const long long pass = 500 + (long long)M * N * 3 / 4400;
    return (per_pair - 1) * (mma > silu ? mma : silu) + silu < (per_pair - 1) * (mma > plain ? mma : plain) + plain + pass;
}

bool gemm_pair_takes(const uint8_t* packed, const uint8_t* scales, int N, int K) {
    return N > 128 && K % GP_BK == 0 && (((uintptr_t)packed | (uintptr_t)scales) & 15) == 0;
}

int gemm_pair_launch(const uint8_t* packed, const uint8_t* scales, const __half* act, long long ld_act,
                     bool in_tm, __half* out, int ld_out, int M, int N, int n_tokens, int K, int out_mode,
                     cudaStream_t st) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return -3;
    const int bn = gp_tile_tokens(current_device_index(), M, N);
    CUtensorMap wm, sm, am;
    if (!packed_map(enc, &wm, packed, M, K, GP_BM, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
        !scales_map(enc, &sm, scales, M, K, GP_BM, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
        !tile_map(enc, &am, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, act, in_tm ? K : N, in_tm ? n_tokens : K,
                  ld_act * (long long)sizeof(__half), 64, in_tm ? bn / 2 : 64, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
        return -3;
    const int slots = gp_slots(current_device_index());
    const long long tiles = (long long)((M + 2 * GP_BM - 1) / (2 * GP_BM)) * ((N + bn - 1) / bn);
    const int pairs = (int)(tiles < slots ? tiles : slots);
    const auto launch = tiles <= slots ? (in_tm ? gp_launch<true, true> : gp_launch<false, true>)
                                       : (in_tm ? gp_launch<true, false> : gp_launch<false, false>);
    const cudaError_t e = launch(wm, sm, am, out, M, N, K, ld_out, out_mode, n_tokens, bn, pairs, st);
    return (int)e;
}

int gemm_pair_shared_bytes() { return GP_SMEM; }

int gemm_pair_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_pair_status, sizeof(int)) != cudaSuccess) return -1;
    if (reset) {
        const int z = 0;
        cudaMemcpyToSymbol(g_pair_status, &z, sizeof(int));
    }
    return v;
}

}  // namespace nvfp4
