// Dense W4A16 GEMM for more than 128 tokens on CTA pairs: out = dequant(W)[M, K] . act, the arithmetic of
// gemm.cu (weight x block scale in fp16, fp16 products, fp32 accumulation; the same MMAs in the same
// order, so the same bits).
//
// The pair kernel of gemm.cu passes both operands through shared memory: per 64 elements of K an SM
// writes 32 KB there and its tensor core reads 48 KB back, 640 cycles at 128 bytes a clock against 514
// cycles of MMAs.  Here the dequantised weights never enter shared memory: they go to TENSOR MEMORY
// and are the A operand from there, which leaves 16 KB written and 32 KB read; and the weight bytes
// come by TMA instead of through the dequantising warps' registers.
// A cluster of two CTAs (384 threads each) = 256 weight rows x BN tokens; each CTA dequantises its own
// 128 rows and loads half of the token tile; one tcgen05.mma.cta_group::2 (M 256, N BN, K 16) runs on
// both SMs.  Roles, in both CTAs unless said otherwise:
//   warp 0       TMA producer of the weight ring (stages of 256 k: 128 rows x 128 packed bytes and
//                128 x 16 scale bytes)
//   warp 1       first CTA only: MMA issuer, units of 128 k = 8 MMAs
//   warp 2       TMA producer of the activation units (BN / 2 tokens x 128 k)
//   warps 4..11  dequantisation: a group of four warps takes every other unit, a warp one 32-row
//                quarter, a lane one row
// then warps 4..11 write the output.  ready[u] lives in the first CTA and collects four warps and one
// copy from each CTA; free[u] and accum are committed to in both.  Tensor memory: BN accumulator
// columns and four units of 64 columns of A (all 512 for BN = 256).
// Every wait is bounded and reported through nvfp4_gemm_status.
//
// Measured, us (in brackets the better of the two kernels of gemm.cu), 136 / 2048 tokens:
//   5120 x 6144    26.4 (44.7) /  88 (154)     16480 x 5120   27.1 (41.4) / 251 (289)
//   5120 x 17408   63.5 (110)  / 231 (410)     34816 x 5120   64.1 (83.4) / 506 (617)
// i.e. 1.4 to 1.6 PFLOP/s at 2048 tokens.
#include <cuda.h>

#include "common.cuh"
#include "gemm_pair.cuh"
#include "gemm_tile.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nvfp4 {

constexpr int GP_THREADS = 384;
constexpr int GP_BM = 128;                         // rows of a CTA
constexpr int GP_BK = 256;                         // K elements of a weight stage
constexpr int GP_UK = 128;                         // K elements of an MMA unit
constexpr int GP_W_BYTES = GP_BM * 128;
constexpr int GP_S_BYTES = GP_BM * 16;
constexpr int GP_NS = 4, GP_NU = 4;
constexpr int GP_B_HALF = 16384;                   // room for 128 tokens x 64 k
constexpr int GP_B_BYTES = 2 * GP_B_HALF;
constexpr int GP_SMEM = GP_NU * GP_B_BYTES + GP_NS * (GP_W_BYTES + GP_S_BYTES) + 1024;
constexpr uint32_t GP_SPIN_LIMIT = 1u << 24;

__device__ int g_pair_status = 0;

__device__ __forceinline__ bool gp_wait(uint32_t bar, uint32_t parity, int id) {
    for (uint32_t i = 0; i < GP_SPIN_LIMIT; i++)
        if (mbar_try_wait(bar, parity)) return true;
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

template <int BN, bool IN_TM>
__global__ void __launch_bounds__(GP_THREADS, 1)
gemm_w4a16_pair_tm_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap s_map,
                          const __grid_constant__ CUtensorMap act_map, __half* out, int M, int N, int K, int ld_out,
                          int out_mode, int n_out) {
    constexpr int HALF = BN / 2;                   // tokens of this CTA's half of the tile
    constexpr int BOXES = (HALF + 63) / 64;        // token-minor boxes (64 tokens wide) of a half
    constexpr int TX = IN_TM ? 2 * HALF * 128 : 2 * BOXES * 8192;
    extern __shared__ __align__(1024) uint8_t gp_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gp_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_w = smem + GP_NU * GP_B_BYTES;
    uint8_t* smem_s = smem_w + GP_NS * GP_W_BYTES;
    __shared__ __align__(8) uint64_t bar_full[GP_NS];    // weight stage landed
    __shared__ __align__(8) uint64_t bar_empty[GP_NS];   // all 8 dequantising warps have read it
    __shared__ __align__(8) uint64_t bar_ready[GP_NU];   // first CTA: both CTAs' A in tensor memory, both halves of B
    __shared__ __align__(8) uint64_t bar_free[GP_NU];    // unit's MMAs retired
    __shared__ __align__(8) uint64_t bar_accum;
    __shared__ uint32_t s_tmem;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();            // 0 = the CTA that issues the MMAs
    const int m0 = (int)blockIdx.x * GP_BM;              // blockIdx.x = 2 * pair + rank
    const int n0 = (int)blockIdx.y * BN, nh = n0 + (int)rank * HALF;
    const int nst = K / GP_BK, nun = 2 * nst;

    auto request = [&](int i, int s) {                   // weight stage i into slot s
        const uint32_t bar = smem_u32(&bar_full[s]);
        mbar_arrive_expect_tx(bar, GP_W_BYTES + GP_S_BYTES);
        tma_load_2d(smem_u32(smem_w + s * GP_W_BYTES), &w_map, i * 128, m0, bar);
        tma_load_2d(smem_u32(smem_s + s * GP_S_BYTES), &s_map, i * 16, m0, bar);
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
        fence_barrier_init();
        // weights too wait for the previous kernel: it may be the one that writes them
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        for (int i = 0; i < GP_NS && i < nst; i++) request(i, i);
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
            int s = 0, issued = min(GP_NS, nst);
            uint32_t ph = 0;
            for (int i = GP_NS; i < nst; i++, issued++) {
                if (!gp_wait(smem_u32(&bar_empty[s]), ph, 0)) break;
                request(i, s);
                if (++s == GP_NS) { s = 0; ph ^= 1u; }
            }
            // no copy may be in flight when the CTA leaves, also where a wait has run out
            for (int i = max(issued - GP_NS, 0); i < issued; i++)
                gp_wait(smem_u32(&bar_full[i % GP_NS]), (uint32_t)(i / GP_NS) & 1u, 6);
        }
    } else if (warp == 2) {
        if (lane == 0) {
            int u = 0, issued = 0;
            uint32_t ph = 0;
            for (int i = 0; i < nun; i++, issued++) {
                if (!gp_wait(smem_u32(&bar_free[u]), ph ^ 1u, 1)) break;
                const uint32_t bar = cluster_map_shared(smem_u32(&bar_ready[u]), 0);
                mbar_arrive_expect_tx_cluster(bar, TX);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t dst = smem_u32(smem + u * GP_B_BYTES + h * GP_B_HALF);
                    const int k = i * GP_UK + h * 64;
                    if constexpr (IN_TM) {               // HALF token rows x 64 k
                        tma_load_2d_pair(dst, &act_map, k, nh, bar);
                    } else {                             // boxes of 64 k rows x 64 tokens
#pragma unroll
                        for (int b = 0; b < BOXES; b++) tma_load_2d_pair(dst + b * 8192, &act_map, nh + b * 64, k, bar);
                    }
                }
                if (++u == GP_NU) { u = 0; ph ^= 1u; }
            }
            // (ready is the first CTA's and counts both CTAs' copies; the second stays until the first has synced)
            if (rank == 0)
                for (int i = max(issued - GP_NU, 0); i < issued; i++)
                    gp_wait(smem_u32(&bar_ready[i % GP_NU]), (uint32_t)(i / GP_NU) & 1u, 7);
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // D fp32, A fp16 (tensor memory), B fp16 (K-major, or MN-major if token-minor), N = BN, M = 256
            const uint32_t idesc = (1u << 4) | (IN_TM ? 0u : (1u << 16)) | ((uint32_t)(BN >> 3) << 17) |
                                   ((uint32_t)((2 * GP_BM) >> 4) << 24);
            int u = 0;
            uint32_t ph = 0;
            bool ok = true;
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
    } else if (warp >= 4) {
        const int q = warp & 3, grp = (warp - 4) >> 2;         // lane quarter; which units of a stage
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const int r = q * 32 + lane;
        int s = 0, u = grp;                                    // unit i = 2 * stage + grp
        uint32_t sph = 0, uph = 0;
        bool ok = true;
        for (int i = 0; i < nst; i++) {
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
        gp_wait(smem_u32(&bar_accum), 0, 5);
        __syncwarp();
        tcgen05_fence_after();
        constexpr int CB = BN / 32 / 2;                        // 32-token blocks of a column half
        int piece = 0;
#pragma unroll 1
        for (int cbi = 0; cbi < CB; cbi++) {
            const int cb = grp * CB + cbi;
            uint32_t v[32];
            tcgen05_ld_32x32b_x32(tmem + lane_base + (uint32_t)(cb * 32), v);
            tcgen05_wait_ld();
            gemm_store_block(v, out, out_mode, smem, grp, piece, q, lane, m0 + r, m0, n0 + cb * 32, M, N, ld_out,
                             n_out);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();      // neither CTA leaves (or frees tensor memory) while the other may still use it
    if (warp == 1) tcgen05_dealloc_pair(tmem, 512);
}

// Token tile: the launch runs in rounds of as many pairs as the GPU holds, each of them about
// BN tokens long (plus a fixed part of some 30 tokens' worth), so the width that wastes least of the
// last round wins.  5120 rows at 512 tokens: 40 pairs of 256 tokens on 74, or 60 of 192.
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
    auto cost = [&](int bn) { return ((rows * ((N + bn - 1) / bn) + slots - 1) / slots) * (long long)(bn + 30); };
    return cost(192) < cost(256) ? 192 : 256;
}

// Against the 256-row tiles of gemm.cu (one CTA per 256 rows x 256 tokens), which overlap less but have
// twice the tensor memory to themselves: both run in rounds, a round costs a fixed part (set-up, first
// bytes, epilogue) and a part per k, in ns.  The fixed part counts twice here, two rounds of pairs doing the
// work of one of tiles.  17408 x K at 2048 tokens, token-major / added into the output / feature-major, us:
//   K =  512   tiles 64 / 103 / 57, pairs 70 / 124 / 74       K = 3072   tiles 191 / 249 / 183, pairs 169 / 243 / 180
bool gemm_pair_beats_tiles(int M, int N, int K, int out_mode) {
    const int dev = current_device_index();
    const long long slots = gp_slots(dev), rows = (M + 255) / 256, bn = gp_tile_tokens(dev, M, N);
    static const int tile_fixed[3] = {8700, 9700, 17000};                // by out_mode
    static const int pair_fixed[2][3] = {{6800, 6300, 10500}, {7100, 6100, 11700}};   // 192, 256 tokens
    const long long tile_rounds = (rows * ((N + 255) / 256) + 2 * slots - 1) / (2 * slots);
    const long long pair_rounds = (rows * ((N + bn - 1) / bn) + slots - 1) / slots;
    const long long tiles = tile_rounds * (tile_fixed[out_mode] + 119LL * K / 10);
    const long long pairs = pair_rounds * (pair_fixed[bn == 256][out_mode] + 5LL * K * bn / 256);
    return pairs < tiles;
}

template <int BN, bool IN_TM>
static cudaError_t gp_launch(const CUtensorMap& wm, const CUtensorMap& sm, const CUtensorMap& am, __half* out, int M,
                             int N, int K, int ld_out, int out_mode, int n_out, cudaStream_t st) {
    static bool opted[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index();
    if (!opted[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_w4a16_pair_tm_kernel<BN, IN_TM>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM);
        if (e != cudaSuccess) return e;
        opted[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * ((M + 2 * GP_BM - 1) / (2 * GP_BM))), (unsigned)((N + BN - 1) / BN), 1);
    cfg.blockDim = dim3(GP_THREADS, 1, 1);
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
    return cudaLaunchKernelEx(&cfg, gemm_w4a16_pair_tm_kernel<BN, IN_TM>, wm, sm, am, out, M, N, K, ld_out, out_mode,
                              n_out);
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
    const cuuint32_t estr[2] = {1, 1};
    auto encode = [&](CUtensorMap& m, CUtensorMapDataType type, const void* p, cuuint64_t d0, cuuint64_t d1,
                      cuuint64_t stride, cuuint32_t b0, cuuint32_t b1, CUtensorMapSwizzle swizzle) {
        const cuuint64_t dims[2] = {d0, d1}, strides[1] = {stride};
        const cuuint32_t box[2] = {b0, b1};
        return enc(&m, type, 2, const_cast<void*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!encode(wm, CU_TENSOR_MAP_DATA_TYPE_UINT8, packed, (cuuint64_t)(K / 2), (cuuint64_t)M, (cuuint64_t)(K / 2), 128,
                GP_BM, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode(sm, CU_TENSOR_MAP_DATA_TYPE_UINT8, scales, (cuuint64_t)(K / 16), (cuuint64_t)M, (cuuint64_t)(K / 16), 16,
                GP_BM, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !encode(am, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, act, (cuuint64_t)(in_tm ? K : N), (cuuint64_t)(in_tm ? n_tokens : K),
                (cuuint64_t)ld_act * sizeof(__half), 64, (cuuint32_t)(in_tm ? bn / 2 : 64), CU_TENSOR_MAP_SWIZZLE_128B))
        return -3;
    cudaError_t e;
    if (bn == 256)
        e = in_tm ? gp_launch<256, true>(wm, sm, am, out, M, N, K, ld_out, out_mode, n_tokens, st)
                  : gp_launch<256, false>(wm, sm, am, out, M, N, K, ld_out, out_mode, n_tokens, st);
    else
        e = in_tm ? gp_launch<192, true>(wm, sm, am, out, M, N, K, ld_out, out_mode, n_tokens, st)
                  : gp_launch<192, false>(wm, sm, am, out, M, N, K, ld_out, out_mode, n_tokens, st);
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
