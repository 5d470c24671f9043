// Dense W4A16 GEMM for at most 128 tokens, 256 on narrow matrices (batched decode, short prompts, ragged prompt ends):
// out = dequant(W)[M, K] . act, the arithmetic of gemm.cu (weight x block scale in fp16, fp16
// products, fp32 accumulation), bound by reading the weights from HBM (0.5625 bytes each).
//
// The tile kernel of gemm.cu keeps 16 KB of weight bytes in flight per SM (registers of the
// dequantising warps) and runs one CTA of K / 64 dependent steps per 128 rows: at 32 tokens it took
// 42 us for 17408 x 5120 (1.2 TB/s) and 129 us for 5120 x 17408 (40 CTAs on 148 SMs).  Here:
//   * raw weight and scale bytes come by TMA into a shared-memory ring (54 to 90 KB in flight per
//     CTA, two CTAs per SM), so the stream does not depend on the dequantising warps' registers;
//   * the dequantised fp16 tile goes to TENSOR MEMORY (tcgen05.st) and is the MMA's A operand from
//     there: no shared-memory write, no second read of it, no proxy fence;
//   * K is split over the CTAs of a cluster (up to 8) until the launch fills the SMs; the fp32 partial
//     tiles meet in distributed shared memory and are added in rank order (reproducible, no
//     workspace in global memory, nobody polls).
// One CTA (384 threads) = 128 weight rows x BN tokens x its share of K, in stages of 256 elements:
//   warp 0       TMA producer of the weight ring (128 rows x 128 packed bytes, 128-byte swizzle, and
//                128 x 16 scale bytes per stage)
//   warp 1       MMA issuer: units of 128 k = 8 x tcgen05.mma.kind::f16 (M 128, N BN, K 16)
//   warp 2       TMA producer of the activation units (BN tokens x 128 k, from L2)
//   warps 4..11  dequantisation: the four warps of a group own one 32-row quarter each and a group
//                takes every other unit; a lane converts 128 weights of its row (16 bytes at a time)
//                and stores 16 tensor-memory columns per chunk
// then all warps: accumulator -> shared memory -> sum over the cluster -> output.
// Every wait is bounded and reported through nvfp4_gemm_status.
//
// Measured (weights cold, graph replay, us; in brackets the tile kernel of gemm.cu), 3 / 32 / 128 tokens:
//   5120 x 6144     9.4 / 10.5 / 15.6   (51 /  50 /  44)      17408 x 5120   17.4 / 18.1 / 22.9   (47 / 42 / 39)
//   5120 x 17408   19.0 / 20.2 / 27.0  (132 / 129 / 111)      34816 x 5120   34.7 / 36.2 / 48.4  (112 / 87 / 89)
// i.e. some 6 us fixed (launch, first bytes, cluster sum) plus 3.5 to 4.5 TB/s.  The stream alone, without
// conversion and MMAs, runs at 6.3 TB/s; the conversions (2 instructions per pair of weights) take
// most of the rest.  128 tokens are bound by the activation units from L2 (32 KB for 9 KB of weights).
#include <cuda.h>

#include "common.cuh"
#include "gemm_few.cuh"
#include "gemm_tile.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nvfp4 {

constexpr int FEW_THREADS = 384;
constexpr int FEW_BM = 128;
constexpr int FEW_BK = 256;                        // K elements of a weight stage
constexpr int FEW_UK = 128;                        // K elements of an MMA unit
constexpr int FEW_A_BYTES = FEW_BM * 128;          // packed bytes of a stage
constexpr int FEW_S_BYTES = FEW_BM * 16;           // scale bytes of a stage
constexpr int FEW_PRE = 2;                         // weight stages requested before the activations
constexpr int FEW_MAX_SPLIT = 8;
constexpr uint32_t FEW_SPIN_LIMIT = 100000;

// weight stages and MMA units in flight, chosen so that two CTAs share an SM's 227 KB
__host__ __device__ constexpr int few_stages(int bn) { return bn <= 16 ? 5 : bn <= 32 ? 4 : bn <= 64 ? 3 : 2; }
__host__ __device__ constexpr int few_units(int bn) { return bn <= 64 ? 3 : 2; }
__host__ __device__ constexpr int few_b_bytes(int bn) { return bn * FEW_UK * 2; }
__host__ __device__ constexpr int few_smem_bytes(int bn) {
    return few_stages(bn) * (FEW_A_BYTES + FEW_S_BYTES) + few_units(bn) * few_b_bytes(bn) + 1024;
}

__device__ int g_few_status = 0;

// Bounded wait (about 2 s); the hardware parks the thread meanwhile.  That matters: CTAs of the next
// kernel in the stream share the SM under programmatic dependent launch and would otherwise take
// issue slots from this one's while they wait.
__device__ __forceinline__ bool few_wait(uint32_t bar, uint32_t parity, int id) {
    for (uint32_t i = 0; i < FEW_SPIN_LIMIT; i++)
        if (mbar_try_wait_hint(bar, parity, 20000)) return true;
    atomicExch(&g_few_status, 1 + id);
    return false;
}

__device__ __forceinline__ void few_ld_x8(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ float4 few_ld_cluster(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

__device__ __forceinline__ float few_ld_cluster1(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

template <int BN, bool IN_TM>
__global__ void __launch_bounds__(FEW_THREADS, 2)
gemm_w4a16_few_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap s_map,
                      const __grid_constant__ CUtensorMap act_map, __half* out, int M, int N, int K, int ld_out,
                      int out_mode, int n_out, int split) {
    constexpr int NS = few_stages(BN), NU = few_units(BN), B_BYTES = few_b_bytes(BN);
    constexpr uint32_t TMEM_COLS = 256;            // BN accumulator columns + NU x 64 columns of A
    static_assert(BN + NU * 64 <= 256, "two CTAs share the 512 tensor-memory columns");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~(uintptr_t)1023);
    uint8_t* smem_w = smem;                                    // NS x 16 KB packed weights
    uint8_t* smem_b = smem_w + NS * FEW_A_BYTES;               // NU activation units
    uint8_t* smem_s = smem_b + NU * B_BYTES;                   // NS x 2 KB scale bytes
    __shared__ __align__(8) uint64_t bar_full[NS];     // weight stage landed
    __shared__ __align__(8) uint64_t bar_empty[NS];    // all 8 dequantising warps have read it
    __shared__ __align__(8) uint64_t bar_ready[NU];    // unit's A in tensor memory, its B landed
    __shared__ __align__(8) uint64_t bar_free[NU];     // unit's MMAs retired
    __shared__ __align__(8) uint64_t bar_accum;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t bar_breq;         // the first activation units have been requested

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % split;                  // = rank in the cluster (split CTAs along x)
    const int m0 = ((int)blockIdx.x / split) * FEW_BM, n0 = (int)blockIdx.y * BN;
    const int nk = K / FEW_BK;
    const int st0 = nk * rank / split, nst = nk * (rank + 1) / split - st0;   // this CTA's stages

    auto request = [&](int i, int s) {                         // weight stage i of this CTA into slot s
        const uint32_t bar = smem_u32(&bar_full[s]);
        mbar_arrive_expect_tx(bar, FEW_A_BYTES + FEW_S_BYTES);
        tma_load_2d(smem_u32(smem_w + s * FEW_A_BYTES), &w_map, (st0 + i) * 128, m0, bar);
        tma_load_2d(smem_u32(smem_s + s * FEW_S_BYTES), &s_map, (st0 + i) * 16, m0, bar);
    };
    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&w_map) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&s_map) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&act_map) : "memory");
        for (int s = 0; s < NS; s++) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 8);
        }
        for (int u = 0; u < NU; u++) {
            mbar_init(smem_u32(&bar_ready[u]), 5);             // four dequantising warps + the copy's issuer
            mbar_init(smem_u32(&bar_free[u]), 1);
        }
        mbar_init(smem_u32(&bar_accum), 1);
        mbar_init(smem_u32(&bar_breq), 1);
        fence_barrier_init();
        // Weights too wait for the previous kernel: it may be the one that writes them (requested ahead
        // of the wait, a launch is 0.3 to 0.9 us shorter and reads what was there before).
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        for (int i = 0; i < FEW_PRE && i < nst; i++) request(i, i);
    }
    if (warp == 1) {
        tcgen05_alloc(smem_u32(&s_tmem), TMEM_COLS);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = s_tmem, tmem_a = tmem + BN;
    // The next kernel starts after the wait, not before: it may read weights of its own ahead of its wait
    // (the GEMVs do), and those may come from a kernel in front of this one.
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            // the other stages follow the first activation units, which would queue behind them in
            // the SM's request path
            few_wait(smem_u32(&bar_breq), 0, 6);
            int s = FEW_PRE, issued = min(FEW_PRE, nst);
            uint32_t ph = 0;
            for (int i = FEW_PRE; i < nst; i++, issued++) {
                if (s == NS) { s = 0; ph ^= 1u; }
                if (!few_wait(smem_u32(&bar_empty[s]), ph ^ 1u, 0)) break;
                request(i, s++);
            }
            // no copy may be in flight when the CTA leaves, also where a wait has run out
            for (int i = max(issued - NS, 0); i < issued; i++)
                few_wait(smem_u32(&bar_full[i % NS]), (uint32_t)(i / NS) & 1u, 7);
        }
    } else if (warp == 2) {
        if (lane == 0) {
            int u = 0, issued = 0;
            uint32_t ph = 0;
            for (int i = 0; i < 2 * nst; i++, issued++) {
                if (!few_wait(smem_u32(&bar_free[u]), ph ^ 1u, 1)) break;
                const uint32_t bar = smem_u32(&bar_ready[u]);
                const uint32_t dst = smem_u32(smem_b + u * B_BYTES);
                const int k = st0 * FEW_BK + i * FEW_UK;
                mbar_arrive_expect_tx(bar, B_BYTES);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if constexpr (IN_TM) {         // BN token rows x 64 k
                        tma_load_2d(dst + h * (BN * 128), &act_map, k + h * 64, n0, bar);
                    } else {                       // boxes of 64 k rows x 64 tokens
#pragma unroll
                        for (int b = 0; b < BN / 64; b++)
                            tma_load_2d(dst + h * (BN * 128) + b * 8192, &act_map, n0 + b * 64, k + h * 64, bar);
                    }
                }
                if (i == (NU < 2 * nst ? NU : 2 * nst) - 1) mbar_arrive(smem_u32(&bar_breq));
                if (++u == NU) { u = 0; ph ^= 1u; }
            }
            for (int i = max(issued - NU, 0); i < issued; i++)
                few_wait(smem_u32(&bar_ready[i % NU]), (uint32_t)(i / NU) & 1u, 8);
        }
    } else if (warp == 1) {
        // D fp32, A fp16 (tensor memory), B fp16 (K-major, or MN-major if token-minor), N = BN, M = 128
        const uint32_t idesc = (1u << 4) | (IN_TM ? 0u : (1u << 16)) | ((uint32_t)(BN >> 3) << 17) |
                               ((uint32_t)(FEW_BM >> 4) << 24);
        int u = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int i = 0; i < 2 * nst; i++) {
            if (ok) ok = few_wait(smem_u32(&bar_ready[u]), ph, 2);
            tcgen05_fence_after();
            const uint32_t b = smem_u32(smem_b + u * B_BYTES);
            const uint32_t a = tmem_a + (uint32_t)(u * 64);
#pragma unroll
            for (int kk = 0; kk < 8; kk++) {
                const uint32_t bb = b + (kk >> 2) * (BN * 128);
                const uint64_t bdesc = IN_TM ? make_desc_sw128(bb + (kk & 3) * 32, 16, 1024)
                                             : make_desc_sw128(bb + (kk & 3) * 2048, 8192, 1024);
                tcgen05_mma_f16_ta(tmem, a + (uint32_t)(kk * 8), bdesc, idesc, (i | kk) != 0 ? 1u : 0u);
            }
            tcgen05_commit(smem_u32(&bar_free[u]));
            if (++u == NU) { u = 0; ph ^= 1u; }
        }
        tcgen05_commit(smem_u32(&bar_accum));
    } else if (warp >= 4) {
        const int q = warp & 3, grp = (warp - 4) >> 2;         // lane quarter; which units of a stage
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const int r = q * 32 + lane;
        int s = 0, u = grp;                                    // unit i = 2 * stage + grp
        uint32_t sph = 0, uph = 0;
        bool ok = true;
        for (int i = 0; i < nst; i++) {
            if (ok) ok = few_wait(smem_u32(&bar_full[s]), sph, 3);
            const uint8_t* row = smem_w + s * FEW_A_BYTES + r * 128;
            uint4 p[4];
#pragma unroll
            for (int c = 0; c < 4; c++)
                p[c] = *reinterpret_cast<const uint4*>(row + (((grp * 4 + c) ^ (r & 7)) << 4));
            const uint2 sc = *reinterpret_cast<const uint2*>(smem_s + s * FEW_S_BYTES + r * 16 + grp * 8);
            if (ok) ok = few_wait(smem_u32(&bar_free[u]), uph ^ 1u, 4);
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
            if (lane == 0) mbar_arrive(smem_u32(&bar_ready[u]));
            if (++s == NS) { s = 0; sph ^= 1u; }
            u += 2;
            if (u >= NU) { u -= NU; uph ^= 1u; }
        }
        // accumulator -> shared memory [token][row] (the rings are idle: every copy has been consumed)
        few_wait(smem_u32(&bar_accum), 0, 5);
        __syncwarp();
        tcgen05_fence_after();
        float* red = reinterpret_cast<float*>(smem);
        constexpr int CW = BN / 2;                             // token columns per group
        uint32_t v[CW];
#pragma unroll
        for (int c = 0; c < CW; c += 8) few_ld_x8(tmem + lane_base + (uint32_t)(grp * CW + c), v + c);
        tcgen05_wait_ld();
#pragma unroll
        for (int c = 0; c < CW; c++) red[(grp * CW + c) * FEW_BM + r] = __uint_as_float(v[c]);
    }
    tcgen05_fence_before();
    __syncthreads();
    if (split > 1) cluster_sync_all();

    // ---- sum over the cluster and output ----
    const uint32_t red0 = smem_u32(smem);
    if (out_mode == GEMM_OUT_FM) {
        // A warp takes 32 rows, a lane one row's 8 tokens: one 16-byte store (N % 8 == 0).  Storing a token's
        // rows two bytes at a time, N halves apart, cost 65536 x 1024 at 128 tokens 55 us of 95.
        const int groups = min(BN, N - n0) / 8;
        for (int w = rank + split * warp; w < 4 * groups; w += split * (FEW_THREADS / 32)) {
            const int r = (w & 3) * 32 + lane, t = (w >> 2) * 8;
            const uint32_t at = red0 + (uint32_t)(t * FEW_BM + r) * 4u;
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; e++) f[e] = 0.0f;
            for (int c = 0; c < split; c++) {
                const uint32_t src = cluster_map_shared(at, (uint32_t)c);
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = few_ld_cluster1(src + (uint32_t)(e * FEW_BM * 4));
#pragma unroll
                for (int e = 0; e < 8; e++) f[e] = c == 0 ? v[e] : f[e] + v[e];
            }
            if (m0 + r >= M) continue;
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const __half2 h = __floats2half2_rn(f[2 * e], f[2 * e + 1]);
                o[e] = *reinterpret_cast<const uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(out + (size_t)(m0 + r) * (size_t)N + n0 + t) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
    // token-major: a warp takes one token's 128 rows, a lane four of them
    const int limit = out_mode == GEMM_OUT_FM ? 0 : n_out - n0;
    for (int t = rank + split * warp; t < BN && t < limit; t += split * (FEW_THREADS / 32)) {
        const uint32_t at = red0 + (uint32_t)(t * FEW_BM + lane * 4) * 4u;
        float4 part[FEW_MAX_SPLIT];
#pragma unroll
        for (int c = 0; c < FEW_MAX_SPLIT; c++)
            if (c < split) part[c] = few_ld_cluster(cluster_map_shared(at, (uint32_t)c));
        float4 a = part[0];
#pragma unroll
        for (int c = 1; c < FEW_MAX_SPLIT; c++)
            if (c < split) { a.x += part[c].x; a.y += part[c].y; a.z += part[c].z; a.w += part[c].w; }
        float f[4] = {a.x, a.y, a.z, a.w};
        const int m = m0 + lane * 4;
        __half* o = out + (size_t)(n0 + t) * (size_t)ld_out + m;
        if (m + 4 <= M && (((uintptr_t)o & 7) == 0)) {
            if (out_mode == GEMM_OUT_TM_ADD) {
                const uint2 old = *reinterpret_cast<const uint2*>(o);
                const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&old.x));
                const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&old.y));
                f[0] = round_f16(f[0]) + lo.x; f[1] = round_f16(f[1]) + lo.y;
                f[2] = round_f16(f[2]) + hi.x; f[3] = round_f16(f[3]) + hi.y;
            }
            const __half2 h0 = __floats2half2_rn(f[0], f[1]), h1 = __floats2half2_rn(f[2], f[3]);
            uint2 w;
            w.x = *reinterpret_cast<const uint32_t*>(&h0);
            w.y = *reinterpret_cast<const uint32_t*>(&h1);
            *reinterpret_cast<uint2*>(o) = w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (m + e < M)
                    o[e] = out_mode == GEMM_OUT_TM_ADD
                               ? __float2half(round_f16(f[e]) + __half2float(o[e])) : __float2half(f[e]);
        }
    }
    if (split > 1) cluster_sync_all();       // nobody leaves while a peer still reads its shared memory
    if (warp == 1) tcgen05_dealloc(tmem, TMEM_COLS);
}

// the opt-in to more than 48 KB of dynamic shared memory, once per instantiation and device
template <int BN, bool IN_TM>
static cudaError_t few_opt_in(int dev) {
    static bool done[NVFP4_MAX_DEVICES] = {false};
    if (done[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(gemm_w4a16_few_kernel<BN, IN_TM>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, few_smem_bytes(BN));
    if (e == cudaSuccess)      // two CTAs per SM need the whole carve-out
        e = cudaFuncSetAttribute(gemm_w4a16_few_kernel<BN, IN_TM>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) done[dev] = true;
    return e;
}

// How many clusters of `split` CTAs run at once with two CTAs per SM.  Clusters live inside a GPC
// and GPCs differ in size, so the driver is asked, with a kernel that fills an SM's shared memory by
// itself (one CTA per SM): a GPC of n SMs then holds n / split clusters, and with two CTAs per SM
// 2 n / split - for an even split the answer for split / 2.
__global__ void few_one_per_sm_kernel() {}
static int few_clusters_one_per_sm(int dev, int split) {
    static int cached[NVFP4_MAX_DEVICES][FEW_MAX_SPLIT + 1] = {};
    int& c = cached[dev][split];
    if (c == 0) {
        constexpr int SMEM = 200 * 1024;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)split, 1, 1);
        cfg.blockDim = dim3(FEW_THREADS, 1, 1);
        cfg.dynamicSmemBytes = SMEM;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)split;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(few_one_per_sm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, few_one_per_sm_kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        c = n > 0 ? n : -1;
    }
    return c > 0 ? c : 0;
}
static int few_clusters(int dev, int split) {
    if (split % 2 == 0) return few_clusters_one_per_sm(dev, split / 2);
    const int twice = 2 * few_clusters_one_per_sm(dev, split);
    const int wider = few_clusters_one_per_sm(dev, (split + 1) / 2);
    return twice > wider ? twice : wider;
}
// Of four CTAs fewer clusters are placed than the answer for two, 74: 71 run at once, and a launch of 72 takes half as
// long again and more.  66 always fit, two layers of clusters with a CTA per SM; this is the mean of both.
int gemm_few_clusters(int dev, int split) {
    return split == 4 ? (few_clusters(dev, 4) + 2 * few_clusters_one_per_sm(dev, 4)) / 2 : few_clusters(dev, split);
}

template <int BN, bool IN_TM>
static cudaError_t few_launch(const CUtensorMap& wm, const CUtensorMap& sm, const CUtensorMap& am, __half* out,
                              int M, int N, int K, int ld_out, int out_mode, int n_out, cudaStream_t st) {
    const int dev = current_device_index();
    const cudaError_t opt = few_opt_in<BN, IN_TM>(dev);
    if (opt != cudaSuccess) return opt;
    const int rows = (M + FEW_BM - 1) / FEW_BM, cols = (N + BN - 1) / BN, nk = K / FEW_BK;
    // K split: the fewest stages per CTA among the splits whose clusters all run at once.  (One column tile keeps to four
    // parts for 71 to 74 row tiles too: 9216 x 5120 at 26 tokens takes 15.8 us with them and 11.9 with three, but with
    // fewer parts the sums in them are longer, and a third more of the results are not the correctly rounded ones.)
    int split = 1;
    for (int s = 2; s <= FEW_MAX_SPLIT && s <= nk; s++)
        if ((long long)rows * cols <= (cols == 1 ? few_clusters(dev, s) : gemm_few_clusters(dev, s)) && (nk + s - 1) / s < (nk + split - 1) / split) split = s;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(rows * split), (unsigned)cols, 1);
    cfg.blockDim = dim3(FEW_THREADS, 1, 1);
    cfg.dynamicSmemBytes = few_smem_bytes(BN);
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)split;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, gemm_w4a16_few_kernel<BN, IN_TM>, wm, sm, am, out, M, N, K, ld_out, out_mode,
                              n_out, split);
}

bool gemm_few_takes(const uint8_t* packed, const uint8_t* scales, int N, int K) {
    return N <= GEMM_FEW_MAX_TOKENS && K % FEW_BK == 0 && (((uintptr_t)packed | (uintptr_t)scales) & 15) == 0;
}

// 129 to 256 tokens are two column tiles of 128.  For narrow matrices the CTA pairs of gemm_pair.cu leave most of the GPU
// idle, while here K is split until the SMs are full: pairs / this kernel at 129 and 256 tokens, us: 1024 x 5120 19.3
// / 9.9 and 19.7 / 11.8, 5120 x 6144 23.7 / 19.3 and 24.8 / 19.5, 5120 x 17408 53.7 / 39.3 and 56.1 / 41.6, 1024 x 17408
// 51.4 / 18.2 and 51.4 / 20.5.  Wider ones are split less and read their weights twice (6144 x 5120 21.0 / 20.0,
// feature-major 22.7 / 24.8; 10240 x 5120 23.3 / 31.4), and a short K leaves a CTA too little
// (5120 x 1024 9.2 / 9.7 at 256, feature-major 9.3 / 10.4; 2048 x 1024 8.7 / 7.0).  The line is at 42 row tiles of 148 SMs:
// 84 of the 90 clusters of three CTAs that run at once; with more, K is split over two, and 48 row tiles already lose.
bool gemm_few_takes_two(const uint8_t* packed, const uint8_t* scales, int M, int N, int K) {
    const int rows = (M + FEW_BM - 1) / FEW_BM;
    return N > GEMM_FEW_MAX_TOKENS && N <= 2 * GEMM_FEW_MAX_TOKENS && K % FEW_BK == 0 &&
           (((uintptr_t)packed | (uintptr_t)scales) & 15) == 0 && (K >= 12 * FEW_BK || rows <= 20) &&
           rows * 7 <= 2 * device_sms(current_device_index());
}

int gemm_few_launch(const uint8_t* packed, const uint8_t* scales, const __half* act, long long ld_act,
                    bool in_tm, __half* out, int ld_out, int M, int N, int n_tokens, int K, int out_mode,
                    cudaStream_t st) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return -3;
    // token tile: the narrowest that holds all tokens; token-minor boxes are 64 tokens wide
    const int bn = N > 64 ? 128 : (!in_tm || N > 32) ? 64 : N > 16 ? 32 : 16;
    CUtensorMap wm, sm, am;
    if (!packed_map(enc, &wm, packed, M, K, FEW_BM, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) ||
        !scales_map(enc, &sm, scales, M, K, FEW_BM) ||
        !tile_map(enc, &am, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, act, in_tm ? K : N, in_tm ? n_tokens : K,
                  ld_act * (long long)sizeof(__half), 64, in_tm ? bn : 64, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
        return -3;
    cudaError_t e;
#define FEW_CASE(B) \
    if (bn == B) e = in_tm ? few_launch<B, true>(wm, sm, am, out, M, N, K, ld_out, out_mode, n_tokens, st) \
                           : few_launch<(B < 64 ? 64 : B), false>(wm, sm, am, out, M, N, K, ld_out, out_mode, n_tokens, st); else
    FEW_CASE(16) FEW_CASE(32) FEW_CASE(64) FEW_CASE(128) e = cudaErrorInvalidValue;
#undef FEW_CASE
    return (e == cudaSuccess) ? 0 : (int)e;
}

int gemm_few_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_few_status, sizeof(int)) != cudaSuccess) return -1;
    if (reset) {
        const int z = 0;
        cudaMemcpyToSymbol(g_few_status, &z, sizeof(int));
    }
    return v;
}

}  // namespace nvfp4
