// NVFP4 GEMV of two activations on the block-scaled FP4 tensor-core path: the data path of gemv_tc.cu (weights HBM -> shared
// memory -> tensor core, the fp16 activations as exact base-4 digit columns, fp32 accumulation) with 32 digit columns in
// the place of 16, which cost the tensor core the same.  The register-streaming kernel converts every weight and
// activation to fp16 operands in registers and stops at 3 TB/s.
//
// One row tile of 128 is one CLUSTER of up to eight CTAs that split its K; their sums meet in the first one's shared memory
// through distributed shared memory, in rank order.  So launches on several streams share nothing (the one-activation
// kernel's partial sums meet in a workspace of the device).  One round: problems of more tiles than clusters run at once
// stay with the register-streaming kernel.
//
// CTA of 320 threads, two per SM (roles as in gemv_tc.cu):
//   warp 0      TMA producer: 5-stage ring of 128 rows x 256 k (16 KB) and its scale bytes (2 KB); two stages are
//               requested at entry, ahead of the previous kernel's end (weights), the others behind the activation loads
//   warp 1      MMA issuer: four MMAs M128 N32 K64 a stage
//   warps 2..5  scale bytes of the weights and of the digit columns -> tensor memory
//   warps 6..9  digit conversion, a warp one activation of every other stage; then the sums of their rows
// An activation with a value that is not finite has no digits: its sums are NaN, and rows that are not finite are summed in
// plain fp32 from global memory.
// Every wait is bounded and reported through nvfp4_gemv_tc_status (20 + id).
//
// Measured: at gemv_tc2_faster.
#include <cuda.h>

#include "common.cuh"
#include "gemm_few.cuh"
#include "gemv_tc.cuh"
#include "gemv_tc2.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nvfp4 {

constexpr int T2_THREADS = 320;
constexpr int T2_ST = 5;                        // weight ring
constexpr int T2_NB = 3;                        // ring of digit planes (with four, an SM holds one CTA only)
constexpr int T2_B_BYTES = 32 * 128;            // both activations' digit planes of a stage
constexpr int T2_SF_COLS = 32;                  // tensor-memory columns of a stage's scale bytes
constexpr int T2_PRE = 2;                       // weight stages requested at entry
constexpr int T2_MAX_SPLIT = 8;
constexpr int T2_SMEM = T2_ST * (TC_A_BYTES + TC_S_BYTES) + T2_NB * (T2_B_BYTES + 32) + 1024;

__device__ int g_tc2_status = 0;

__device__ __forceinline__ bool t2_wait(uint32_t bar, uint32_t parity, int id) {
    for (uint32_t i = 0; i < (1u << 24); i++)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(&g_tc2_status, 1 + id);
    return false;
}

// eight elements from k on of activation a
template <bool IL>
__device__ __forceinline__ uint4 t2_load(const __half* x0, const __half* x1, int a, int k) {
    if (!IL) return *reinterpret_cast<const uint4*>((a ? x1 : x0) + k);
    const uint4 p = *reinterpret_cast<const uint4*>(x0 + 2 * k), q = *reinterpret_cast<const uint4*>(x0 + 2 * k + 8);
    const uint32_t sel = a ? 0x7632u : 0x5410u;
    return make_uint4(tc_prmt(p.x, p.y, sel), tc_prmt(p.z, p.w, sel), tc_prmt(q.x, q.y, sel), tc_prmt(q.z, q.w, sel));
}

template <bool IL>
struct T2Load {
    const __half *x0, *x1;
    int a;
    __device__ __forceinline__ uint4 operator()(int k) const { return t2_load<IL>(x0, x1, a, k); }
};

template <bool IL>
__global__ void __launch_bounds__(T2_THREADS)
gemv_tc2_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap s_map,
                const uint8_t* __restrict__ packed, const uint8_t* __restrict__ scales, const __half* x0, const __half* x1,
                __half* y, int M, int K, int split) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    constexpr int ST = T2_ST, NB = T2_NB;
    extern __shared__ __align__(1024) uint8_t t2_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(t2_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_a = smem;                                   // packed weights
    uint8_t* smem_b = smem_a + ST * TC_A_BYTES;               // digit planes: 16 rows of each activation
    uint8_t* smem_s = smem_b + NB * T2_B_BYTES;               // weight scale bytes
    uint8_t* smem_l = smem_s + ST * TC_S_BYTES;               // exponent bytes, 16 of each activation
    __shared__ __align__(8) uint64_t bar_full[ST];            // TMA bytes landed
    __shared__ __align__(8) uint64_t bar_ready[ST];           // scale bytes in tensor memory, digits written
    __shared__ __align__(8) uint64_t bar_empty[ST];           // the stage's MMAs retired
    __shared__ __align__(8) uint64_t bar_bfull[NB], bar_bempty[NB];
    __shared__ __align__(8) uint64_t bar_acc;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_xreq;                           // the activation loads have been issued
    __shared__ float s_red[T2_MAX_SPLIT][2][TC_BM];           // (first CTA) every CTA's sums

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % split, tile = (int)blockIdx.x / split;
    const int nk = K / TC_BK, st0 = rank * nk / split, nst = (rank + 1) * nk / split - st0;
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");       // this CTA runs (waited for below)

    auto request = [&](int i, int s) {
        const uint32_t bar = smem_u32(&bar_full[s]);
        mbar_arrive_expect_tx(bar, TC_A_BYTES + TC_S_BYTES);
        tma_load_2d(smem_u32(smem_a + s * TC_A_BYTES), &w_map, (st0 + i) * 128, tile * TC_BM, bar);
        tma_load_2d(smem_u32(smem_s + s * TC_S_BYTES), &s_map, (st0 + i) * 16, tile * TC_BM, bar);
    };
    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&w_map) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&s_map) : "memory");
        for (int s = 0; s < ST; s++) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_ready[s]), 128);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int s = 0; s < NB; s++) {
            mbar_init(smem_u32(&bar_bfull[s]), 2);            // a warp for each activation
            mbar_init(smem_u32(&bar_bempty[s]), 1);
        }
        mbar_init(smem_u32(&bar_acc), 1);
        s_xreq = 0;
        fence_barrier_init();
        for (int i = 0; i < T2_PRE && i < nst; i++) request(i, i);
    }
    if (warp == 1) {
        tcgen05_alloc(smem_u32(&s_tmem), 256);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = s_tmem, tmem_sf = tmem + 32;

    float sum[2] = {0.0f, 0.0f};
    if (warp == 0) {
        if (lane == 0) {
            for (uint32_t w = 0; w < (1u << 24) && s_xreq == 0; w++) {}
            int s = T2_PRE % ST, issued = min(T2_PRE, nst);
            uint32_t ph = 0;
            for (int i = T2_PRE; i < nst; i++, issued++) {
                if (!t2_wait(smem_u32(&bar_empty[s]), ph ^ 1u, 0)) break;
                request(i, s);
                if (++s == ST) { s = 0; ph ^= 1u; }
            }
            // no copy may be in flight when the CTA leaves, also where a wait has run out
            for (int i = max(issued - ST, 0); i < issued; i++) t2_wait(smem_u32(&bar_full[i % ST]), (uint32_t)(i / ST) & 1u, 1);
        }
        __syncwarp();
    } else {
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        PDL_FRESH(x0); PDL_FRESH(x1); PDL_FRESH(y);
        if (warp == 1) {
            // A, B E2M1 K-major; N = 32; E8M0 scales; M = 128
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(32 >> 3) << 17) | (1u << 23) |
                                   ((uint32_t)(TC_BM >> 4) << 24);
            const uint64_t a_desc0 = make_desc_sw128(smem_u32(smem_a), 16, 1024);
            const uint64_t b_desc0 = make_desc_sw128(smem_u32(smem_b), 16, 1024);
            int s = 0, bs = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int i = 0; i < nst; i++) {
                if (ok) ok = t2_wait(smem_u32(&bar_ready[s]), ph, 2);
                __syncwarp();
                tcgen05_fence_after();
                const uint64_t adesc = a_desc0 + (uint64_t)(s * (TC_A_BYTES >> 4));
                const uint64_t bdesc = b_desc0 + (uint64_t)(bs * (T2_B_BYTES >> 4));
                const uint32_t sf = tmem_sf + (uint32_t)(s * T2_SF_COLS);
                tc_mma(tmem, adesc, bdesc, idesc, sf, sf + 16, i == 0 ? 0u : 1u);
                tc_mma(tmem, adesc + 2, bdesc + 2, idesc, sf + 4, sf + 20, 1u);
                tc_mma(tmem, adesc + 4, bdesc + 4, idesc, sf + 8, sf + 24, 1u);
                tc_mma(tmem, adesc + 6, bdesc + 6, idesc, sf + 12, sf + 28, 1u);
                tcgen05_commit(smem_u32(&bar_empty[s]));
                tcgen05_commit(smem_u32(&bar_bempty[bs]));
                if (++s == ST) { s = 0; ph ^= 1u; }
                if (++bs == NB) bs = 0;
            }
            tcgen05_commit(smem_u32(&bar_acc));
        } else if (warp < 6) {
            const int q = warp & 3;                               // lane quarter
            const uint32_t lane_base = (uint32_t)(q * 32) << 16;
            const uint32_t sub = 0x01010101u * (uint32_t)(2 * (lane & 15));
            bool ok = true;
            int s = 0, bs = 0;
            uint32_t ph = 0, bph = 0;
            for (int i = 0; i < nst; i++) {
                if (ok) ok = t2_wait(smem_u32(&bar_bfull[bs]), bph, 3);
                // digit column n of activation lane / 16, block blk: exponent byte L_blk + 125 - 2n
                const uint4 lw = *reinterpret_cast<const uint4*>(smem_l + bs * 32 + (lane >> 4) * 16);
                if (ok) ok = t2_wait(smem_u32(&bar_full[s]), ph, 4);
                __syncwarp();
                tcgen05_fence_after();
                const uint8_t* ss = smem_s + s * TC_S_BYTES + lane * 16;      // row c * 32 + lane: 4 MMAs x 4 blocks
                const uint4 r0 = *reinterpret_cast<const uint4*>(ss);
                const uint4 r1 = *reinterpret_cast<const uint4*>(ss + 512);
                const uint4 r2 = *reinterpret_cast<const uint4*>(ss + 1024);
                const uint4 r3 = *reinterpret_cast<const uint4*>(ss + 1536);
                const uint32_t cols[32] = {r0.x, r1.x, r2.x, r3.x, r0.y, r1.y, r2.y, r3.y,
                                           r0.z, r1.z, r2.z, r3.z, r0.w, r1.w, r2.w, r3.w,
                                           lw.x - sub, 0u, 0u, 0u, lw.y - sub, 0u, 0u, 0u,
                                           lw.z - sub, 0u, 0u, 0u, lw.w - sub, 0u, 0u, 0u};
                tc_st_x32(tmem_sf + (uint32_t)(s * T2_SF_COLS) + lane_base, cols);
                tcgen05_wait_st();
                tcgen05_fence_before();
                mbar_arrive(smem_u32(&bar_ready[s]));
                if (++s == ST) { s = 0; ph ^= 1u; }
                if (++bs == NB) { bs = 0; bph ^= 1u; }
            }
        } else {
            // warp f of the four: activation f & 1, stages f >> 1, (f >> 1) + 2, ..
            const int f = warp - 6, a = f & 1, q = warp & 3;
            const uint32_t lane_base = (uint32_t)(q * 32) << 16;
            int i = f >> 1;
            uint4 next = make_uint4(0u, 0u, 0u, 0u);
            if (i < nst) next = t2_load<IL>(x0, x1, a, (st0 + i) * TC_BK + lane * 8);
            if (threadIdx.x == 192) s_xreq = 1;
            for (; i < nst; i += 2) {
                const int slot = i % NB;
                const uint4 xv = next;
                if (i + 2 < nst) next = t2_load<IL>(x0, x1, a, (st0 + i + 2) * TC_BK + lane * 8);
                t2_wait(smem_u32(&bar_bempty[slot]), ((uint32_t)(i / NB) & 1u) ^ 1u, 5);
                __syncwarp();
                tc_digit_planes(xv, smem_b + slot * T2_B_BYTES + a * 2048, smem_l + slot * 32 + a * 16, lane);
                fence_proxy_async_smem();        // the tensor core reads the planes (async proxy)
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bar_bfull[slot]));
            }
            t2_wait(smem_u32(&bar_acc), 0, 6);
            __syncwarp();
            tcgen05_fence_after();
            uint32_t v[32];
            tcgen05_ld_32x32b_x32(tmem + lane_base, v);
            tcgen05_wait_ld();
#pragma unroll
            for (int j = 15; j >= 0; j--) {      // small digits first
                sum[0] += __uint_as_float(v[j]);
                sum[1] += __uint_as_float(v[16 + j]);
            }
        }
    }
    asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");                 // the first CTA runs
    const int r = (warp & 3) * 32 + lane;                        // (warps 6..9)
    if (warp >= 6)
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const uint32_t dst = cluster_map_shared(smem_u32(&s_red[rank][t][r]), 0);
            asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(dst), "f"(sum[t]) : "memory");
        }
    tcgen05_fence_before();
    asm volatile("barrier.cluster.arrive.release.aligned;\n"
                 "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");         // every CTA's sums are there
    tcgen05_fence_after();
    if (warp == 1) tcgen05_dealloc(tmem, 256);
    const int row = tile * TC_BM + r;
    if (rank == 0 && warp >= 6 && row < M)
#pragma unroll
        for (int t = 0; t < 2; t++) {
            float tot = s_red[0][t][r];
            for (int c = 1; c < split; c++) tot += s_red[c][t][r];
            if (tc_not_finite(tot)) tot = tc_plain_row(packed, scales, T2Load<IL>{x0, x1, t}, row, K);
            y[(size_t)t * M + row] = __float2half(tot);
        }
}

template <bool IL>
static cudaError_t t2_launch(const CUtensorMap& wm, const CUtensorMap& sm, const uint8_t* packed, const uint8_t* scales,
                             const __half* x0, const __half* x1, __half* y, int M, int K, int split, cudaStream_t st) {
    static bool opted[NVFP4_MAX_DEVICES] = {false};
    const int dev = current_device_index();
    if (!opted[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemv_tc2_kernel<IL>, cudaFuncAttributeMaxDynamicSharedMemorySize, T2_SMEM);
        if (e == cudaSuccess)      // two CTAs per SM need the whole carve-out
            e = cudaFuncSetAttribute(gemv_tc2_kernel<IL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        opted[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((M + TC_BM - 1) / TC_BM * split));
    cfg.blockDim = dim3(T2_THREADS);
    cfg.dynamicSmemBytes = T2_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)split;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = gemv_reads_ahead() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemv_tc2_kernel<IL>, wm, sm, packed, scales, x0, x1, y, M, K, split);
}

// K split: the fewest stages per CTA among the splits whose clusters all run at once; 0 where none does.
static int t2_split(int M, int K) {
    const int dev = current_device_index(), tiles = (M + TC_BM - 1) / TC_BM, nk = K / TC_BK;
    int best = 0;
    for (int s = 1; s <= T2_MAX_SPLIT && s <= nk; s++) {
        const int fit = s == 1 ? 2 * device_sms(dev) : gemm_few_clusters(dev, s);
        if (tiles <= fit && (!best || (nk + s - 1) / s < (nk + best - 1) / best)) best = s;
    }
    return best;
}

// us of a chain of launches with the weights cold / in L2, register-streaming kernel and this one:
//    2048 x 5120   5.3 / 4.1   4.6 / 4.6       9216 x 3072   6.2 / 5.9   6.1 / 5.9       19456 x 4096  13.5 / 12.8  13.8 / 13.4
//    6144 x 3072   4.6 / 4.5   4.8 / 4.7      10240 x 4096   8.1 / 7.5   7.4 / 7.0       19456 x 6144  18.9 / 17.8  19.1 / 18.3
//    4096 x 4096   4.9 / 4.5   5.3 / 5.2      12288 x 4096   8.8 / 7.9   8.5 / 8.1       24576 x 4096  16.1 / 15.0  14.2 / 13.4
//    2560 x 5120   5.5 / 5.1   4.6 / 4.7      12288 x 5120  10.8 / 9.3  10.1 / 9.3       17408 x 5120  17.1 / 16.5  11.4 /  9.5
//    6144 x 5120   6.6 / 6.2   6.2 / 5.9      12288 x 6144  12.9 / 11.2 11.6 / 10.6       5120 x 17408 17.2 / 14.9  11.5 / 10.8
// A stage of a CTA costs this kernel 0.6 us on top of 3.4, whichever way the tiles are split.  The other one goes in rounds of
// three 16-row tiles an SM, each as long as K, but is there sooner; so the line is by its rounds, where this kernel is the
// faster one with the weights cold and with them in L2 (launched one by one, three matrices of 12288 x 5120 in turn: 9.7
// and 10.4).
static bool gemv_tc2_faster(int M, int K, int split) {
    const int sms = device_sms(current_device_index()), tiles = (M + 15) / 16, rounds = (tiles + 3 * sms - 1) / (3 * sms);
    if (K < 12 * TC_BK) return false;
    if (rounds == 1) return tiles > sms && K >= 20 * TC_BK;
    if (rounds == 2) return K >= (split > 2 ? 16 : 24) * TC_BK;
    return rounds > 3 || split > 1;
}
// CTAs that split K, 0 where the other kernel takes the problem
int gemv_tc2_split(int M, int K) {
    if (M <= 0 || K <= 0 || K % TC_BK != 0) return 0;
    const int split = t2_split(M, K);
    return split > 0 && gemv_tc2_faster(M, K, split) ? split : 0;
}

int gemv_tc2_launch(const uint8_t* packed, const uint8_t* scales, const void* act0, const void* act1, bool interleaved,
                    void* out, int M, int K, cudaStream_t st) {
    if (K % TC_BK != 0 || (((uintptr_t)packed | (uintptr_t)scales) & 15) != 0) return NVFP4_ERR_SHAPE;
    const int split = gemv_tc2_split(M, K);
    if (split == 0) return NVFP4_ERR_SHAPE;
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return -3;
    CUtensorMap wm, sm;
    if (!packed_map(enc, &wm, packed, M, K, TC_BM, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) ||
        !scales_map(enc, &sm, scales, M, K, TC_BM))
        return -3;
    const __half* x0 = static_cast<const __half*>(act0);
    const __half* x1 = static_cast<const __half*>(act1);
    const cudaError_t e = interleaved ? t2_launch<true>(wm, sm, packed, scales, x0, x0, static_cast<__half*>(out), M, K, split, st)
                                      : t2_launch<false>(wm, sm, packed, scales, x0, x1, static_cast<__half*>(out), M, K, split, st);
    return (int)e;
}

}  // namespace nvfp4

extern "C" int nvfp4_gemv_tc2_split(int M, int K) { return nvfp4::gemv_tc2_split(M, K); }

namespace nvfp4 {

int gemv_tc2_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_tc2_status, sizeof(int)) != cudaSuccess) return -1;
    if (reset) {
        const int z = 0;
        cudaMemcpyToSymbol(g_tc2_status, &z, sizeof(int));
    }
    return v;
}

}  // namespace nvfp4
