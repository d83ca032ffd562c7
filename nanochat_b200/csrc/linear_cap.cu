// Soft-capped logits of many rows: out[r, n] = cap * tanh(sum_k x[r, k] w[n, k] / cap), bf16 operands, fp32 sums and results.
//
// The logits are the largest tensor of a forward pass (2.1 GB for 16384 tokens of 32768 words).  As a product and a
// pass over its result they cross memory three times, and the second pass alone took 731 us; here the cap is applied to
// the accumulators on their way out of tensor memory, beside the next tile's products.
//
// A pair of CTAs (cta_group::2) works on a tile of 256 rows by 256 words, each holding its 128 rows and half of the
// words in shared memory: 64 bytes of operands per SM and cycle instead of the 96 that a CTA with a 128 x 256 tile of
// its own needs.  Pairs are persistent, one per two SMs.  Roles, connected by mbarriers:
//   warp 0      one thread moves both operands by TMA, 64 channels a step, through a ring of six stages; the copies of
//               both CTAs are counted by the even CTA's barrier
//   warp 1      (even CTA) one thread issues the products into one of two accumulators; its commits reach both CTAs
//   warps 2-9   two warps per 32 rows, each with half of the words: accumulator -> cap -> turned in shared memory ->
//               128 bytes of a row by 8 lanes
// Tiles run through the rows first: a group of LC_GROUP word tiles stays in L2 while all rows pass.
// 16384 rows of 1536 by 32768 words: 1302 us where product and pass take 1957 (the product alone 1289); which sizes pay is the
// caller's rule (cap_in_product).  Bound: the tensor pipe (80 percent of its cycles busy, by ncu) under the power limit; the caps of a tile
// take 7.6 us beside it.  With a division for each value they took 11 and were the bound (1526 us; 4096 rows 373, now 299; 2048 rows
// of 2048 226, now 186; 1000 rows 120, now 101).  A shorter tanh gave 2 percent at a third less accuracy.
// Every wait is bounded; one that runs out sets NCKV_ST_TIMEOUT, the roles stop, copies in flight are waited for, both
// CTAs leave together and tensor memory is freed.
#include "nckv_common.cuh"
#include "tc05.cuh"

namespace nckv {

constexpr int LC_M = 128, LC_BN = 256, LC_K = 64, LC_STAGES = 6;  // LC_M: rows per CTA
constexpr int LC_A_BYTES = LC_M * LC_K * 2, LC_B_BYTES = LC_BN / 2 * LC_K * 2, LC_STAGE = LC_A_BYTES + LC_B_BYTES;
constexpr int LC_OUT_WARPS = 8, LC_THREADS = 64 + 32 * LC_OUT_WARPS;
constexpr int LC_TURN = 32 * 128;  // a warp's 32 rows by 32 results on their way out
constexpr int LC_SMEM = LC_STAGES * LC_STAGE + LC_OUT_WARPS * LC_TURN;
constexpr int LC_GROUP = 8;        // word tiles (256 words) that all rows pass together

struct LinearCapParams {
    float *out;
    int32_t *status;
    float cap;
    int R, N, K;
};

// v / cap for two values, correctly rounded (to the bits of the division) where quotient and residue are normal numbers: the product with
// the rounded reciprocal, corrected twice by its exact residue (Markstein's method; a uniform divisor leaves 2.5 instructions a value where
// a division takes about ten and a check).  Values beyond 16 caps count as 16 caps, whose tanh is 1 too, so that an infinite one
// leaves a quotient; what is no number stays none.  (-0 would leave +0; a sum of products, which starts from +0, is never -0.)
struct CapQuotient {
    float2 neg_cap, rcp;
    float most;
    __device__ __forceinline__ explicit CapQuotient(float cap)
        : neg_cap(make_float2(-cap, -cap)), rcp(make_float2(1.f / cap, 1.f / cap)), most(16.f * cap) {}
    __device__ __forceinline__ float within(float v) const {  // |most| > 0: the sign is v's
        float r;
        asm("min.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "f"(most));
        return r;
    }
    __device__ __forceinline__ float2 operator()(float v0, float v1) const {
        const float2 v = make_float2(within(v0), within(v1));
        float2 q = fmul2(v, rcp);
        q = ffma2(ffma2(neg_cap, q, v), rcp, q);
        return ffma2(ffma2(neg_cap, q, v), rcp, q);
    }
};

// QUOTIENT: the cap is far from the ends of the numbers, where its reciprocal and the residues are exact enough; else plain divisions.
template <bool QUOTIENT>
__global__ void __launch_bounds__(LC_THREADS, 1) linear_cap_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                   const LinearCapParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bar_full[LC_STAGES], bar_free[LC_STAGES];  // a stage's operands landed (even CTA) / were read
    __shared__ uint64_t bar_acc[2], bar_read[2];                    // an accumulator is complete / was read (even CTA)
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int *abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster_rank();
    const bool aligned = (smem_u32(smem) & 1023u) == 0;  // the same in all CTAs; checked rather than assumed
    if (warp == 0) {
        tmem_alloc_pair(&tmem_slot, 2 * LC_BN);
    } else if (tid == 32) {
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_w);
        for (int i = 0; i < LC_STAGES; ++i) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_acc[i], 1);
            mbar_init(&bar_read[i], 2 * LC_OUT_WARPS);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers are ready
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int m_tiles = (p.R + 2 * LC_M - 1) / (2 * LC_M), n_tiles = (p.N + LC_BN - 1) / LC_BN, k_steps = (p.K + LC_K - 1) / LC_K;
    const int total = aligned ? m_tiles * n_tiles : 0;
    auto tile_at = [&](int idx, int &m0, int &n0) {  // this CTA's first row, the tile's first word
        const int per_group = LC_GROUP * m_tiles, grp = idx / per_group, in = idx - grp * per_group;
        const int width = min(LC_GROUP, n_tiles - grp * LC_GROUP), m = in / width;
        m0 = m * 2 * LC_M + rank * LC_M;
        n0 = (grp * LC_GROUP + in - m * width) * LC_BN;
    };
    auto timed_out = [&]() {
        *abort_flag = 1;
        atomicOr(p.status, (int)NCKV_ST_TIMEOUT);
    };
    if (!aligned && tid == 0) timed_out();

    if (warp == 0) {
        // =============== operands ===================================================================
        if (elect_one()) {
            uint32_t fill = 0;
            bool ok = true;
            auto freed = [&](uint32_t f) -> bool { return mbar_wait_bounded(&bar_free[f % LC_STAGES], (f / LC_STAGES) & 1u); };
            for (int idx = blockIdx.x >> 1; idx < total && ok; idx += gridDim.x >> 1) {
                int m0, n0;
                tile_at(idx, m0, n0);
                for (int ks = 0; ks < k_steps; ++ks, ++fill) {
                    const uint32_t st = fill % LC_STAGES;
                    if (fill >= LC_STAGES && (*abort_flag != 0 || !freed(fill - LC_STAGES))) {
                        ok = false;
                        break;
                    }
                    uint8_t *a = smem + st * LC_STAGE;
                    const uint32_t full = smem_of_rank(&bar_full[st], 0);
                    if (rank == 0) mbar_arrive_expect_tx(&bar_full[st], 2 * LC_STAGE);
                    tma_load_2d_pair(a, &map_x, full, ks * LC_K, m0);
                    tma_load_2d_pair(a + LC_A_BYTES, &map_w, full, ks * LC_K, n0 + rank * (LC_BN / 2));
                }
            }
            if (ok)  // the issuer's commits reach both CTAs: all of them before either leaves
                for (uint32_t f = fill > LC_STAGES ? fill - LC_STAGES : 0; f < fill && ok; ++f) ok = freed(f);
            if (!ok) {
                timed_out();
                // copies already issued land before the CTA's memory is released (the even CTA's barrier counts for
                // both, and both leave together)
                if (rank == 0)
                    for (uint32_t f = fill > LC_STAGES ? fill - LC_STAGES : 0; f < fill; ++f)
                        mbar_wait_bounded(&bar_full[f % LC_STAGES], (f / LC_STAGES) & 1u, 100000000ull);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // =============== products ===================================================================
        if (rank == 0 && elect_one()) {
            constexpr uint32_t IDESC = umma_idesc(2 * LC_M, LC_BN, 0, 0);
            const uint64_t desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
            uint32_t fill = 0, tile = 0;
            bool ok = true;
            for (int idx = blockIdx.x >> 1; idx < total && ok; idx += gridDim.x >> 1, ++tile) {
                const uint32_t buf = tile & 1u, use = tile >> 1;
                if (use > 0 && !mbar_wait_bounded(&bar_read[buf], (use - 1) & 1u)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + buf * LC_BN;
                for (int ks = 0; ks < k_steps; ++ks, ++fill) {
                    const uint32_t st = fill % LC_STAGES;
                    if (*abort_flag != 0 || !mbar_wait_bounded(&bar_full[st], (fill / LC_STAGES) & 1u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = desc0 + (uint64_t)((st * LC_STAGE) >> 4), db = da + (uint64_t)(LC_A_BYTES >> 4);
#pragma unroll
                    for (int kk = 0; kk < LC_K / 16; ++kk)
                        umma_bf16_pair(d, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), IDESC, ks > 0 || kk > 0 ? 1u : 0u);
                    umma_commit_pair(&bar_free[st]);
                }
                if (ok) umma_commit_pair(&bar_acc[buf]);
            }
            if (!ok) timed_out();
        }
        __syncwarp();
    } else {
        // =============== results ====================================================================
        const int q = warp & 3, part = (warp - 2) >> 2;  // a warp reaches tensor-memory lanes 32 (warp % 4) ..
        uint8_t *turn = smem + LC_STAGES * LC_STAGE + (warp - 2) * LC_TURN;
        const bool vec = p.N % 4 == 0;
        const CapQuotient quotient(p.cap);
        auto warp_wait = [&](uint64_t *bar, uint32_t parity) -> bool {
            if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
            int ok = 1;
            if (lane == 0) ok = *abort_flag == 0 && mbar_wait_bounded(bar, parity) ? 1 : 0;
            return __shfl_sync(0xffffffffu, ok, 0) != 0;
        };
        uint32_t tile = 0;
        for (int idx = blockIdx.x >> 1; idx < total; idx += gridDim.x >> 1, ++tile) {
            int m0, n0;
            tile_at(idx, m0, n0);
            const uint32_t buf = tile & 1u;
            if (!warp_wait(&bar_acc[buf], (tile >> 1) & 1u)) {
                if (lane == 0 && *abort_flag == 0) timed_out();
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + buf * LC_BN + ((uint32_t)(q * 32) << 16);
            const int row0 = m0 + q * 32;
#pragma unroll 1
            for (int c = part * (LC_BN / 2); c < (part + 1) * (LC_BN / 2); c += 32) {
                if (n0 + c >= p.N || row0 >= p.R) break;  // uniform over the warp
                float v[32];
                tmem_ld32(acc + (uint32_t)c, v);
                if (row0 + lane < p.R) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float2 x = QUOTIENT ? quotient(v[i], v[i + 1]) : make_float2(v[i] / p.cap, v[i + 1] / p.cap);
                        const float2 y = QUOTIENT ? quotient(v[i + 2], v[i + 3]) : make_float2(v[i + 2] / p.cap, v[i + 3] / p.cap);
                        *reinterpret_cast<float4 *>(turn + lane * 128 + (((i / 4) ^ (lane & 7)) << 4)) =
                            make_float4(p.cap * tanhf(x.x), p.cap * tanhf(x.y), p.cap * tanhf(y.x), p.cap * tanhf(y.y));
                    }
                }
                __syncwarp();
                const int n = n0 + c + (lane & 7) * 4;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = i * 4 + (lane >> 3);
                    const float4 w = *reinterpret_cast<const float4 *>(turn + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
                    if (row0 + r >= p.R) continue;
                    float *dst = p.out + (long long)(row0 + r) * p.N + n;
                    if (vec) {
                        if (n < p.N) *reinterpret_cast<float4 *>(dst) = w;
                    } else {
                        const float e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (n + k < p.N) dst[k] = e[k];
                    }
                }
                __syncwarp();  // read, before the next results are put there
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(smem_of_rank(&bar_read[buf], 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // nothing of either CTA reaches for the other's memory any more
    if (warp == 0) tmem_dealloc_pair(tmem, 2 * LC_BN);
}

}  // namespace nckv

extern "C" int nckv_linear_cap(const void *x, const void *w, float *out, int R, int N, int K, float cap, int32_t *status, void *stream) {
    using namespace nckv;
    if (!x || !w || !out || !status || !(cap > 0.f)) {
        set_error("linear_cap: null pointer argument or cap not positive");
        return NCKV_E_ARG;
    }
    if (R <= 0 || N <= 0 || K <= 0) {
        set_error("linear_cap: size out of range (R=%d N=%d K=%d)", R, N, K);
        return NCKV_E_ARG;
    }
    const long long tiles = ((long long)R + 2 * LC_M - 1) / (2 * LC_M) * (((long long)N + LC_BN - 1) / LC_BN);
    if (K % 8 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) || tiles > 0x3fffffffLL) {
        set_error("linear_cap: R=%d N=%d K=%d unsupported (rows of whole, aligned 16-byte pieces)", R, N, K);
        return NCKV_E_UNSUPPORTED;
    }
    CUtensorMap mx, mw;
    {
        const int64_t dims[2] = {K, R}, strides[1] = {K};
        const int box[2] = {LC_K, LC_M};
        const int rc = make_tensor_map(&mx, x, 2, dims, strides, box);
        if (rc != NCKV_OK) return rc;
    }
    {
        const int64_t dims[2] = {K, N}, strides[1] = {K};
        const int box[2] = {LC_K, LC_BN / 2};
        const int rc = make_tensor_map(&mw, w, 2, dims, strides, box);
        if (rc != NCKV_OK) return rc;
    }
    LinearCapParams p;
    p.out = out; p.status = status; p.cap = cap;
    p.R = R; p.N = N; p.K = K;
    const auto kernel = cap >= 0x1p-60f && cap <= 0x1p60f ? linear_cap_kernel<true> : linear_cap_kernel<false>;
    NCKV_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LC_SMEM));
    const int most = sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * (tiles < most ? (int)tiles : most)));
    cfg.blockDim = dim3(LC_THREADS);
    cfg.dynamicSmemBytes = LC_SMEM;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NCKV_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, mx, mw, p));
    return NCKV_OK;
}
