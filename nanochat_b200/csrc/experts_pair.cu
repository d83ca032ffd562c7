// The experts' products for many rows on pairs of CTAs (cta_group::2): tiles of 256 sorted positions by 256 weight rows, the form of
// linear_cap.cu.  A CTA holds its 128 positions and half of the weight rows in shared memory, 32 KB a step of 64 channels where a tile
// of one CTA (experts_tc.cu, 128 x 256) takes 48: those arrived at 64 bytes per SM and cycle, what an SM takes in, so that a step of 512 cycles of
// products took 750.  With UP a pass ahead (expert_gather_kernel) puts the tokens into sorted order; fetched token by token into the swizzled places
// a step took 950 cycles.
//   warp 0      one thread moves both operands by TMA through a ring of six stages; the copies of both CTAs are counted by the even
//               CTA's barrier
//   warp 1      (even CTA) one thread issues the products into one of two accumulators; its commits reach both CTAs
//   warps 2-9   two warps per 32 positions, each with half of the columns: accumulator -> activation and weight (UP) -> turned in shared
//               memory -> 128 bytes of a row by 8 lanes
// With UP the weight rows of a tile are 128 gate rows (even CTA's half) and the 128 up rows of the same channels (odd CTA's).
// Tiles of one expert are consecutive, positions fastest within a group of them (eq_group).  What stands in a tile behind an expert's last position is not stored.
// Every wait is bounded; one that runs out sets NCKV_ST_TIMEOUT, the roles stop, copies in flight are waited for, both CTAs
// leave together and tensor memory is freed.
#include <algorithm>
#include <cmath>

#include "experts.cuh"
#include "tc05.cuh"

namespace nckv {

constexpr int EQ_M = 128, EQ_BN = 256, EQ_K = 64, EQ_STAGES = 6;  // EQ_M: positions per CTA
constexpr int EQ_A_BYTES = EQ_M * EQ_K * 2, EQ_B_BYTES = EQ_BN / 2 * EQ_K * 2, EQ_STAGE = EQ_A_BYTES + EQ_B_BYTES;
constexpr int EQ_OUT_WARPS = 8, EQ_THREADS = 64 + 32 * EQ_OUT_WARPS;
constexpr int EQ_TURN = 32 * 128;  // a warp's 32 rows by 64 results on their way out
constexpr int EQ_SMEM = EQ_STAGES * EQ_STAGE + EQ_OUT_WARPS * EQ_TURN;

__device__ __forceinline__ void tma_load_4d_pair(void *smem_dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(smem_dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}

// Tiles of positions whose rows, 32 MB, stay in L2 while all weights pass by.  16384 rows of 4096 with 2 x 11008 weight rows, all positions to a
// weight tile / in groups: 2884 us / 2143.  An expert with no more tiles than a group, 42 at 1536 channels, has all of them to a weight tile.
__host__ __device__ constexpr int eq_group(int K) { return K <= 65536 ? 65536 / K : 1; }
// One tile, found by walking on from the tile before.
struct EqCursor {
    int e, m_hi, m0, n;
    __device__ __forceinline__ bool seek(const int *s_first, const ExpertParams &p, int n_tiles, int idx) {
        while (e < p.E && idx >= s_first[e + 1] * n_tiles) ++e;
        if (e >= p.E) return false;
        const int tiles = s_first[e + 1] - s_first[e], local = idx - s_first[e] * n_tiles;
        m_hi = p.offsets ? p.offsets[e + 1] : p.R;
        const int most = min(eq_group(p.K), tiles);  // (so its product with n_tiles is not above the number of all tiles)
        const int group = local / (most * n_tiles), in_group = local - group * most * n_tiles;
        const int size = min(most, tiles - group * most);
        n = in_group / size;
        m0 = (p.offsets ? p.offsets[e] : 0) + (group * most + in_group - n * size) * 2 * EQ_M;
        return true;
    }
};

template <bool UP>
__global__ void __launch_bounds__(EQ_THREADS, 1)
experts_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const ExpertParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ int s_first[EQ_MAX_EXPERTS + 1];                    // tiles of positions before expert e
    __shared__ uint64_t bar_full[EQ_STAGES], bar_free[EQ_STAGES];  // a stage's operands landed (even CTA) / were read
    __shared__ uint64_t bar_acc[2], bar_read[2];                   // an accumulator is complete / was read (even CTA)
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int *abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster_rank();
    const bool aligned = (smem_u32(smem) & 1023u) == 0;  // the same in all CTAs; checked rather than assumed
    const int n_tiles = UP ? (p.N + EQ_BN / 2 - 1) / (EQ_BN / 2) : (p.N + EQ_BN - 1) / EQ_BN, k_steps = (p.K + EQ_K - 1) / EQ_K;
    if (warp == 0) {
        tmem_alloc_pair(&tmem_slot, 2 * EQ_BN);
    } else if (warp == 1) {
        int carry = 0;
        for (int e0 = 0; e0 < p.E; e0 += 32) {
            const int e = e0 + lane;
            const int positions = e < p.E ? (p.offsets ? p.offsets[e + 1] - p.offsets[e] : p.R) : 0;
            int inc = (positions + 2 * EQ_M - 1) / (2 * EQ_M);
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += v;
            }
            if (e < p.E) s_first[e + 1] = carry + inc;
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) s_first[0] = 0;
    } else if (tid == 64) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_w);
        for (int i = 0; i < EQ_STAGES; ++i) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_acc[i], 1);
            mbar_init(&bar_read[i], 2 * EQ_OUT_WARPS);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers are ready
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int total = aligned ? s_first[p.E] * n_tiles : 0, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    auto timed_out = [&]() {
        *abort_flag = 1;
        atomicOr(p.status, (int)NCKV_ST_TIMEOUT);
    };
    if (!aligned && tid == 0) timed_out();

    EqCursor cur;
    cur.e = 0;
    if (warp == 0) {
        // =============== operands ===================================================================
        if (elect_one()) {
            uint32_t fill = 0;
            bool ok = true;
            auto freed = [&](uint32_t f) -> bool { return mbar_wait_bounded(&bar_free[f % EQ_STAGES], (f / EQ_STAGES) & 1u); };
            for (int idx = pair; idx < total && ok; idx += pairs) {
                if (!cur.seek(s_first, p, n_tiles, idx)) break;
                for (int ks = 0; ks < k_steps; ++ks, ++fill) {
                    const uint32_t st = fill % EQ_STAGES;
                    if (fill >= EQ_STAGES && (*abort_flag != 0 || !freed(fill - EQ_STAGES))) {
                        ok = false;
                        break;
                    }
                    uint8_t *a = smem + st * EQ_STAGE;
                    const uint32_t full = smem_of_rank(&bar_full[st], 0);
                    if (rank == 0) mbar_arrive_expect_tx(&bar_full[st], 2 * EQ_STAGE);
                    tma_load_2d_pair(a, &map_a, full, ks * EQ_K, cur.m0 + rank * EQ_M);
                    if (UP) tma_load_4d_pair(a + EQ_A_BYTES, &map_w, full, ks * EQ_K, cur.n * (EQ_BN / 2), rank, cur.e);
                    else tma_load_4d_pair(a + EQ_A_BYTES, &map_w, full, ks * EQ_K, cur.n * EQ_BN + rank * (EQ_BN / 2), 0, cur.e);
                }
            }
            if (ok)  // the issuer's commits reach both CTAs: all of them before either leaves
                for (uint32_t f = fill > EQ_STAGES ? fill - EQ_STAGES : 0; f < fill && ok; ++f) ok = freed(f);
            if (!ok) {
                timed_out();
                // copies already issued land before the CTA's memory is released (the even CTA's barrier counts for
                // both, and both leave together)
                if (rank == 0)
                    for (uint32_t f = fill > EQ_STAGES ? fill - EQ_STAGES : 0; f < fill; ++f)
                        mbar_wait_bounded(&bar_full[f % EQ_STAGES], (f / EQ_STAGES) & 1u, 100000000ull);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // =============== products ===================================================================
        if (rank == 0 && elect_one()) {
            constexpr uint32_t IDESC = umma_idesc(2 * EQ_M, EQ_BN, 0, 0);
            const uint64_t desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
            uint32_t fill = 0, tile = 0;
            bool ok = true;
            for (int idx = pair; idx < total && ok; idx += pairs, ++tile) {
                const uint32_t buf = tile & 1u, use = tile >> 1;
                if (use > 0 && !mbar_wait_bounded(&bar_read[buf], (use - 1) & 1u)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + buf * EQ_BN;
                for (int ks = 0; ks < k_steps; ++ks, ++fill) {
                    const uint32_t st = fill % EQ_STAGES;
                    if (*abort_flag != 0 || !mbar_wait_bounded(&bar_full[st], (fill / EQ_STAGES) & 1u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = desc0 + (uint64_t)((st * EQ_STAGE) >> 4), db = da + (uint64_t)(EQ_A_BYTES >> 4);
#pragma unroll
                    for (int kk = 0; kk < EQ_K / 16; ++kk)
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
        constexpr int COLS = UP ? EQ_BN / 4 : EQ_BN / 2;  // results of a warp's rows
        const int q = warp & 3, part = (warp - 2) >> 2;   // a warp reaches tensor-memory lanes 32 (warp % 4) ..
        uint8_t *turn = smem + EQ_STAGES * EQ_STAGE + (warp - 2) * EQ_TURN;
        const bool vec = p.N % 8 == 0 && (((uintptr_t)p.out) & 15) == 0;
        auto warp_wait = [&](uint64_t *bar, uint32_t parity) -> bool {
            if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
            int ok = 1;
            if (lane == 0) ok = *abort_flag == 0 && mbar_wait_bounded(bar, parity) ? 1 : 0;
            return __shfl_sync(0xffffffffu, ok, 0) != 0;
        };
        uint32_t tile = 0;
        for (int idx = pair; idx < total; idx += pairs, ++tile) {
            if (!cur.seek(s_first, p, n_tiles, idx)) break;
            const int m = cur.m0 + rank * EQ_M + q * 32 + lane;
            const bool have = m < cur.m_hi;
            const float s = UP && have ? (p.scale ? p.scale[m] : 1.f) : 0.f;
            const int to = UP ? m : (have ? p.slot[m] : 0);  // this row's place in out
            const int n0 = cur.n * (UP ? EQ_BN / 2 : EQ_BN);
            const uint32_t buf = tile & 1u;
            if (!warp_wait(&bar_acc[buf], (tile >> 1) & 1u)) {
                if (lane == 0 && *abort_flag == 0) timed_out();
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + buf * EQ_BN + ((uint32_t)(q * 32) << 16);
            // 64 results of the warp's 32 rows at a time, turned in shared memory (16-byte pieces, swizzled by row)
#pragma unroll 1
            for (int c = part * COLS; c < (part + 1) * COLS; c += 64) {
                if (n0 + c >= p.N || !__any_sync(0xffffffffu, have)) break;  // uniform over the warp
#pragma unroll
                for (int half = 0; half < 64; half += 32) {
                    float v[32];
                    if (UP) {
                        float u[32];
                        tmem_ld32x2(acc + c + half, v, acc + EQ_BN / 2 + c + half, u);
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = Fn<__nv_bfloat16>::silu(s * v[i]) * (s * u[i]);
                    } else {
                        tmem_ld32(acc + c + half, v);
                    }
#pragma unroll
                    for (int i = 0; i < 32; i += 8)
                        *reinterpret_cast<uint4 *>(turn + lane * 128 + ((((half + i) / 8) ^ (lane & 7)) << 4)) =
                            make_uint4(pack_bf16x2(v[i], v[i + 1]), pack_bf16x2(v[i + 2], v[i + 3]), pack_bf16x2(v[i + 4], v[i + 5]),
                                       pack_bf16x2(v[i + 6], v[i + 7]));
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = i * 4 + (lane >> 3), n = n0 + c + (lane & 7) * 8;
                    const int place = __shfl_sync(0xffffffffu, have ? to : -1, r);
                    const uint4 w = *reinterpret_cast<const uint4 *>(turn + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
                    if (place < 0) continue;
                    __nv_bfloat16 *dst = static_cast<__nv_bfloat16 *>(p.out) + (long long)place * p.N + n;
                    if (vec) {
                        if (n < p.N) *reinterpret_cast<uint4 *>(dst) = w;
                    } else {
                        const uint32_t e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            if (n + k < p.N) *reinterpret_cast<uint16_t *>(dst + k) = (uint16_t)(e[k >> 1] >> ((k & 1) * 16));
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
    if (warp == 0) tmem_dealloc_pair(tmem, 2 * EQ_BN);
}

// to[i] = the token of sorted position i, a warp each
__global__ void __launch_bounds__(256) expert_gather_kernel(const uint4 *h, const int32_t *slot, uint4 *to, int R, int top, int per_row) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= R) return;
    const uint4 *from = h + (long long)(slot[i] / top) * per_row;
    uint4 *dst = to + (long long)i * per_row;
    constexpr int AHEAD = 8;
    for (int c = threadIdx.x & 31; c < per_row; c += 32 * AHEAD) {
        uint4 v[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (c + 32 * k < per_row) v[k] = from[c + 32 * k];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (c + 32 * k < per_row) dst[c + 32 * k] = v[k];
    }
}

template <bool UP> static cudaError_t eq_launch(const ExpertParams &p, cudaStream_t s, int *rc) {
    CUtensorMap ma, mw;
    {
        const int64_t dims[2] = {p.K, p.R}, strides[1] = {p.K};
        const int box[2] = {EQ_K, EQ_M};
        *rc = make_tensor_map(&ma, p.a, 2, dims, strides, box);
    }
    if (*rc != NCKV_OK) return cudaSuccess;
    const int64_t N = p.N, K = p.K, halves = UP ? 2 : 1;
    const int64_t dims[4] = {K, N, halves, p.E}, strides[3] = {K, N * K, halves * N * K};
    const int box[4] = {EQ_K, EQ_BN / 2, 1, 1};
    *rc = make_tensor_map(&mw, p.w, 4, dims, strides, box);
    if (*rc != NCKV_OK) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(experts_pair_kernel<UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, EQ_SMEM);
    if (e != cudaSuccess) return e;
    const long long tiles = ((long long)p.R / (2 * EQ_M) + p.E) * ((p.N + EQ_BN / halves - 1) / (EQ_BN / halves));
    const int most = sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * (tiles < most ? (int)tiles : most)));
    cfg.blockDim = dim3(EQ_THREADS);
    cfg.dynamicSmemBytes = EQ_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, experts_pair_kernel<UP>, ma, mw, p);
}

// By the rounds of tiles that either form needs at an even spread of the positions, each expert with one tile at least.  A round of pairs takes 64
// (up) or 82 percent of the time of a wave of the other form's wide tiles, which is 0.62 us a step, a wave of its narrow tiles 80; the gather
// reads and writes at 5 TB/s behind a launch.  With up to 256 positions an expert the down product waits for its weights in either form.
// us, 16 experts, 4 a token, other form / pairs, B200: 1536 x 1024 up 6007 tokens 153.6 / 117.7, 16384 385 / 308, 1024 73.7 / 48.1, 384
// 43.0 / 40.0, and the other way 1500 57.4 / 58.4, 256 34.8 / 39.9; down 6007 68.4 / 60.3, 1500 35.8 / 32.8, 1024 30.7 / 32.8; 2048 x
// 1376 up 6007 251.9 / 199.7, 512 59.4 / 62.5, down 118.8 / 100.4, 1500 49.2 / 51.2.  The bits are the same.
// The results of a tile of the down product take the time of some ten steps, in either form: with fewer steps they are the bound, and the other form's
// tiles, half as large, fill the chip better.  us, other form / pairs: 512 channels, 16 experts, 1536 results 17584 positions 32.5 / 37.2, 41848 64.1 / 66.5;
// 8 experts, 2048 results 2894 positions 13.6 / 14.9; 640 channels, 64 experts, 1024 results 21872 positions 42.5 / 45.0; 768 channels, 16 experts, 2048
// results 12064 positions 48.9 / 45.3.  Of 35 sizes of up to 640 channels pairs lost in 28, of 110 of more in 9.
constexpr int EQ_SHORT = 10;
bool experts_in_pairs(bool up, int R, int E, int N, int K) {
    const int per = up ? EQ_BN / 2 : EQ_BN, steps = (K + EQ_K - 1) / EQ_K;
    if (E > EQ_MAX_EXPERTS || (!up && (R <= 256LL * E || steps <= EQ_SHORT))) return false;
    const double m_tiles = std::max(R / (2. * EQ_M) + E / 2., (double)std::min(R, E));
    const double rounds = std::ceil(m_tiles * ((N + per - 1) / per) / (sm_count() / 2));
    const double pairs = up ? 64 * rounds + 100 * (8e-7 * R * K + 2) / (0.62 * steps) : 82 * rounds;
    return pairs < 97. / 100 * (experts_tc_wide(up, R, E, N) ? 100 * experts_tc_waves(up, R, E, N, 256) : 80 * experts_tc_waves(up, R, E, N, 128));
}

cudaError_t experts_pair(ExpertParams p, bool up, void *sorted, cudaStream_t s, int *rc) {
    if (!up) return eq_launch<false>(p, s, rc);
    const int per_row = p.K / 8;
    expert_gather_kernel<<<(unsigned)((p.R + 7) / 8), 256, 0, s>>>(static_cast<const uint4 *>(p.a), p.slot, static_cast<uint4 *>(sorted), p.R,
                                                                 p.top, per_row);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    p.a = sorted;
    return eq_launch<true>(p, s, rc);
}

}  // namespace nckv

// The feed-forward's gate and up product with its activation: the up form with one expert that has all rows, in their order (which sizes pay is the
// caller's rule, gate_up_in_one).  Against the
// library's product and an activation that reads its result (two halves, rounded between), B200, us: 1536 x 4096, 16384 rows 334 / 266, 4096 89 /
// 68, 1024 25.4 / 21.4, 640 19.7 / 20.8, 300 11.4 / 14.0; 2048 x 5504, 16384 rows 575 / 483, 2048 79 / 64, 1024 41.9 / 36.3, 512 23.7 / 26.1;
// 1024 x 2752, 4096 rows 52.6 / 33.3, 1024 15.7 / 16.2; 512 x 1024, 4096 rows 15.7 / 12.4, 2048 10.2 / 9.0, 1024 7.4 / 8.5; 256 x 512, 4096 rows 9.9
// / 7.6, 1536 7.0 / 7.2.  Error against 64 bits, relative: 3.1e-3 / 1.7e-3, one rounding instead of three.
extern "C" int nckv_gate_up(const void *h, const void *w, void *out, int rows, int N, int K, int32_t *status, void *stream) {
    using namespace nckv;
    if (!h || !w || !out || !status) {
        set_error("gate_up: null pointer argument");
        return NCKV_E_ARG;
    }
    if (rows <= 0 || N <= 0 || K <= 0 || K % 8 || (((uintptr_t)h | (uintptr_t)w) & 15) ||
        ((long long)rows / (2 * EQ_M) + 1) * ((N + EQ_BN / 2 - 1) / (EQ_BN / 2)) > 0x7fffffffLL) {
        set_error("gate_up: size or alignment out of range (rows=%d N=%d K=%d)", rows, N, K);
        return NCKV_E_ARG;
    }
    ExpertParams p = {};
    p.a = h; p.w = w; p.out = out; p.status = status;
    p.R = rows; p.E = p.top = 1; p.N = N; p.K = K;
    int rc = NCKV_OK;
    NCKV_CUDA_CHECK(eq_launch<true>(p, static_cast<cudaStream_t>(stream), &rc));
    return rc;
}
