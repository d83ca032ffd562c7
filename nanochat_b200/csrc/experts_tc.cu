// The experts' products for many rows, on the tensor cores (tcgen05, accumulators in tensor memory).  The largest take the form on pairs of
// CTAs (experts_pair.cu).
//
// Persistent CTAs, one per SM, walk over the tiles of all experts: 128 of an expert's sorted positions by BN
// weight rows (UP: BN / 2 gate and the BN / 2 up rows of the same channels, so that a thread holds both
// factors of an output).  A tile's K runs in steps of 64 through a ring in shared memory (128-byte
// swizzle).  Roles, connected by mbarriers:
//   warp 0      moves the weights, and without UP the positions (rows of act), by TMA
//   warps 6-13  UP: the tokens of a tile lie anywhere in h; these warps fetch them with 16-byte asynchronous copies
//               into the place the swizzle gives them, so h is never copied into sorted order (a gather by
//               TMA, four rows per instruction, was three times slower than the products).  A group of warps takes a
//               step at a time and waits for its own copies.  With four stages (wide tiles) four groups of two: four
//               steps are on their way at any time (two groups that handed a step over behind the next one's request
//               had two: 178 us at 6007 tokens x 4 of 16 experts of 1536 x 1024, now 154).  With six stages (narrow
//               tiles) two groups of four, two steps on their way: handed over two of its own steps later, which has
//               six, a step took longer: 25.6 against 29.0 us at 32 tokens, 41.5 / 43.7 at 512, 60.5 / 66.3 at 1024,
//               104 / 112 at 2300.
//   warp 1      one thread issues the products into one of two accumulators
//   warps 2-5   one thread per position reads the other accumulator, applies the router's weight and the
//               activation (UP) or finds the pair's place (down); results are turned in shared memory and stored 128
//               bytes of a row by 8 lanes (16 bytes of 32 rows per instruction held up the operands of the next
//               tile's products: down 83 us, now 69)
// Tiles of one expert are consecutive, positions fastest: the CTAs that run side by side share weights and rows
// in L2.  What stands in a tile behind an expert's last position is not stored.  Every wait is bounded; one that
// runs out sets NCKV_ST_TIMEOUT, the roles stop, copies in flight are waited for and tensor memory is freed.
#include "experts.cuh"
#include "tc05.cuh"

namespace nckv {

constexpr int ET_M = 128, ET_K = 64;
constexpr int ET_THREADS = 192, ET_GATHER = 256;  // UP has ET_GATHER more, in two halves
template <int STAGES> constexpr int ET_GROUPS = STAGES == 4 ? 4 : 2;  // groups of warps that fetch tokens: a divisor of the stages
constexpr int ET_MAX_EXPERTS = 1024;
constexpr int ET_A_BYTES = ET_M * ET_K * 2;
constexpr int ET_OUT_BYTES = 4 * 32 * 128;  // a warp's 32 rows by 64 results on their way out

template <int BN> struct EtShape {
    static constexpr int B_BYTES = BN * ET_K * 2, STAGE = ET_A_BYTES + B_BYTES;
    static constexpr int STAGES = BN == 256 ? 4 : 6;
    static constexpr int SMEM = STAGES * STAGE + ET_OUT_BYTES + 256;
};

// One tile, found by walking on from the tile before.
struct EtCursor {
    int e, m_lo, m_hi, m0, n;
    __device__ __forceinline__ bool seek(const int *s_first, const ExpertParams &p, int n_tiles, int idx) {
        while (e < p.E && idx >= s_first[e + 1] * n_tiles) ++e;
        if (e >= p.E) return false;
        const int tiles = s_first[e + 1] - s_first[e], local = idx - s_first[e] * n_tiles;
        m_lo = p.offsets[e];
        m_hi = p.offsets[e + 1];
        n = local / tiles;
        m0 = m_lo + (local - n * tiles) * ET_M;
        return true;
    }
};

template <bool UP, int BN>
__global__ void __launch_bounds__(ET_THREADS + (UP ? ET_GATHER : 0), 1)
experts_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const ExpertParams p) {
    using Shape = EtShape<BN>;
    constexpr int STAGES = Shape::STAGES;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ int s_first[ET_MAX_EXPERTS + 1];  // token tiles before expert e
    if ((smem_u32(smem) & 1023u) != 0) {         // uniform; checked rather than assumed
        if (threadIdx.x == 0) atomicOr(p.status, (int)NCKV_ST_TIMEOUT);
        return;
    }
    uint8_t *s_out = smem + STAGES * Shape::STAGE;
    uint64_t *bars = reinterpret_cast<uint64_t *>(s_out + ET_OUT_BYTES);
    uint64_t *bar_full = bars, *bar_free = bars + STAGES;                         // a stage's operands landed / were read
    uint64_t *bar_acc = bars + 2 * STAGES, *bar_read = bars + 2 * STAGES + 2;     // an accumulator is complete / was read
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_tiles = UP ? (p.N + BN / 2 - 1) / (BN / 2) : (p.N + BN - 1) / BN, k_steps = (p.K + ET_K - 1) / ET_K;
    if (warp == 0) {
        tmem_alloc(tmem_slot, 2 * BN);
        tmem_relinquish();
    } else if (warp == 1) {
        int carry = 0;
        for (int e0 = 0; e0 < p.E; e0 += 32) {
            const int e = e0 + lane;
            const int t = e < p.E ? (p.offsets[e + 1] - p.offsets[e] + ET_M - 1) / ET_M : 0;
            int inc = t;
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
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&bar_full[i], UP ? 1 + ET_GATHER / 32 / ET_GROUPS<STAGES> : 1);
            mbar_init(&bar_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_acc[i], 1);
            mbar_init(&bar_read[i], 4);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int total = s_first[p.E] * n_tiles;
    auto timed_out = [&]() {
        *abort_flag = 1;
        atomicOr(p.status, (int)NCKV_ST_TIMEOUT);
    };
    auto warp_wait = [&](uint64_t *bar, uint32_t parity) -> bool {  // one lane polls
        int ok = 1;
        if (lane == 0) ok = *abort_flag == 0 && mbar_wait_bounded(bar, parity) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();
        return ok != 0;
    };

    EtCursor cur;
    cur.e = 0;
    if (warp == 0) {
        // =============== operands ===================================================================
        if (elect_one()) {
            uint32_t fill = 0;  // number of the fill: stage fill % STAGES
            bool ok = true;
            auto freed = [&](uint32_t f) -> bool { return mbar_wait_bounded(&bar_free[f % STAGES], (f / STAGES) & 1u); };
            for (int idx = blockIdx.x; idx < total && ok; idx += gridDim.x) {
                if (!cur.seek(s_first, p, n_tiles, idx)) break;
                for (int ks = 0; ks < k_steps; ++ks, ++fill) {
                    const uint32_t st = fill % STAGES;
                    if (fill >= STAGES && (*abort_flag != 0 || !freed(fill - STAGES))) {
                        ok = false;
                        break;
                    }
                    uint8_t *a = smem + st * Shape::STAGE, *b = a + ET_A_BYTES;
                    mbar_arrive_expect_tx(&bar_full[st], UP ? Shape::B_BYTES : Shape::STAGE);
                    if (UP) {
                        tma_load_4d(b, &map_w, &bar_full[st], ks * ET_K, cur.n * (BN / 2), 0, cur.e);
                        tma_load_4d(b + Shape::B_BYTES / 2, &map_w, &bar_full[st], ks * ET_K, cur.n * (BN / 2), 1, cur.e);
                    } else {
                        tma_load_2d(a, &map_a, &bar_full[st], ks * ET_K, cur.m0);
                        tma_load_4d(b, &map_w, &bar_full[st], ks * ET_K, cur.n * BN, 0, cur.e);
                    }
                }
            }
            if (!ok) {
                timed_out();
                // copies already issued land before the CTA's memory is released
                for (uint32_t f = fill > STAGES ? fill - STAGES : 0; f < fill; ++f)
                    mbar_wait_bounded(&bar_full[f % STAGES], (f / STAGES) & 1u, 100000000ull);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // =============== products ===================================================================
        if (elect_one()) {
            constexpr uint32_t IDESC = umma_idesc(ET_M, BN, 0, 0);
            const uint64_t desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
            uint32_t fill = 0, tile = 0;
            bool ok = true;
            for (int idx = blockIdx.x; idx < total && ok; idx += gridDim.x, ++tile) {
                const uint32_t buf = tile & 1u, use = tile >> 1;
                if (use > 0 && !mbar_wait_bounded(&bar_read[buf], (use - 1) & 1u)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + buf * BN;
                for (int ks = 0; ks < k_steps; ++ks, ++fill) {
                    const uint32_t st = fill % STAGES;
                    if (*abort_flag != 0 || !mbar_wait_bounded(&bar_full[st], (fill / STAGES) & 1u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = desc0 + (uint64_t)((st * Shape::STAGE) >> 4), db = da + (uint64_t)(ET_A_BYTES >> 4);
#pragma unroll
                    for (int kk = 0; kk < ET_K / 16; ++kk)
                        umma_bf16(d, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), IDESC, ks > 0 || kk > 0 ? 1u : 0u);
                    umma_commit(&bar_free[st]);
                }
                if (ok) umma_commit(&bar_acc[buf]);
            }
            if (!ok) timed_out();
        }
        __syncwarp();
    } else if (UP && warp >= 6) {
        // =============== tokens =====================================================================
        // 8 threads fetch the 128 bytes a token has in a step.  Each group of warps takes every GROUPS-th step and waits
        // for its copies, so as many steps are on their way as there are groups.
        constexpr int GROUPS = ET_GROUPS<STAGES>, GT = ET_GATHER / GROUPS, PER = ET_M * 8 / GT, ROWS = GT / 8;
        const uint32_t group = (uint32_t)(tid - ET_THREADS) / GT;
        const int pt = (tid - ET_THREADS) % GT, chunk = pt & 7, r0 = pt >> 3;
        uint32_t fill = 0;
        bool ok = true;
        for (int idx = blockIdx.x; idx < total && ok; idx += gridDim.x) {
            if (!cur.seek(s_first, p, n_tiles, idx)) break;
            const __nv_bfloat16 *src[PER];
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int m = cur.m0 + r0 + ROWS * i;  // nobody reads the results of rows behind the expert's last
                src[i] = m < cur.m_hi ? static_cast<const __nv_bfloat16 *>(p.a) + (long long)(p.slot[m] / p.top) * p.K + chunk * 8 : nullptr;
            }
            for (int ks = 0; ks < k_steps; ++ks, ++fill) {
                if (fill % GROUPS != group) continue;
                const uint32_t st = fill % STAGES, round = fill / STAGES;
                if (round > 0 && !warp_wait(&bar_free[st], (round - 1) & 1u)) {
                    ok = false;
                    break;
                }
                const uint32_t base = smem_u32(smem + st * Shape::STAGE);
                const int bytes = ks * ET_K + chunk * 8 < p.K ? 16 : 0;  // zeros behind the last channel
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int r = r0 + ROWS * i;
                    if (src[i])
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + r * 128 + ((chunk ^ (r & 7)) << 4)),
                                     "l"(bytes ? src[i] + ks * ET_K : src[i]), "r"(bytes)
                                     : "memory");
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                fence_proxy_async_smem();  // this thread's copies, before the products read them
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_full[st]);
            }
        }
        if (!ok && lane == 0 && *abort_flag == 0) timed_out();
        __syncwarp();
    } else {
        // =============== results ====================================================================
        const int q = warp & 3, row = q * 32 + lane;  // a warp reaches tensor-memory lanes 32 (warp % 4) ..
        const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
        const bool vec = p.N % 8 == 0 && (((uintptr_t)p.out) & 15) == 0;
        uint32_t tile = 0;
        for (int idx = blockIdx.x; idx < total; idx += gridDim.x, ++tile) {
            if (!cur.seek(s_first, p, n_tiles, idx)) break;
            const int m = cur.m0 + row;
            const bool have = m < cur.m_hi;
            const float s = UP && have ? p.scale[m] : 0.f;
            const int n0 = cur.n * (UP ? BN / 2 : BN);
            const int to = UP ? m : (have ? p.slot[m] : 0);  // this row's place in out
            const uint32_t buf = tile & 1u;
            if (!warp_wait(&bar_acc[buf], (tile >> 1) & 1u)) {
                if (lane == 0 && *abort_flag == 0) timed_out();
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + buf * BN + lane_sel;
            // 64 results of the warp's 32 rows at a time, turned in shared memory (16-byte pieces, swizzled by row): a
            // store instruction then writes 128 bytes of four rows instead of 16 bytes of 32
            uint8_t *turn = s_out + q * 32 * 128;
#pragma unroll 1
            for (int c = 0; c < (UP ? BN / 2 : BN); c += 64) {
                if (n0 + c >= p.N) break;  // uniform over the CTA
#pragma unroll
                for (int half = 0; half < 64; half += 32) {
                    float v[32];
                    if (UP) {
                        float u[32];
                        tmem_ld32x2(acc + c + half, v, acc + BN / 2 + c + half, u);
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
            if (lane == 0) mbar_arrive(&bar_read[buf]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 2 * BN);
}

template <bool UP, int BN>
static cudaError_t et_launch(const ExpertParams &p, cudaStream_t s, int *rc) {
    CUtensorMap ma, mw;
    {
        const int64_t dims[2] = {p.K, UP ? p.R / p.top : p.R}, strides[1] = {p.K};
        const int box[2] = {ET_K, ET_M};
        *rc = make_tensor_map(&ma, p.a, 2, dims, strides, box);  // not used by UP
    }
    if (*rc != NCKV_OK) return cudaSuccess;
    const int64_t N = p.N, K = p.K, halves = UP ? 2 : 1;
    const int64_t dims[4] = {K, N, halves, p.E}, strides[3] = {K, N * K, halves * N * K};
    const int box[4] = {ET_K, UP ? BN / 2 : BN, 1, 1};
    *rc = make_tensor_map(&mw, p.w, 4, dims, strides, box);
    if (*rc != NCKV_OK) return cudaSuccess;
    using Shape = EtShape<BN>;
    const cudaError_t e = cudaFuncSetAttribute(experts_tc_kernel<UP, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM);
    if (e != cudaSuccess) return e;
    const long long tiles = ((long long)p.R / ET_M + p.E) * ((p.N + BN / halves - 1) / (BN / halves));
    const int grid = tiles < sm_count() ? (int)tiles : sm_count();
    experts_tc_kernel<UP, BN><<<grid, ET_THREADS + (UP ? ET_GATHER : 0), Shape::SMEM, s>>>(ma, mw, p);
    return cudaGetLastError();
}

long long experts_tc_waves(bool up, int R, int E, int N, int bn) {
    const long long m_tiles = R / ET_M + (E + 1) / 2;
    const int per = up ? bn / 2 : bn;
    return (m_tiles * ((N + per - 1) / per) + sm_count() - 1) / sm_count();
}

// Narrow tiles read the operands more often, but leave smaller last waves: take them where that wins
// at an even spread of the positions.
bool experts_tc_wide(bool up, int R, int E, int N) {
    return 2 * experts_tc_waves(up, R, E, N, 256) * 10 <= experts_tc_waves(up, R, E, N, 128) * 11;
}

cudaError_t experts_tc(const ExpertParams &p, bool up, cudaStream_t s, int *rc) {
    if (p.E > ET_MAX_EXPERTS) {
        set_error("experts: at most %d experts", ET_MAX_EXPERTS);
        *rc = NCKV_E_UNSUPPORTED;
        return cudaSuccess;
    }
    const bool wide = experts_tc_wide(up, p.R, p.E, p.N);
    if (up) return wide ? et_launch<true, 256>(p, s, rc) : et_launch<true, 128>(p, s, rc);
    return wide ? et_launch<false, 256>(p, s, rc) : et_launch<false, 128>(p, s, rc);
}

}  // namespace nckv
