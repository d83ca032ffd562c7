// One decode step of a layer in one launch, for few (row, kv head) pairs and short caches: RoPE, norm and scale of q and k, the
// append of k and v and the attention of one new token per row (append.cu and decode_attn.cu take three launches for it).
//
// With a handful of pairs the three launches' latencies and the host's time for them are all there is: 4 rows of 2 heads with some 64 keys took
// 14 us a call (8.0 from a graph), all of it launches; now 9 to 11 (5.1), the host's time for one.  A cluster of CTAs takes a pair; its warps take
// the pair's keys 16 at a time, consecutive groups on different CTAs, on the grid of multiples of 16 (so a group lies in one page).  Every CTA
// transforms the G query rows and the new key for itself while its first keys and values are on their way; the first CTA writes the new rows
// into the cache.  No CTA reads a row that another one writes: the new token's key and value come from the inputs, as a group of their own.
//
// A warp loads a group straight into the fragments of m16n8k16: a lane's 16-byte pieces of a key row are the channels of its places in two
// steps of the sum (its order is free, q is arranged alike), a lane's 32 bytes of four value rows are turned into 16 columns' pairs with byte
// permutes.  Two groups are on their way at once, all that a warp of an ordinary call has.  Eight warps to a CTA: with four of them, each with
// twice the groups one after the other, 2000 keys of 12 heads took 9.4 us, now 7.9.  The warps' (max, sum, output) meet in shared memory
// (rows padded: unpadded, 16 heads to a kv head took 11.8 us for 2000 keys, now 10.1), the CTAs' through the cluster's.
#include <math.h>

#include <atomic>

#include "rope_row.cuh"
#include "tc05.cuh"

namespace nckv {

constexpr int DS_WARPS = 8, DS_THREADS = 32 * DS_WARPS, DS_KEYS = 16, DS_MAX_G = 16;
constexpr int DS_O_ROW = NCKV_D + 16;  // floats between rows of partial outputs: channel d at out_place(d), free of conflicts as the fragments write them
__host__ __device__ constexpr int out_place(int d) { return d + 4 * (d >> 5); }
constexpr int small_smem(bool ghi) { return DS_WARPS * (ghi ? DS_MAX_G : 8) * DS_O_ROW * 4; }  // the warps' partial outputs
constexpr int DS_Q_ROW = NCKV_D + 8;  // elements between q rows in shared memory: 16-byte reads of 8 rows are free of conflicts

struct DecodeSmallParams {
    const __nv_bfloat16 *q, *k, *v;            // (B, heads, 128), rows of a token q_stride .. elements apart
    long long q_stride, k_stride, v_stride;
    __nv_bfloat16 *k_cache, *v_cache;
    long long batch_stride, token_stride;      // paged: batch_stride is the distance between pages
    const int32_t *block_table;                // null: dense rows
    int page_tokens, max_pages, n_pages;
    const int32_t *seqlens;
    const uint2 *cos, *sin;
    __nv_bfloat16 *out;
    int32_t *status;
    int Hq, Hkv, G, T_max, rope_len, window_left;
    float scale_log2, qk_scale, eps;
};

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float4 remote_load4(const float *p, uint32_t rank) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_of_rank(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ float2 remote_load2(const float *p, uint32_t rank) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(smem_of_rank(p, rank)) : "memory");
    return v;
}

// 16 keys and values in fragments.  k[n][c]: key 8 n + g, channels 32 c + 8 t ..; v[r][h]: token 2 t, 2 t + 1, 8 + 2 t, 9 + 2 t, channels 16 g + 8 h ..
struct KeyGroup {
    uint4 k[2][4], v[4][2];
    int first;  // position of its first key
};

template <bool GHI>  // more than 8 query heads to a kv head
__global__ void __launch_bounds__(DS_THREADS) decode_small_kernel(const DecodeSmallParams p) {
    constexpr int ROW_LANES = 2 * DS_WARPS, MAX_G = GHI ? DS_MAX_G : 8;  // ROW_LANES: half-warps
    extern __shared__ __align__(16) float s_parts[];
    float (*s_o)[MAX_G][DS_O_ROW] = reinterpret_cast<float (*)[MAX_G][DS_O_ROW]>(s_parts);
    __shared__ __align__(16) __nv_bfloat16 s_q[MAX_G][DS_Q_ROW];
    __shared__ __align__(16) __nv_bfloat16 s_k[NCKV_D];
    __shared__ __align__(8) float s_ml[DS_WARPS][16][2];   // per warp and row: max (of base-2 logarithms), sum
    __shared__ __align__(8) float s_part[16][2];           // the CTA's
    // No early release of what follows: an attention kernel behind the next append reads older cache rows before its own wait, and this
    // grid's new row may be one of them.
    pdl_wait_prior_grids();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int ctas = (int)cluster_ctas(), rank = (int)cluster_rank(), pair = blockIdx.x / ctas, G = p.G;
    const int b = pair / p.Hkv, h = pair - b * p.Hkv;
    // the input rows do not depend on the row's length: a half-warp each, G of q and the key
    const int hw = tid >> 4, j = tid & 15;
    constexpr int ROWS = (MAX_G + ROW_LANES) / ROW_LANES;
    uint2 lo[ROWS], hi[ROWS];
    const __nv_bfloat16 *q_in = p.q + b * p.q_stride + (long long)h * G * NCKV_D, *k_in = p.k + b * p.k_stride + (long long)h * NCKV_D;
    const __nv_bfloat16 *v_in = p.v + b * p.v_stride + (long long)h * NCKV_D;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = hw + ROW_LANES * i;
        lo[i] = hi[i] = make_uint2(0, 0);
        if (r > G) continue;
        const uint2 *row = reinterpret_cast<const uint2 *>(r < G ? q_in + r * NCKV_D : k_in);
        lo[i] = row[j];
        hi[i] = row[16 + j];
    }
    const int len = p.seqlens[b];
    const bool ok = len >= 0 && len < p.T_max && len < p.rope_len;
    if (!ok && rank == 0 && tid == 0 && h == 0) atomicOr(p.status, (int)(len < 0 ? NCKV_ST_BAD_SEQLEN : NCKV_ST_OVERFLOW));
    // old keys [from, len), in groups on the grid of 16; the new one is a group of its own behind the last
    const int from = ok && p.window_left >= 0 ? max(0, len - p.window_left) : 0;
    const int first = from / DS_KEYS, groups = ok ? (len > from ? (len + DS_KEYS - 1) / DS_KEYS - first : 0) : 0, warps = ctas * DS_WARPS;
    const int own = warp * ctas + rank;  // consecutive groups go to different CTAs
    // a group's place in the caches, or -1 where the table names no page of the pool
    auto place = [&](int pos) -> long long {
        if (!p.block_table) return b * p.batch_stride + pos * p.token_stride;
        const int idx = pos / p.page_tokens, page = p.block_table[(long long)b * p.max_pages + idx];
        if (page < 0 || page >= p.n_pages) {
            atomicOr(p.status, (int)NCKV_ST_BAD_PAGE);
            return -1;
        }
        return page * p.batch_stride + (pos - idx * p.page_tokens) * p.token_stride;
    };
    auto load = [&](KeyGroup &x, int i) {  // group i
        x.first = (first + i) * DS_KEYS;
        const long long at = place(x.first);
        const __nv_bfloat16 *kr = p.k_cache + at + (long long)h * NCKV_D + 8 * t4, *vr = p.v_cache + at + (long long)h * NCKV_D + 16 * g;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int key = 8 * n + g;
                x.k[n][c] = make_uint4(0, 0, 0, 0);
                if (at >= 0 && x.first + key < len && x.first + key >= from)
                    x.k[n][c] = *reinterpret_cast<const uint4 *>(kr + key * p.token_stride + 32 * c);
            }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int key = 8 * (r >> 1) + 2 * t4 + (r & 1);
                x.v[r][half] = make_uint4(0, 0, 0, 0);
                if (at >= 0 && x.first + key < len && x.first + key >= from)
                    x.v[r][half] = *reinterpret_cast<const uint4 *>(vr + key * p.token_stride + 8 * half);
            }
    };
    KeyGroup a, c;
    if (own < groups) load(a, own);
    if (own + warps < groups) load(c, own + warps);

    // ---- q' and k', and the new rows into the cache ----
    {
        uint2 cs = make_uint2(0, 0), sn = make_uint2(0, 0);
        if (ok) {
            cs = p.cos[(long long)len * 16 + j];
            sn = p.sin[(long long)len * 16 + j];
        }
        long long at = -1;
        if (ok && rank == 0) at = place(len);
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const int r = hw + ROW_LANES * i;
            if (ROW_LANES * i > G) break;  // uniform
            rope_norm_scale(lo[i], hi[i], cs, sn, p.qk_scale, p.eps);
            if (r > G) continue;
            uint2 *to = reinterpret_cast<uint2 *>(r < G ? s_q[r] : s_k);
            to[j] = lo[i];
            to[16 + j] = hi[i];
            if (r == G && at >= 0) {
                uint2 *dst = reinterpret_cast<uint2 *>(p.k_cache + at + (long long)h * NCKV_D);
                dst[j] = lo[i];
                dst[16 + j] = hi[i];
            }
        }
        if (at >= 0 && hw == ROW_LANES - 1) reinterpret_cast<uint4 *>(p.v_cache + at + (long long)h * NCKV_D)[j] = reinterpret_cast<const uint4 *>(v_in)[j];
    }
    __syncthreads();
    uint4 q0[4], q1[GHI ? 4 : 1];  // rows g and g + 8, channels 32 c + 8 t ..
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        q0[x] = g < G ? *reinterpret_cast<const uint4 *>(&s_q[g][32 * x + 8 * t4]) : make_uint4(0, 0, 0, 0);
        if (GHI) q1[x] = g + 8 < G ? *reinterpret_cast<const uint4 *>(&s_q[g + 8][32 * x + 8 * t4]) : make_uint4(0, 0, 0, 0);
    }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f}, o[16][4];
#pragma unroll
    for (int n = 0; n < 16; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    auto consume = [&](const KeyGroup &x, int lo_key, int hi_key) {  // keys [lo_key, hi_key) of the group are seen
        float s[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {
                mma_16816(s[n], q0[ch].x, GHI ? q1[ch].x : 0u, q0[ch].y, GHI ? q1[ch].y : 0u, x.k[n][ch].x, x.k[n][ch].y);
                mma_16816(s[n], q0[ch].z, GHI ? q1[ch].z : 0u, q0[ch].w, GHI ? q1[ch].w : 0u, x.k[n][ch].z, x.k[n][ch].w);
            }
        }
        uint32_t pa[2][2];
#pragma unroll
        for (int r = 0; r < (GHI ? 2 : 1); ++r) {
            float top = -INFINITY;
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int key = 8 * n + 2 * t4 + e;
                    float &v = s[n][2 * r + e];
                    if (key < lo_key || key >= hi_key) v = -INFINITY;
                    top = fmaxf(top, v);
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float m_old = m_run[r];
            m_run[r] = fmaxf(m_old, top * p.scale_log2);
            // nothing but scores of -inf so far: weights and sums of 0, not 2^(-inf + inf)
            const float m = m_run[r] == -INFINITY ? 0.f : m_run[r], alpha = exp2f(m_old - m);
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const float e0 = exp2f(fmaf(s[n][2 * r], p.scale_log2, -m)), e1 = exp2f(fmaf(s[n][2 * r + 1], p.scale_log2, -m));
                sum += e0 + e1;
                pa[n][r] = pack_bf16x2(e0, e1);
            }
            l_run[r] = l_run[r] * alpha + sum;
#pragma unroll
            for (int n = 0; n < 16; ++n) {
                o[n][2 * r] *= alpha;
                o[n][2 * r + 1] *= alpha;
            }
        }
        if (!GHI) pa[0][1] = pa[1][1] = 0u;
        // column n of tile i is channel 16 n + i
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint4 &v0 = x.v[0][i >> 3], &v1 = x.v[1][i >> 3], &v2 = x.v[2][i >> 3], &v3 = x.v[3][i >> 3];
            const int w = (i & 7) >> 1;
            auto word = [&](const uint4 &v) { return w == 0 ? v.x : (w == 1 ? v.y : (w == 2 ? v.z : v.w)); };
            const uint32_t pick = i & 1 ? 0x7632u : 0x5410u;
            mma_16816(o[i], pa[0][0], pa[0][1], pa[1][0], pa[1][1], __byte_perm(word(v0), word(v1), pick), __byte_perm(word(v2), word(v3), pick));
        }
    };
    for (int i = own; i < groups; i += 2 * warps) {
        consume(a, max(0, from - a.first), len - a.first);
        if (i + 2 * warps < groups) load(a, i + 2 * warps);
        if (i + warps < groups) {
            consume(c, max(0, from - c.first), len - c.first);
            if (i + 3 * warps < groups) load(c, i + 3 * warps);
        }
    }
    if (ok && own == groups % warps) {  // the new token, in the first place of a group
        KeyGroup x;
        const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
            x.k[0][ch] = g == 0 ? *reinterpret_cast<const uint4 *>(s_k + 32 * ch + 8 * t4) : zero;
            x.k[1][ch] = zero;
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            x.v[0][half] = t4 == 0 ? *reinterpret_cast<const uint4 *>(v_in + 16 * g + 8 * half) : zero;
            x.v[1][half] = x.v[2][half] = x.v[3][half] = zero;
        }
        consume(x, 0, 1);
    }
    // ---- the warps' parts: a lane holds channels 32 t + i and 32 t + 16 + i of its rows ----
#pragma unroll
    for (int r = 0; r < (GHI ? 2 : 1); ++r) {
        float l = l_run[r];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        const int row = g + 8 * r;
        if (t4 == 0) *reinterpret_cast<float2 *>(s_ml[warp][row]) = make_float2(m_run[r], l);
        if (row < G) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                *reinterpret_cast<float4 *>(&s_o[warp][row][out_place(32 * t4 + i)]) = make_float4(o[i][2 * r], o[i + 1][2 * r], o[i + 2][2 * r], o[i + 3][2 * r]);
                *reinterpret_cast<float4 *>(&s_o[warp][row][out_place(32 * t4 + 16 + i)]) =
                    make_float4(o[i][2 * r + 1], o[i + 1][2 * r + 1], o[i + 2][2 * r + 1], o[i + 3][2 * r + 1]);
            }
        }
    }
    __syncthreads();
    const int ch = tid & (NCKV_D - 1);
    for (int r = tid / NCKV_D; r < G; r += DS_WARPS * 32 / NCKV_D) {  // a channel each
        float m = -INFINITY, l = 0.f, sum = 0.f, f[DS_WARPS];
#pragma unroll
        for (int w = 0; w < DS_WARPS; ++w) m = fmaxf(m, s_ml[w][r][0]);
#pragma unroll
        for (int w = 0; w < DS_WARPS; ++w) {
            f[w] = s_ml[w][r][0] == -INFINITY ? 0.f : exp2f(s_ml[w][r][0] - m);
            l = fmaf(f[w], s_ml[w][r][1], l);
            sum = fmaf(f[w], s_o[w][r][out_place(ch)], sum);
        }
        s_o[0][r][out_place(ch)] = sum;  // nobody else reads or writes this channel
        if (ch == 0) *reinterpret_cast<float2 *>(s_part[r]) = make_float2(m, l);
    }
    cluster_sync();
    // ---- the CTAs' parts: four channels a thread, rows dealt over CTAs and warps ----
    for (int r = rank * DS_WARPS + warp; r < G; r += ctas * DS_WARPS) {
        float m = -INFINITY, l = 0.f;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 ml[8];
        float4 part[8];
#pragma unroll
        for (int x = 0; x < 8; ++x)
            if (x < ctas) {
                ml[x] = remote_load2(s_part[r], x);
                part[x] = remote_load4(&s_o[0][r][out_place(4 * lane)], x);
            }
#pragma unroll
        for (int x = 0; x < 8; ++x)
            if (x < ctas) m = fmaxf(m, ml[x].x);
#pragma unroll
        for (int x = 0; x < 8; ++x)
            if (x < ctas) {
                const float f = ml[x].x == -INFINITY ? 0.f : exp2f(ml[x].x - m);
                l = fmaf(f, ml[x].y, l);
                sum.x = fmaf(f, part[x].x, sum.x); sum.y = fmaf(f, part[x].y, sum.y);
                sum.z = fmaf(f, part[x].z, sum.z); sum.w = fmaf(f, part[x].w, sum.w);
            }
        const float inv = ok ? 1.f / l : 0.f;
        *reinterpret_cast<uint2 *>(p.out + ((long long)b * p.Hq + (long long)h * G + r) * NCKV_D + 4 * lane) =
            make_uint2(pack_bf16x2(sum.x * inv, sum.y * inv), pack_bf16x2(sum.z * inv, sum.w * inv));
    }
    cluster_sync();  // nobody reaches for this CTA's memory any more
}

// Clusters of `ctas` CTAs that the device holds at once, 0 where it cannot say.
static int small_clusters(bool ghi, int ctas) {
    static std::atomic<int> known[64][2][4];  // one more than the answer
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
    std::atomic<int> &slot = known[dev][ghi][ctas == 8 ? 3 : ctas / 2];
    if (const int v = slot.load(std::memory_order_relaxed)) return v - 1;
    const auto kernel = ghi ? decode_small_kernel<true> : decode_small_kernel<false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(DS_THREADS);
    cfg.dynamicSmemBytes = small_smem(ghi);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, small_smem(ghi)) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    slot.store(n + 1, std::memory_order_relaxed);
    return n;
}

// CTAs to a pair, 0: not taken.  As many as there are SMs for, all in one wave, and at most three groups of keys to a warp, where the other
// kernels' single launches still cost more.  us from a CUDA graph, three launches / one, all keys present; a call by itself costs 13.9-15 / 8.5-11:
//   4 x 2 + 2 heads: 64 keys 8.0 / 5.1, 2000 keys 8.9 / 7.4; 1 x 12 + 12 heads: 100 keys 8.4 / 5.5, 2000 keys 9.3 / 7.9, 3000 keys 10.4 / 9.0,
//   four groups, 4000 keys, 10.2 / 10.8; 6 x 12 + 12: 500 keys 10.1 / 7.7; 8 x 16 + 16: 250 keys 10.5 / 7.8; 16 x 16 + 2: 1000 keys 11.1 / 8.8.
// A group of more than 8 heads has twice the work: 1 x 16 + 1, 2000 keys 9.1 / 10.1 on clusters of 8, but 70 rows, 500 keys 23.0 / 10.9 and 140
// rows, 250 keys 30.1 / 10.9.  Clusters of 8 that did not fit at once took 19 us for 2000 keys.
static int small_ctas(int B, int Hq, int Hkv, long long capacity, int window_left) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || Hq / Hkv > DS_MAX_G) return 0;
    const long long pairs = (long long)B * Hkv, keys = window_left >= 0 && window_left + 1LL < capacity ? window_left + 1LL : capacity;
    for (int ctas = 8; ctas >= 1; ctas /= 2) {
        if (pairs * ctas > sm_count()) continue;
        const int to_a_warp = Hq / Hkv <= 8 ? 3 : (ctas == 8 ? 1 : 2);
        if (keys > (long long)ctas * DS_WARPS * DS_KEYS * to_a_warp) return 0;
        if (pairs <= small_clusters(Hq / Hkv > 8, ctas)) return ctas;
    }
    return 0;
}

}  // namespace nckv

extern "C" {

int nckv_decode_small_fits(int B, int Hq, int Hkv, int64_t capacity, int window_left) {
    return nckv::small_ctas(B, Hq, Hkv, capacity, window_left) > 0;
}

int nckv_decode_small(const void *q, const void *k, const void *v, int64_t q_stride, int64_t k_stride, int64_t v_stride, void *k_cache,
                      void *v_cache, const int32_t *block_table, const int32_t *cache_seqlens, const void *cos, const void *sin, void *out,
                      int B, int Hq, int Hkv, int D, int T_max, int max_pages, int n_pages, int64_t batch_stride, int64_t token_stride,
                      int rope_len, int window_left, float qk_scale, float eps, int32_t *status, void *stream) {
    using namespace nckv;
    if (!q || !k || !v || !k_cache || !v_cache || !cache_seqlens || !cos || !sin || !out || !status) {
        set_error("decode_small: null pointer argument");
        return NCKV_E_ARG;
    }
    if (D != NCKV_D || B <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || T_max <= 0 || rope_len <= 0 || (block_table && (max_pages <= 0 || n_pages <= 0))) {
        set_error("decode_small: size out of range (B=%d Hq=%d Hkv=%d D=%d T_max=%d)", B, Hq, Hkv, D, T_max);
        return NCKV_E_ARG;
    }
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)cos | (uintptr_t)sin | (uintptr_t)out) & 15 ||
        (q_stride | k_stride | v_stride | batch_stride | token_stride) % 8 || token_stride < (int64_t)Hkv * D || (block_table && T_max % DS_KEYS)) {
        set_error("decode_small: tensors must be 16-byte aligned with strides of whole 16-byte pieces, pages of whole groups of %d keys", DS_KEYS);
        return NCKV_E_ARG;
    }
    const long long capacity = block_table ? (long long)T_max * max_pages : T_max;
    const int ctas = capacity <= 0x7fffffffLL ? small_ctas(B, Hq, Hkv, capacity, window_left) : 0;
    if (ctas == 0) {
        set_error("decode_small: B=%d x Hkv=%d pairs over %lld keys are too many", B, Hkv, capacity);
        return NCKV_E_UNSUPPORTED;
    }
    DecodeSmallParams p;
    p.q = static_cast<const __nv_bfloat16 *>(q); p.k = static_cast<const __nv_bfloat16 *>(k); p.v = static_cast<const __nv_bfloat16 *>(v);
    p.q_stride = q_stride ? q_stride : (long long)Hq * D;
    p.k_stride = k_stride ? k_stride : (long long)Hkv * D;
    p.v_stride = v_stride ? v_stride : (long long)Hkv * D;
    p.k_cache = static_cast<__nv_bfloat16 *>(k_cache); p.v_cache = static_cast<__nv_bfloat16 *>(v_cache);
    p.batch_stride = batch_stride; p.token_stride = token_stride;
    p.block_table = block_table; p.page_tokens = T_max; p.max_pages = max_pages; p.n_pages = n_pages;
    p.seqlens = cache_seqlens; p.cos = static_cast<const uint2 *>(cos); p.sin = static_cast<const uint2 *>(sin);
    p.out = static_cast<__nv_bfloat16 *>(out); p.status = status;
    p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv; p.T_max = (int)capacity; p.rope_len = rope_len; p.window_left = window_left;
    p.scale_log2 = (float)(1.4426950408889634 / sqrt((double)D));
    p.qk_scale = qk_scale; p.eps = eps;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(B * Hkv * ctas));
    cfg.blockDim = dim3(DS_THREADS);
    cfg.dynamicSmemBytes = small_smem(p.G > 8);
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    NCKV_CUDA_CHECK(cudaLaunchKernelEx(&cfg, p.G > 8 ? decode_small_kernel<true> : decode_small_kernel<false>, p));
    return NCKV_OK;
}

}  // extern "C"
