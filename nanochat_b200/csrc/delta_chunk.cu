// The gated delta rule of delta.cu for bf16 prompts, in chunks of 16 tokens whose products run as m16n8k8 tf32
// matrix instructions.  Every fp32 operand enters as two tf32 terms (hi * hi + hi * lo + lo * hi, fp32 sums), which
// keeps about 22 bits of it; the state itself stays in fp32 accumulators.
//
// With c_t = w_1 .. w_t (products from the chunk's first token on) and the state S before the chunk
//   u = T v - W S            T = (1 + diag(beta) A)^-1 diag(beta),   A_ti = sum_c k_t k_i w_(i+1) .. w_t  (i < t)
//                            W_t = sum_i T_ti c_i k_i
//   o = QT v + Y S           QT = Q T,   Q_ti = sum_c q_t k_i w_(i+1) .. w_t  (i <= t),   Y_t = c_t q_t - sum_i Q_ti W_i
//   S <- diag(c_16) S + sum_i (w_(i+1) .. w_16 k_i) u_i^T
// Only products of decays appear (each <= 1), so nothing overflows however strong the decay.
//
//   delta_chunk_prepare_kernel   one CTA per (row, head, chunk), a thread per key channel: norms, decays, T, QT, W and Y,
//                                left as one record in the order the matrix fragments want
//   delta_chunk_kernel           a warp owns 16 value columns of one (row, head).  S^T (16 x Dk) lives in
//                                accumulator fragments: they are the left operand of the next chunk's products
//                                as they stand (the order of the summed index is free), so no value crosses
//                                lanes.  Records arrive by bulk copies through a ring in shared memory.
//   delta_chunk_split_kernel     the same with few heads: the warps of a CTA share 16 value columns, 16 key channels each
//
// The chunks of a head follow one another, and with few heads the chain from one state to the next is the bound.  It holds two products
// only (W S, then u into S): T and Q are multiplied into the rows beforehand, T v and QT v do not wait for the state.  us, both kernels,
// heads of 128 x 128 (before: R = S^T k, u = T (v - R), o = P + Q u one after the other, two or four warps to 16 columns, values and
// outputs moved by the warps of the chain), B200: 1 x 6007 tokens, 12 heads 644 / 449, 1 x 2048 228 / 165, 4 x 1024 332 / 229, 8 x 1024 408 /
// 401, 3 x 1024, 16 heads 334 / 230.  A chunk of the chain takes 1 800 cycles, most of them latency.  Against 64 bits 1 x 2048 tokens, 12
// heads: outputs 3.0e-6 / 1.7e-6, state 2.8e-6 / 1.6e-6.
// A chunk's share of the state is summed from zero and added to the decayed state by one fused multiply-add, rounded to nearest (matrix
// instructions round their sums towards zero, which would pile up in the state).
#include "chunk.cuh"
#include "tc05.cuh"

namespace nckv {

constexpr int DC_RING = 3;  // records in flight
// record: [-W : 16 rows][Y : 16 rows][k_i to the end : KP x 16 tokens][c_16 in two terms : 2 x KP][T : 16 x 16][QT : 16 x 16]
__host__ __device__ constexpr int dc_record(int KP) { return 2 * CH_T * KP + KP * CH_T + 2 * KP + 2 * CH_T * CH_T; }

struct DeltaChunkParams {
    const __nv_bfloat16 *q, *k, *v;  // (B * T) rows; heads packed inside a row
    long long q_stride, k_stride, v_stride;
    const float *x;                  // (B * T) rows of H * Dk decay logits
    long long x_stride;
    const float *x0, *rate;          // (H * Dk), (H)
    const __nv_bfloat16 *b;          // (B * T) rows of H step-size logits
    long long b_stride;
    float *records;                  // (B, H, chunks, dc_record(KP))
    float *state;                    // (B, H, Dk, Dv)
    float *out;                      // (B * T, H * Dv)
    int32_t *status;
    int B, T, H, G, Dk, Dv, n_chunks, n_cols;
    int pairs;                       // rows of v and out allow accesses of two columns
};

template <int KP>
__global__ void __launch_bounds__(KP, 640 / KP) delta_chunk_prepare_kernel(const DeltaChunkParams p) {
    constexpr int NW = KP / 32;
    __shared__ __align__(16) float s_work[NW][CH_PAIR_ROWS * CH_PAIR_STRIDE];  // a warp's operands, then its sums of pairs
    __shared__ float s_sum[2][NW][32], s_beta[CH_T], s_scale[2][CH_T], s_a[CH_T][CH_T];
    __shared__ __align__(16) float s_q[CH_T][CH_T], s_t[CH_T][CH_T];
    const int c = threadIdx.x, lane = c & 31, warp = c >> 5;
    const int h = blockIdx.x % p.H, chunk = blockIdx.x / p.H, b = blockIdx.y;  // heads fastest: rows are shared in L2
    const int g = h / (p.H / p.G), t0 = chunk * CH_T, n = min(CH_T, p.T - t0);
    const bool on = c < p.Dk;
    const float rate = p.rate[h], x0 = on ? p.x0[h * p.Dk + c] : 0.f;
    const long long row = (long long)b * p.T + t0;
    const __nv_bfloat16 *gq = p.q + row * p.q_stride + (long long)g * p.Dk + c, *gk = p.k + row * p.k_stride + (long long)g * p.Dk + c;
    const float *gx = p.x + row * p.x_stride + (long long)h * p.Dk + c;
    float q[CH_T], k[CH_T], w[CH_T];  // tokens behind the last leave the state as it is
#pragma unroll
    for (int t = 0; t < CH_T; ++t) {
        const bool in = on && t < n;
        q[t] = in ? to_f(gq[t * p.q_stride]) : 0.f;
        k[t] = in ? to_f(gk[t * p.k_stride]) : 0.f;
        w[t] = in ? gx[t * p.x_stride] : 0.f;
    }
    if (c < CH_T) s_beta[c] = c < n ? Fn<__nv_bfloat16>::sigmoid(to_f(p.b[(row + c) * p.b_stride + h])) : 0.f;
    {
        float part[32];
#pragma unroll
        for (int t = 0; t < CH_T; ++t) {
            part[t] = q[t] * q[t];
            part[CH_T + t] = k[t] * k[t];
            // softplus in the fast functions: what it loses for very negative logits is far below one rounding of w
            const float z = w[t] + x0;
            w[t] = on && t < n ? __expf(-rate * (fmaxf(z, 0.f) + __logf(1.f + __expf(-fabsf(z))))) : 1.f;
        }
        const int at = scatter_sum<16, 32>(part, lane);
        s_sum[0][warp][at] = part[0];
    }
    __syncthreads();
    if (c < 32) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < NW; ++i) s += s_sum[0][i][c];
        s_scale[c >> 4][c & 15] = (c < CH_T ? rsqrtf((float)p.Dk) : 1.f) / sqrtf(s + 1e-6f);
    }
    __syncthreads();
    {
        float part[CH_T];
#pragma unroll
        for (int t = 0; t < CH_T; ++t) {
            q[t] *= s_scale[0][t];
            k[t] *= s_scale[1][t];
            part[t] = q[t] * k[t];
        }
        const int at = scatter_sum<16, CH_T>(part, lane);
        if (!(lane & 1)) s_sum[1][warp][at] = part[0];
    }
    float *rec = p.records + (((long long)b * p.H + h) * p.n_chunks + chunk) * dc_record(KP);
    {
        // the keys carried to the end, this channel's 16 tokens in the order of ch_place
        float ke[CH_T], f = 1.f;
#pragma unroll
        for (int i = CH_T - 1; i >= 0; --i) {
            ke[i] = f * k[i];
            f *= w[i];
        }
        float4 *dst = reinterpret_cast<float4 *>(rec + 2 * CH_T * KP + c * CH_T);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_float4(ke[2 * i], ke[2 * i + 1], ke[8 + 2 * i], ke[9 + 2 * i]);
    }
    {
        float4 acc[4];
        pair_products<true, false>(s_work[warp], lane, k, q, w, acc);
#pragma unroll
        for (int l = 0; l < 4; ++l) reinterpret_cast<float4 *>(s_work[warp])[l * 32 + lane] = acc[l];
    }
    // the rows carried from the start (k's place takes them; the products of decays in two terms)
    {
        float hi = 1.f, lo = 0.f;
#pragma unroll
        for (int t = 0; t < CH_T; ++t) {
            const float next = hi * w[t];
            lo = fmaf(lo, w[t], fmaf(hi, w[t], -next));
            hi = next;
            k[t] = fmaf(hi, k[t], lo * k[t]);
            q[t] = fmaf(hi, q[t], lo * q[t]);
        }
        rec[2 * CH_T * KP + KP * CH_T + c] = hi;
        rec[2 * CH_T * KP + KP * CH_T + KP + c] = lo;
    }
    __syncthreads();
    for (int i = c; i < CH_T * CH_T; i += KP) {
        const int t = i / CH_T, j = i % CH_T;
        float a = 0.f, qk = 0.f;
        if (j < t) {
            int level, at, part;
            pair_place(t, j, 0, level, at, part);
#pragma unroll
            for (int l = 0; l < NW; ++l) {
                const float *from = s_work[l] + (level * 32 + at) * 4 + part;
                a += from[0];
                qk += from[2];
            }
        } else if (j == t) {
#pragma unroll
            for (int l = 0; l < NW; ++l) qk += s_sum[1][l][t];
        }
        s_a[t][j] = a;
        s_q[t][j] = qk;
    }
    __syncthreads();
    float *tail = rec + 2 * CH_T * KP + KP * CH_T + 2 * KP;
    if (c < CH_T) {  // column c of T by forward substitution
        float u[CH_T];
#pragma unroll
        for (int t = 0; t < CH_T; ++t) {
            float s = t == c ? 1.f : 0.f;
#pragma unroll
            for (int i = 0; i < CH_T; ++i)
                if (i < t) s = fmaf(-s_a[t][i], u[i], s);  // u[i] is zero for i < c
            u[t] = s_beta[t] * s;
            s_t[t][c] = u[t];
            tail[t * CH_T + ch_place(c)] = u[t];
        }
    }
    __syncthreads();
    for (int i = c; i < CH_T * CH_T; i += KP) {
        const int t = i / CH_T, j = i % CH_T;
        float s = 0.f;
#pragma unroll
        for (int l = 0; l < CH_T; ++l) s = fmaf(s_q[t][l], s_t[l][j], s);  // zero above both diagonals
        tail[CH_T * CH_T + t * CH_T + ch_place(j)] = s;
    }
    // row t of a lower triangular matrix times this channel's values of tokens 0 .. t, two tokens at a time
    auto row_times = [&](const float *m, int t, const float (&x)[CH_T]) {
        float2 sum = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < t; i += 2) sum = ffma2(*reinterpret_cast<const float2 *>(m + i), make_float2(x[i], x[i + 1]), sum);
        float r = sum.x + sum.y;
        if (t % 2 == 0) r = fmaf(m[t], x[t], r);
        return r;
    };
#pragma unroll
    for (int t = 0; t < CH_T; ++t) {
        w[t] = row_times(s_t[t], t, k);
        rec[ch_at<KP>(t, c)] = -w[t];
    }
#pragma unroll
    for (int t = 0; t < CH_T; ++t) rec[ch_at<KP>(CH_T + t, c)] = q[t] - row_times(s_q[t], t, w);
}

// A step's operands in the matrix fragments' order.  Fragment tiles 2 j and 2 j + 1 hold channels 16 j + 4 t + {0, 1} and + {2, 3} in
// columns 2 t and 2 t + 1; rows g and g + 8 are value columns 2 g and 2 g + 1, so that values and outputs move in pairs where their rows
// allow it.

// tokens 8 m .. of 16 columns of S^T (channels 16 j .. in a0, a1) times the rows -W (m = 0, 1) or Y (m = 2, 3).  r: leading terms, rb and ra: cross
// terms of the rows' and the state's low terms.  A matrix instruction takes longer to finish than to issue: neighbours in the order below
// add to different accumulators.
template <int RS>
__device__ __forceinline__ void rows_product(float (*r)[4], float (*rb)[4], float (*ra)[4], const float *at, bool first, const LeftFrag &a0,
                                             const LeftFrag &a1) {
    const Pair4 bb[2] = {Pair4(*reinterpret_cast<const float4 *>(at)), Pair4(*reinterpret_cast<const float4 *>(at + 8 * RS))};
#pragma unroll
    for (int m = 0; m < 2; ++m) mma_tf32(r[m], a0.hi, bb[m].hi[0], bb[m].hi[1]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (first) mma_tf32_first(rb[m], a0.hi, bb[m].lo[0], bb[m].lo[1]);
        else mma_tf32(rb[m], a0.hi, bb[m].lo[0], bb[m].lo[1]);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (first) mma_tf32_first(ra[m], a0.lo, bb[m].hi[0], bb[m].hi[1]);
        else mma_tf32(ra[m], a0.lo, bb[m].hi[0], bb[m].hi[1]);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) mma_tf32(r[m], a1.hi, bb[m].hi[2], bb[m].hi[3]);
#pragma unroll
    for (int m = 0; m < 2; ++m) mma_tf32(rb[m], a1.hi, bb[m].lo[2], bb[m].lo[3]);
#pragma unroll
    for (int m = 0; m < 2; ++m) mma_tf32(ra[m], a1.lo, bb[m].hi[2], bb[m].hi[3]);
}

// v^T (two halves of the tokens; a bf16 value is exact in one term) times 8 rows of T or QT (at: row g of them), lower triangular: tokens 0-7 (m even)
// take nothing from 8-15
__device__ __forceinline__ void value_product(float (&r)[4], const uint32_t (&va)[2][4], int m, const float *at) {
    const Pair4 bt(*reinterpret_cast<const float4 *>(at));
    mma_tf32(r, va[0], bt.lo[0], bt.lo[1]);
    if (m & 1) mma_tf32(r, va[1], bt.lo[2], bt.lo[3]);
    mma_tf32(r, va[0], bt.hi[0], bt.hi[1]);
    if (m & 1) mma_tf32(r, va[1], bt.hi[2], bt.hi[3]);
}

// N tiles of S^T <- S^T diag(c_16) + u^T K.  at: this lane's place of the first tile's keys, cw: of its decays
template <int N, int KP>
__device__ __forceinline__ void update_tiles(float (*s)[4], const LeftFrag &u0, const LeftFrag &u1, const float *at, const float *cw) {
    float d[N][4];
    const auto keys = [&](int n) { return Pair4(*reinterpret_cast<const float4 *>(at + (16 * (n >> 1) + 2 * (n & 1)) * CH_T)); };
    if constexpr (N == 4) {
        const Pair4 b[4] = {keys(0), keys(1), keys(2), keys(3)};
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_tf32_first(d[n], u0.lo, b[n].hi[0], b[n].hi[1]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_tf32(d[n], u1.lo, b[n].hi[2], b[n].hi[3]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_tf32(d[n], u0.hi, b[n].lo[0], b[n].lo[1]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_tf32(d[n], u1.hi, b[n].lo[2], b[n].lo[3]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_tf32(d[n], u0.hi, b[n].hi[0], b[n].hi[1]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_tf32(d[n], u1.hi, b[n].hi[2], b[n].hi[3]);
    } else {
        float c[N][4];
        const Pair4 b[2] = {keys(0), keys(1)};
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_tf32_first(d[n], u0.hi, b[n].hi[0], b[n].hi[1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_tf32_first(c[n], u0.lo, b[n].hi[0], b[n].hi[1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_tf32(d[n], u1.hi, b[n].hi[2], b[n].hi[3]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_tf32(c[n], u1.lo, b[n].hi[2], b[n].hi[3]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_tf32(d[n], u0.hi, b[n].lo[0], b[n].lo[1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) mma_tf32(c[n], u1.hi, b[n].lo[2], b[n].lo[3]);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) d[n][e] += c[n][e];
    }
#pragma unroll
    for (int n = 0; n < N; ++n) decay_add(s[n], cw + 16 * (n >> 1) + 2 * (n & 1), KP, d[n]);
}

// This lane's part of a state's 16 columns from key channel c0 on: N tiles.
template <int N>
__device__ __forceinline__ void load_state(float (&S)[N][4], const float *state, const DeltaChunkParams &p, int c0, int tg, bool on0, bool on1) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int ch = (i >> 1) * 16 + 4 * tg + (i & 1) * 2 + e;
            S[i][e] = on0 && c0 + ch < p.Dk ? state[(long long)ch * p.Dv] : 0.f;
            S[i][2 + e] = on1 && c0 + ch < p.Dk ? state[(long long)ch * p.Dv + 1] : 0.f;
        }
}
template <int N>
__device__ __forceinline__ void store_state(const float (&S)[N][4], float *state, const DeltaChunkParams &p, int c0, int tg, bool on0, bool on1) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int ch = (i >> 1) * 16 + 4 * tg + (i & 1) * 2 + e;
            if (on0 && c0 + ch < p.Dk) state[(long long)ch * p.Dv] = S[i][e];
            if (on1 && c0 + ch < p.Dk) state[(long long)ch * p.Dv + 1] = S[i][2 + e];
        }
}
// The pair of columns of a token (two values or outputs), whole where rows allow it.
__device__ __forceinline__ uint32_t value_pair(const __nv_bfloat16 *at, bool pairs, bool on0, bool on1) {
    if (pairs) return on0 ? *reinterpret_cast<const uint32_t *>(at) : 0u;
    const uint32_t lo = on0 ? *reinterpret_cast<const uint16_t *>(at) : 0u;
    return lo | (on1 ? (uint32_t)*reinterpret_cast<const uint16_t *>(at + 1) << 16 : 0u);
}
__device__ __forceinline__ void put_pair(float *at, float2 o, bool pairs, bool on0, bool on1) {
    if (pairs) {
        if (on0) *reinterpret_cast<float2 *>(at) = o;
    } else {
        if (on0) at[0] = o.x;
        if (on1) at[1] = o.y;
    }
}

// Many heads: a warp takes 16 columns by itself, the CTA's warps share the records between their columns.
template <int KP>
__global__ void __launch_bounds__(128) delta_chunk_kernel(const DeltaChunkParams p) {
    constexpr int J = KP / 16, RS = KP, REC = dc_record(KP);
    extern __shared__ __align__(128) float dc_smem[];
    __shared__ uint64_t bar[DC_RING];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tg = lane & 3;
    const int h = blockIdx.x / p.n_cols, b = blockIdx.y;
    const int col = ((blockIdx.x % p.n_cols) * (blockDim.x >> 5) + warp) * 16 + 2 * g;  // this lane's columns: col, col + 1
    const bool on0 = col < p.Dv, on1 = col + 1 < p.Dv, pairs = p.pairs != 0;
    const float *src = p.records + ((long long)b * p.H + h) * p.n_chunks * REC;
    auto fetch = [&](int i) {  // by one thread
        mbar_arrive_expect_tx(&bar[i % DC_RING], REC * 4);
        bulk_load(dc_smem + (i % DC_RING) * REC, src + (long long)i * REC, REC * 4, &bar[i % DC_RING]);
    };
    int fetched = 0;
    if (tid == 0) {
        for (int i = 0; i < DC_RING; ++i) mbar_init(&bar[i], 1);
        fence_mbar_init();
        for (; fetched < DC_RING && fetched < p.n_chunks; ++fetched) fetch(fetched);
    }
    float S[2 * J][4];
    float *state = p.state + ((long long)b * p.H + h) * p.Dk * p.Dv + col;
    load_state(S, state, p, 0, tg, on0, on1);
    // tokens 2 tg, 2 tg + 1, 8 + 2 tg, 9 + 2 tg of a chunk are this lane's; `left`: tokens from its first one on
    const __nv_bfloat16 *v = p.v + ((long long)b * p.T + 2 * tg) * p.v_stride + (long long)h * p.Dv + col;
    const long long out_row = (long long)p.H * p.Dv;
    float *out = p.out + ((long long)b * p.T + 2 * tg) * out_row + (long long)h * p.Dv + col;
    int left = p.T - 2 * tg;
    uint32_t v_raw[4];
    auto load_v = [&](int n) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int t = 8 * (s >> 1) + (s & 1);
            v_raw[s] = value_pair(v + t * p.v_stride, pairs, on0 && t < n, on1 && t < n);
        }
        v += CH_T * p.v_stride;
    };
    load_v(left);
    __syncthreads();

    bool failed = false;
    int slot = 0;
    uint32_t parity = 0;
    for (int i = 0; i < p.n_chunks; ++i) {
        int ok = __all_sync(0xffffffffu, mbar_try_wait(&bar[slot], parity));
        if (!ok) {
            if (lane == 0) ok = mbar_wait_bounded(&bar[slot], parity) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
        }
        failed = __syncthreads_or(!ok);  // behind it nobody reads the record before this one any more
        if (failed) break;
        if (tid == 0 && i > 0 && fetched < p.n_chunks) fetch(fetched++);
        const float *rec = dc_smem + slot * REC, *tail = rec + 2 * CH_T * RS + KP * CH_T + 2 * KP;
        // r[0], r[1]: u^T of tokens 0-7 and 8-15, r[2], r[3]: o^T
        float r[4][4], rb[4][4], ra[4][4];
        {
            uint32_t va[2][4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                va[s >> 1][(s & 1) * 2] = v_raw[s] << 16;
                va[s >> 1][(s & 1) * 2 + 1] = v_raw[s] & 0xffff0000u;
            }
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                r[m][0] = r[m][1] = r[m][2] = r[m][3] = 0.f;
                value_product(r[m], va, m, tail + (m >> 1) * CH_T * CH_T + (8 * (m & 1) + g) * CH_T + 4 * tg);
            }
        }
        if (i + 1 < p.n_chunks) load_v(left - CH_T);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const LeftFrag a0(S[2 * j]), a1(S[2 * j + 1]);
            const float *at = rec + ch_at<KP>(g, 16 * j + 4 * tg);
            rows_product<RS>(r, rb, ra, at, j == 0, a0, a1);
            rows_product<RS>(r + 2, rb + 2, ra + 2, at + CH_T * RS, j == 0, a0, a1);
        }
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) r[m][e] += rb[m][e] + ra[m][e];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int m = 2 + (s >> 1), e = s & 1, t = 8 * (s >> 1) + e;
            put_pair(out + t * out_row, make_float2(r[m][e], r[m][2 + e]), pairs, on0 && t < left, on1 && t < left);
        }
        out += CH_T * out_row;
        const LeftFrag u0(r[0]), u1(r[1]);
        const float *kt = rec + 2 * CH_T * RS, *cw = kt + KP * CH_T;
#pragma unroll
        for (int j = 0; j < J; j += 2)
            update_tiles<4, KP>(S + 2 * j, u0, u1, kt + (16 * j + 4 * (g >> 1) + (g & 1)) * CH_T + 4 * tg, cw + 16 * j + 4 * tg);
        left -= CH_T;
        if (++slot == DC_RING) {
            slot = 0;
            parity ^= 1u;
        }
    }
    if (failed) {
        if (tid == 0) {
            atomicOr(p.status, (int)NCKV_ST_TIMEOUT);
            // copies already issued land before the CTA's memory is released
            for (int f = fetched > DC_RING ? fetched - DC_RING : 0; f < fetched; ++f)
                mbar_wait_bounded(&bar[f % DC_RING], (f / DC_RING) & 1u, 100000000ull);
        }
        __syncthreads();
        return;
    }
    store_state(S, state, p, 0, tg, on0, on1);
}

// Few heads: a CTA takes 16 columns, and the chain from a chunk's state to the next is the bound.  NC warps hold 16 key channels
// each, two to a scheduler; their parts of u meet in shared memory, where every thread adds up one value (or two) and leaves it as two tf32
// terms.  A warp of its own keeps global memory off the chain: it fetches values and records ahead and adds up and stores the outputs of the
// chunk before.  (Waiting for values loaded a chunk ahead took 62 of 215 us at 1 x 2048 tokens and 12 heads, stores 24.)
constexpr int DC_V = 4;  // chunks of values in shared memory
template <int KP> constexpr int DC_NC = KP / 16;
__device__ __forceinline__ bool named_barrier_or(int id, int threads, bool bad) {
    uint32_t r;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %3, 0;\nbarrier.cta.red.or.pred q, %1, %2, p;\nselp.u32 %0, 1, 0, q;\n}"
                 : "=r"(r)
                 : "r"(id), "r"(threads), "r"((uint32_t)bad)
                 : "memory");
    return r != 0;
}
__device__ __forceinline__ void named_barrier(int id, int threads) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

template <int KP>
__global__ void __launch_bounds__(32 * DC_NC<KP> + 32) delta_chunk_split_kernel(const DeltaChunkParams p) {
    constexpr int NC = DC_NC<KP>, RS = KP, REC = dc_record(KP), PER = 8 / NC;  // PER: values of u a thread adds up
    static_assert(PER >= 1 && PER * NC == 8, "256 values over the warps");
    extern __shared__ __align__(128) float dc_smem[];
    __shared__ uint64_t bar[DC_RING];
    __shared__ __align__(16) float s_u[NC][2][32][4];     // parts of u
    __shared__ __align__(16) uint32_t s_whole[2][2][32][4];  // u: leading, low terms
    __shared__ __align__(16) float s_o[2][NC][2][32][4];  // parts of o
    __shared__ __align__(16) uint32_t s_v[DC_V][32][4];   // values, a pair of columns a word
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tg = lane & 3;
    const int h = blockIdx.x / p.n_cols, b = blockIdx.y, n = p.n_chunks;
    const int col = (blockIdx.x % p.n_cols) * 16 + 2 * g;  // this lane's columns: col, col + 1
    const bool on0 = col < p.Dv, on1 = col + 1 < p.Dv, pairs = p.pairs != 0;
    if (warp == NC) {
        const float *src = p.records + ((long long)b * p.H + h) * n * REC;
        auto fetch = [&](int i) {
            mbar_arrive_expect_tx(&bar[i % DC_RING], REC * 4);
            bulk_load(dc_smem + (i % DC_RING) * REC, src + (long long)i * REC, REC * 4, &bar[i % DC_RING]);
        };
        int fetched = 0;
        if (lane == 0) {
            for (int i = 0; i < DC_RING; ++i) mbar_init(&bar[i], 1);
            fence_mbar_init();
            for (; fetched < DC_RING && fetched < n; ++fetched) fetch(fetched);
        }
        const long long row = (long long)b * p.T + 2 * tg, out_row = (long long)p.H * p.Dv;
        const __nv_bfloat16 *v = p.v + row * p.v_stride + (long long)h * p.Dv + col;
        float *out = p.out + row * out_row + (long long)h * p.Dv + col;
        int v_left = p.T - 2 * tg, left = v_left;  // tokens from this lane's first one of the chunk on
        auto values = [&](int i) {  // of chunk i, on their way
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int t = 8 * (s >> 1) + (s & 1);
                const __nv_bfloat16 *at = v + t * p.v_stride;
                uint32_t *to = &s_v[i % DC_V][lane][s];
                const bool in = t < v_left;
                if (pairs)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(to)), "l"(in && on0 ? at : p.v), "r"(in && on0 ? 4 : 0) : "memory");
                else
                    *to = value_pair(at, false, in && on0, in && on1);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            v += CH_T * p.v_stride;
            v_left -= CH_T;
        };
        auto outputs = [&](int i) {  // of chunk i
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                float4 sum = *reinterpret_cast<const float4 *>(s_o[i & 1][0][m][lane]);
#pragma unroll
                for (int w = 1; w < NC; ++w) {
                    const float4 f = *reinterpret_cast<const float4 *>(s_o[i & 1][w][m][lane]);
                    sum.x += f.x; sum.y += f.y; sum.z += f.z; sum.w += f.w;
                }
                put_pair(out + 8 * m * out_row, make_float2(sum.x, sum.z), pairs, on0 && 8 * m < left, on1 && 8 * m < left);
                put_pair(out + (8 * m + 1) * out_row, make_float2(sum.y, sum.w), pairs, on0 && 8 * m + 1 < left, on1 && 8 * m + 1 < left);
            }
            out += CH_T * out_row;
            left -= CH_T;
        };
#pragma unroll
        for (int i = 0; i < DC_V - 1; ++i) values(i);
        asm volatile("cp.async.wait_group %0;" ::"n"(DC_V - 2) : "memory");
        __syncthreads();
        bool failed = false;
        for (int i = 0; i < n && !failed; ++i) {
            asm volatile("cp.async.wait_group %0;" ::"n"(DC_V - 3) : "memory");  // the values of the next chunk are there
            failed = named_barrier_or(1, 32 * NC + 32, false);
            if (failed) break;
            // the chunk before is done with: its record, its values, its parts of o
            if (lane == 0 && i > 0 && fetched < n) fetch(fetched++);
            values(i + DC_V - 1);
            if (i > 0) outputs(i - 1);
        }
        if (failed) {
            if (lane == 0) {
                atomicOr(p.status, (int)NCKV_ST_TIMEOUT);
                // copies already issued land before the CTA's memory is released
                for (int f = fetched > DC_RING ? fetched - DC_RING : 0; f < fetched; ++f)
                    mbar_wait_bounded(&bar[f % DC_RING], (f / DC_RING) & 1u, 100000000ull);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (!failed) outputs(n - 1);
        return;
    }
    float S[2][4];
    float *state = p.state + (((long long)b * p.H + h) * p.Dk + 16 * warp) * p.Dv + col;
    load_state(S, state, p, 16 * warp, tg, on0, on1);
    __syncthreads();
    bool failed = false;
    int slot = 0;
    uint32_t parity = 0;
    for (int i = 0; i < n; ++i) {
        int ok = __all_sync(0xffffffffu, mbar_try_wait(&bar[slot], parity));
        if (!ok) {
            if (lane == 0) ok = mbar_wait_bounded(&bar[slot], parity) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
        }
        const float *rec = dc_smem + slot * REC, *tail = rec + 2 * CH_T * RS + KP * CH_T + 2 * KP, *at = rec + ch_at<KP>(g, 16 * warp + 4 * tg);
        // r[0], r[1]: this warp's part of u^T of tokens 0-7 and 8-15, r[2], r[3]: of o^T
        float r[4][4], rb[4][4], ra[4][4];
#pragma unroll
        for (int m = 0; m < 4; ++m) r[m][0] = r[m][1] = r[m][2] = r[m][3] = 0.f;
        if (ok && warp < 4) {  // what does not depend on the state: a part of eight tokens each
            const uint4 f = *reinterpret_cast<const uint4 *>(s_v[i % DC_V][lane]);
            const uint32_t va[2][4] = {{f.x << 16, f.x & 0xffff0000u, f.y << 16, f.y & 0xffff0000u},
                                       {f.z << 16, f.z & 0xffff0000u, f.w << 16, f.w & 0xffff0000u}};
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m == warp) value_product(r[m], va, m, tail + (m >> 1) * CH_T * CH_T + (8 * (m & 1) + g) * CH_T + 4 * tg);
        }
        const LeftFrag a0(S[0]), a1(S[1]);
        rows_product<RS>(r, rb, ra, at, true, a0, a1);
#pragma unroll
        for (int m = 0; m < 2; ++m)
            *reinterpret_cast<float4 *>(s_u[warp][m][lane]) = make_float4(r[m][0] + (rb[m][0] + ra[m][0]), r[m][1] + (rb[m][1] + ra[m][1]),
                                                                        r[m][2] + (rb[m][2] + ra[m][2]), r[m][3] + (rb[m][3] + ra[m][3]));
        failed = named_barrier_or(1, 32 * NC + 32, !ok);  // behind it nobody is busy with the chunk before
        if (failed) break;
        {
            const int at_u = (warp * 32 + lane) * PER;
            float sum[PER], part[NC][PER];
#pragma unroll
            for (int w = 0; w < NC; ++w)
#pragma unroll
                for (int e = 0; e < PER; ++e) part[w][e] = (&s_u[w][0][0][0])[at_u + e];
            // the outputs do not wait for u: their products fill the time until its parts are there
            rows_product<RS>(r + 2, rb + 2, ra + 2, at + CH_T * RS, true, a0, a1);
#pragma unroll
            for (int e = 0; e < PER; ++e) {
                sum[e] = part[0][e];
#pragma unroll
                for (int w = 1; w < NC; ++w) sum[e] += part[w][e];
                uint32_t hi, lo;
                split_tf32(sum[e], hi, lo);
                (&s_whole[0][0][0][0])[at_u + e] = hi;
                (&s_whole[1][0][0][0])[at_u + e] = lo;
            }
        }
        named_barrier(2, 32 * NC);
        LeftFrag u0, u1;
        u0.take(s_whole[0][0][lane], s_whole[1][0][lane]);
        u1.take(s_whole[0][1][lane], s_whole[1][1][lane]);
        const float *kt = rec + 2 * CH_T * RS, *cw = kt + KP * CH_T;
        update_tiles<2, KP>(S, u0, u1, kt + (16 * warp + 4 * (g >> 1) + (g & 1)) * CH_T + 4 * tg, cw + 16 * warp + 4 * tg);
#pragma unroll
        for (int m = 0; m < 2; ++m)
            *reinterpret_cast<float4 *>(s_o[i & 1][warp][m][lane]) =
                make_float4(r[2 + m][0] + (rb[2 + m][0] + ra[2 + m][0]), r[2 + m][1] + (rb[2 + m][1] + ra[2 + m][1]),
                            r[2 + m][2] + (rb[2 + m][2] + ra[2 + m][2]), r[2 + m][3] + (rb[2 + m][3] + ra[2 + m][3]));
        if (++slot == DC_RING) {
            slot = 0;
            parity ^= 1u;
        }
    }
    __syncthreads();
    if (!failed) store_state(S, state, p, 16 * warp, tg, on0, on1);
}

static int dc_pad(int Dk) { return Dk <= 32 ? 32 : (Dk <= 64 ? 64 : 128); }

template <int KP> static cudaError_t dc_run(DeltaChunkParams p, cudaStream_t s) {
    delta_chunk_prepare_kernel<KP><<<dim3(p.n_chunks * p.H, p.B), KP, 0, s>>>(p);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    constexpr int SMEM = DC_RING * dc_record(KP) * (int)sizeof(float);
    const int per_head = (p.Dv + 15) / 16;
    const long long groups = (long long)p.B * p.H * per_head;
    p.n_cols = per_head;
    // Warps share columns while all such CTAs fit the chip at once, two to an SM: 1024 tokens, heads of 128 x 128, 192 to 288 groups of 16
    // columns 100 to 102 us.  With more a second wave would follow; a warp to 16 columns takes 157 us for 384 to 576 groups, 267 for 768.
    if constexpr (KP >= 64) {
        if (groups <= 2LL * sm_count()) {
            e = cudaFuncSetAttribute(delta_chunk_split_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
            if (e != cudaSuccess) return e;
            delta_chunk_split_kernel<KP><<<dim3(p.H * per_head, p.B), 32 * DC_NC<KP> + 32, SMEM, s>>>(p);
            return cudaGetLastError();
        }
    }
    int warps = 1;
    while (warps < 4 && warps < per_head && (long long)p.B * p.H * ((per_head + 2 * warps - 1) / (2 * warps)) >= sm_count()) warps *= 2;
    p.n_cols = (per_head + warps - 1) / warps;
    e = cudaFuncSetAttribute(delta_chunk_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return e;
    delta_chunk_kernel<KP><<<dim3(p.H * p.n_cols, p.B), warps * 32, SMEM, s>>>(p);
    return cudaGetLastError();
}

}  // namespace nckv

extern "C" {

size_t nckv_delta_chunk_workspace_bytes(int B, int T, int H, int Dk) {
    using namespace nckv;
    if (B <= 0 || T <= 0 || H <= 0 || Dk <= 0 || Dk > 128) return 0;
    return sizeof(float) * (size_t)B * H * ((T + CH_T - 1) / CH_T) * dc_record(dc_pad(Dk));
}

int nckv_delta_chunk(const void *q, const void *k, const void *v, int64_t q_stride, int64_t k_stride, int64_t v_stride,
                     const float *x, int64_t x_stride, const float *x0, const float *rate, const void *b, int64_t b_stride,
                     float *out, float *state, int B, int T, int H, int G, int Dk, int Dv, void *workspace,
                     size_t workspace_bytes, int32_t *status, void *stream) {
    using namespace nckv;
    if (!q || !k || !v || !x || !x0 || !rate || !b || !out || !state || !status) {
        set_error("delta_chunk: null pointer argument");
        return NCKV_E_ARG;
    }
    if (B <= 0 || T <= 0 || H <= 0 || G <= 0 || H % G || Dk <= 0 || Dv <= 0 || B > 65535) {
        set_error("delta_chunk: size out of range (B=%d T=%d H=%d G=%d Dk=%d Dv=%d)", B, T, H, G, Dk, Dv);
        return NCKV_E_ARG;
    }
    if (Dk > 128) {
        set_error("delta_chunk: %d key channels per head unsupported (at most 128)", Dk);
        return NCKV_E_UNSUPPORTED;
    }
    if (!workspace || ((uintptr_t)workspace & 15) || workspace_bytes < nckv_delta_chunk_workspace_bytes(B, T, H, Dk)) {
        set_error("delta_chunk: workspace of %zu bytes given, %zu needed", workspace_bytes, nckv_delta_chunk_workspace_bytes(B, T, H, Dk));
        return NCKV_E_CAPACITY;
    }
    DeltaChunkParams p;
    p.q = static_cast<const __nv_bfloat16 *>(q); p.k = static_cast<const __nv_bfloat16 *>(k); p.v = static_cast<const __nv_bfloat16 *>(v);
    p.q_stride = q_stride; p.k_stride = k_stride; p.v_stride = v_stride;
    p.x = x; p.x_stride = x_stride; p.x0 = x0; p.rate = rate;
    p.b = static_cast<const __nv_bfloat16 *>(b); p.b_stride = b_stride;
    p.records = static_cast<float *>(workspace); p.state = state; p.out = out; p.status = status;
    p.B = B; p.T = T; p.H = H; p.G = G; p.Dk = Dk; p.Dv = Dv;
    p.n_chunks = (T + CH_T - 1) / CH_T; p.n_cols = 1;
    p.pairs = Dv % 2 == 0 && v_stride % 2 == 0 && (((uintptr_t)v & 3) | ((uintptr_t)out & 7)) == 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int KP = dc_pad(Dk);
    NCKV_CUDA_CHECK(KP == 32 ? dc_run<32>(p, s) : (KP == 64 ? dc_run<64>(p, s) : dc_run<128>(p, s)));
    return NCKV_OK;
}

}  // extern "C"
