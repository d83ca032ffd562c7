// Kernel (a): fused RoPE + QK rms-norm + scale + KV append, bit-exact against the eager bf16 path.
//
// One half-warp handles head rows of one token of q, k or v: lane j of its 16 holds channels 4j .. 4j + 3 and
// 64 + 4j .. 64 + 4j + 3, the two sides of its rotation pairs (8-byte loads and stores, 128 contiguous bytes per
// half-warp), so the rotation crosses no lanes.  The arithmetic reproduces, rounding for rounding,
// the reference's op sequence on bf16 tensors:
//   apply_rotary_emb (gpt.py:57-63):  y1 = bf16(bf16(x1*cos) + bf16(x2*sin))
//                                     y2 = bf16(bf16(x1*(-sin)) + bf16(x2*cos))
//   norm (gpt.py:42-43):              z  = bf16(y * rsqrt(mean_fp32(y^2) + eps))
//   scale (gpt.py:101-102):           out = bf16(float(z) * 1.2f)
// The fp32 sum of squares is accumulated in the order of torch's vectorised row kernel for a
// 128-wide row (32 lanes x 4 consecutive elements, sequential within a lane, then a
// shuffle-down tree with offsets 16, 8, 4, 2, 1), so that rstd carries the same last bit.
#include "rope_row.cuh"

namespace nckv {

struct AppendParams {
    const uint4 *q_in;
    const uint4 *k_in;
    const uint4 *v_in;
    uint4 *q_out;
    __nv_bfloat16 *k_cache;
    __nv_bfloat16 *v_cache;
    const int32_t *cache_seqlens;
    const int32_t *write_slots;  // optional: cache index of token 0 per row (-1: do not write); null = cache_seqlens
    const uint4 *cos;  // (rope_len, 64) bf16 = 8 uint4 per position
    const uint4 *sin;
    int32_t *status;
    int B, T_new, Hq, Hkv, T_max, rope_len;
    int64_t cache_batch_stride, cache_token_stride;
    float qk_scale, eps;
    int transform_k;  // 0: k is stored as given (plain append)
    KvSplit split;    // block > 0: block-cyclic sequence split, the owner of position cache_seqlens[b] stores k/v
    // paged storage (block_table != null): the caches are page pools (n_pages, page_tokens, Hkv, D);
    // T_max is then max_pages * page_tokens and cache_batch_stride the distance between pages
    const int32_t *block_table;
    int page_tokens, max_pages, n_pages;
    // distance between the tokens of q_in / k_in / v_in in 16-byte units (heads of a token are packed); lets the
    // three be column slices of one projection output
    long long q_stride, k_stride, v_stride;
    int per_tok;  // half-warps per token
};

// NB: head rows a half-warp takes, all of one token and loaded together (rows first, first + per_tok, ...).
template <int NB>
__global__ void __launch_bounds__(256) append_rope_norm_kernel(const AppendParams p) {
    // Programmatic dependent launch: this grid may have been scheduled while its predecessor was
    // still running; its inputs come from that predecessor, so wait before touching anything.
    // The attention kernel that follows may be scheduled right away, even before that wait: it
    // reads only cache_seqlens and older cache rows until it has itself waited for this grid.
    pdl_launch_dependents();
    pdl_wait_prior_grids();
    const int j = threadIdx.x & 15;
    const int q_heads = p.q_in ? p.Hq : 0, heads_per_tok = q_heads + 2 * p.Hkv;
    const unsigned half_warp = half_warp_of(blockIdx.x, threadIdx.x), n_tok = (unsigned)p.B * (unsigned)p.T_new;
    unsigned tok = half_warp / (unsigned)p.per_tok;
    const int first = (int)(half_warp - tok * (unsigned)p.per_tok);
    const bool live = tok < n_tok;
    if (!live) tok = n_tok - 1;  // stays for the shuffles
    const int b = (int)(tok / (unsigned)p.T_new), t = (int)(tok - (unsigned)b * (unsigned)p.T_new);
    // the input rows do not depend on the row's length: their loads go out together with the
    // length's, one round trip ahead of the table rows that do
    uint2 lo[NB], hi[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int slot = first + i * p.per_tok;
        lo[i] = hi[i] = make_uint2(0, 0);
        if (!live || slot >= heads_per_tok) continue;
        // kind: 0 = q head, 1 = k head, 2 = v head
        const int kind = slot < q_heads ? 0 : (slot < q_heads + p.Hkv ? 1 : 2);
        const int h = slot - (kind == 0 ? 0 : (kind == 1 ? q_heads : q_heads + p.Hkv));
        const uint4 *row = (kind == 0 ? p.q_in : (kind == 1 ? p.k_in : p.v_in)) +
                           tok * (kind == 0 ? p.q_stride : (kind == 1 ? p.k_stride : p.v_stride)) + h * 16;
        lo[i] = reinterpret_cast<const uint2 *>(row)[j];
        hi[i] = reinterpret_cast<const uint2 *>(row)[16 + j];
    }
    const int len = p.cache_seqlens[b];          // sequence position of token 0 (drives RoPE)
    int wslot = p.write_slots ? p.write_slots[b] : len;  // cache index of token 0
    if (p.split.block > 0 && len >= 0)
        wslot = (len / p.split.block) % p.split.world == p.split.rank
                    ? owned_below(len, p.split.world, p.split.rank, p.split.block) : -1;
    bool ok = live;
    if (len < 0 || wslot < -1) {
        if (live && j == 0 && first == 0 && t == 0) atomicOr(p.status, (int)NCKV_ST_BAD_SEQLEN);
        ok = false;
    } else if ((wslot >= 0 && wslot + p.T_new > p.T_max) || (p.rope_len > 0 && len + p.T_new > p.rope_len)) {
        if (live && j == 0 && first == 0 && t == 0) atomicOr(p.status, (int)NCKV_ST_OVERFLOW);
        ok = false;
    }
    const bool write_kv = ok && wslot >= 0;  // -1: this row's token belongs to another shard
    uint2 c = make_uint2(0, 0), s = make_uint2(0, 0);
    if (ok && p.rope_len > 0) {
        const long long at = (long long)(len + t) * 16 + j;
        c = reinterpret_cast<const uint2 *>(p.cos)[at];
        s = reinterpret_cast<const uint2 *>(p.sin)[at];
    }
    long long dst_off = 0;  // of the token's heads in the caches
    bool in_cache = write_kv;
    if (write_kv) {
        long long outer = b, at = wslot + t;
        if (p.block_table) {  // row -> page
            const int idx = (int)(at / p.page_tokens);
            at -= (long long)idx * p.page_tokens;
            outer = p.block_table[(long long)b * p.max_pages + idx];
            if (outer < 0 || outer >= p.n_pages) {
                if (j == 0 && first == 0) atomicOr(p.status, (int)NCKV_ST_BAD_PAGE);
                in_cache = false;
            }
        }
        dst_off = outer * p.cache_batch_stride + at * p.cache_token_stride;
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int slot = first + i * p.per_tok;
        const int kind = slot < q_heads ? 0 : (slot < q_heads + p.Hkv ? 1 : 2);
        const int h = slot - (kind == 0 ? 0 : (kind == 1 ? q_heads : q_heads + p.Hkv));
        const bool transform = kind == 0 || (kind == 1 && p.transform_k);
        // the two half-warps may hold different kinds, and the transform shuffles across the warp
        if (__any_sync(0xffffffffu, transform)) {
            uint2 a = lo[i], d = hi[i];
            rope_norm_scale(a, d, c, s, p.qk_scale, p.eps);
            if (transform) {
                lo[i] = a;
                hi[i] = d;
            }
        }
        if (slot >= heads_per_tok || !ok || (kind != 0 && !in_cache)) continue;
        uint2 *dst = kind == 0 ? reinterpret_cast<uint2 *>(p.q_out + ((long long)tok * p.Hq + h) * 16)
                               : reinterpret_cast<uint2 *>((kind == 1 ? p.k_cache : p.v_cache) + dst_off + (long long)h * NCKV_D);
        dst[j] = lo[i];
        dst[16 + j] = hi[i];
    }
}

static int check_common(const void *k_in, const void *v_in, void *k_cache, void *v_cache,
                        const int32_t *cache_seqlens, int B, int T_new, int Hkv, int D, int T_max,
                        int64_t bs, int64_t ts, int32_t *status) {
    if (!k_in || !v_in || !k_cache || !v_cache || !cache_seqlens || !status) {
        set_error("append: null pointer argument");
        return NCKV_E_ARG;
    }
    if (B <= 0 || T_new <= 0 || Hkv <= 0 || T_max <= 0) {
        set_error("append: non-positive size (B=%d T_new=%d Hkv=%d T_max=%d)", B, T_new, Hkv, T_max);
        return NCKV_E_ARG;
    }
    if (D != NCKV_D) {
        set_error("append: head_dim %d unsupported (kernels are built for 128)", D);
        return NCKV_E_UNSUPPORTED;
    }
    if (T_new > T_max) {
        set_error("append: T_new=%d exceeds cache capacity T_max=%d", T_new, T_max);
        return NCKV_E_CAPACITY;
    }
    if (ts < (int64_t)Hkv * D || (ts % 8) != 0 || (bs % 8) != 0) {
        set_error("append: cache strides must be multiples of 8 elements, token stride >= Hkv*D");
        return NCKV_E_ARG;
    }
    const uintptr_t a = (uintptr_t)k_in | (uintptr_t)v_in | (uintptr_t)k_cache | (uintptr_t)v_cache;
    if (a & 15) {
        set_error("append: tensors must be 16-byte aligned");
        return NCKV_E_ARG;
    }
    return NCKV_OK;
}

// Rows per half-warp.  Few rows (a decode step): one each, the shortest chain from the input to the store.  From
// APPEND_WIDE_ROWS head rows on the chip is full either way, and four rows share the index arithmetic and the
// token's table row.  us with one / with four: 1536 head rows 7.2 / 9.2, 16800 10.8 / 11.2, 24000 11.2 / 11.2, 33600 13.3 /
// 13.2, 49152 17 / 15.4, 110232 27.6 / 23.5, 589824 108.5 / 84.5 (one row each with the two sides of a rotation pair in different
// lanes: 9.2, 13.2, 16.8, 19.4, 23.5, 42, 188).
constexpr long long APPEND_WIDE_ROWS = 32768;

static int launch_append(AppendParams p, cudaStream_t stream) {
    const int heads_per_tok = (p.q_in ? p.Hq : 0) + 2 * p.Hkv;
    const bool wide = (long long)p.B * p.T_new * heads_per_tok >= APPEND_WIDE_ROWS;
    p.per_tok = wide ? (heads_per_tok + 3) / 4 : heads_per_tok;
    const long long half_warps = (long long)p.B * p.T_new * p.per_tok;
    if (half_warps > HALF_WARPS_MOST) {  // a terabyte of rows and more
        set_error("append: B=%d x T_new=%d tokens are too many for one launch", p.B, p.T_new);
        return NCKV_E_UNSUPPORTED;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((half_warps + 15) / 16));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NCKV_CUDA_CHECK(cudaLaunchKernelEx(&cfg, wide ? append_rope_norm_kernel<4> : append_rope_norm_kernel<1>, p));
    return NCKV_OK;
}

}  // namespace nckv

extern "C" {

static int append_rope_norm_impl(const void *q_in, const void *k_in, const void *v_in, void *q_out,
                                 void *k_cache, void *v_cache, const int32_t *cache_seqlens,
                                 const int32_t *write_slots, nckv::KvSplit split, const void *cos, const void *sin, int B, int T_new,
                                 int Hq, int Hkv, int D, int T_max, int64_t cache_batch_stride,
                                 int64_t cache_token_stride, int rope_len, float qk_scale, float eps,
                                 int32_t *status, void *stream, const int32_t *block_table = nullptr,
                                 int page_tokens = 0, int max_pages = 0, int n_pages = 0, int64_t q_token_stride = 0,
                                 int64_t k_token_stride = 0, int64_t v_token_stride = 0) {
    using namespace nckv;
    if ((q_token_stride && (q_token_stride % 8 || q_token_stride < (int64_t)Hq * D)) ||
        (k_token_stride && (k_token_stride % 8 || k_token_stride < (int64_t)Hkv * D)) ||
        (v_token_stride && (v_token_stride % 8 || v_token_stride < (int64_t)Hkv * D))) {
        set_error("append_rope_norm: token strides must be multiples of 8 elements and span a token's heads");
        return NCKV_E_ARG;
    }
    int rc = check_common(k_in, v_in, k_cache, v_cache, cache_seqlens, B, T_new, Hkv, D, T_max,
                          cache_batch_stride, cache_token_stride, status);
    if (rc != NCKV_OK) return rc;
    if (!cos || !sin || rope_len <= 0) {
        set_error("append_rope_norm: cos/sin tables are required");
        return NCKV_E_ARG;
    }
    if (q_in && (!q_out || Hq <= 0 || (Hq % Hkv) != 0)) {
        set_error("append_rope_norm: q given but q_out missing or Hq=%d not a multiple of Hkv=%d", Hq, Hkv);
        return NCKV_E_ARG;
    }
    if (((uintptr_t)cos | (uintptr_t)sin | (uintptr_t)q_in | (uintptr_t)q_out) & 15) {
        set_error("append_rope_norm: tensors must be 16-byte aligned");
        return NCKV_E_ARG;
    }
    AppendParams p;
    p.q_in = static_cast<const uint4 *>(q_in);
    p.k_in = static_cast<const uint4 *>(k_in);
    p.v_in = static_cast<const uint4 *>(v_in);
    p.q_out = static_cast<uint4 *>(q_out);
    p.k_cache = static_cast<__nv_bfloat16 *>(k_cache);
    p.v_cache = static_cast<__nv_bfloat16 *>(v_cache);
    p.cache_seqlens = cache_seqlens;
    p.write_slots = write_slots;
    p.cos = static_cast<const uint4 *>(cos);
    p.sin = static_cast<const uint4 *>(sin);
    p.status = status;
    p.B = B; p.T_new = T_new; p.Hq = Hq; p.Hkv = Hkv; p.T_max = T_max; p.rope_len = rope_len;
    p.cache_batch_stride = cache_batch_stride;
    p.cache_token_stride = cache_token_stride;
    p.qk_scale = qk_scale;
    p.eps = eps;
    p.transform_k = 1;
    p.split = split;
    p.block_table = block_table;
    p.page_tokens = page_tokens; p.max_pages = max_pages; p.n_pages = n_pages;
    p.q_stride = q_token_stride ? q_token_stride / 8 : (long long)Hq * 16;
    p.k_stride = k_token_stride ? k_token_stride / 8 : (long long)Hkv * 16;
    p.v_stride = v_token_stride ? v_token_stride / 8 : (long long)Hkv * 16;
    return launch_append(p, static_cast<cudaStream_t>(stream));
}

int nckv_append_rope_norm_strided(const void *q_in, const void *k_in, const void *v_in, int64_t q_token_stride,
                                  int64_t k_token_stride, int64_t v_token_stride, void *q_out, void *k_cache,
                                  void *v_cache, const int32_t *cache_seqlens, const void *cos, const void *sin, int B,
                                  int T_new, int Hq, int Hkv, int D, int T_max, int64_t cache_batch_stride,
                                  int64_t cache_token_stride, int rope_len, float qk_scale, float eps, int32_t *status,
                                  void *stream) {
    if (((uintptr_t)k_in | (uintptr_t)v_in) & 15) {
        nckv::set_error("append_rope_norm_strided: tensors must be 16-byte aligned");
        return NCKV_E_ARG;
    }
    return append_rope_norm_impl(q_in, k_in, v_in, q_out, k_cache, v_cache, cache_seqlens, nullptr, nckv::KvSplit{0, 0, 0}, cos,
                                 sin, B, T_new, Hq, Hkv, D, T_max, cache_batch_stride, cache_token_stride, rope_len,
                                 qk_scale, eps, status, stream, nullptr, 0, 0, 0, q_token_stride, k_token_stride,
                                 v_token_stride);
}

int nckv_append_rope_norm(const void *q_in, const void *k_in, const void *v_in, void *q_out,
                          void *k_cache, void *v_cache, const int32_t *cache_seqlens,
                          const void *cos, const void *sin, int B, int T_new, int Hq, int Hkv,
                          int D, int T_max, int64_t cache_batch_stride,
                          int64_t cache_token_stride, int rope_len, float qk_scale, float eps,
                          int32_t *status, void *stream) {
    return append_rope_norm_impl(q_in, k_in, v_in, q_out, k_cache, v_cache, cache_seqlens, nullptr, nckv::KvSplit{0, 0, 0}, cos, sin, B, T_new,
                                 Hq, Hkv, D, T_max, cache_batch_stride, cache_token_stride, rope_len, qk_scale, eps,
                                 status, stream);
}

int nckv_append_rope_norm_at(const void *q_in, const void *k_in, const void *v_in, void *q_out,
                             void *k_cache, void *v_cache, const int32_t *positions, const int32_t *write_slots,
                             const void *cos, const void *sin, int B, int T_new, int Hq, int Hkv,
                             int D, int T_max, int64_t cache_batch_stride, int64_t cache_token_stride,
                             int rope_len, float qk_scale, float eps, int32_t *status, void *stream) {
    if (!write_slots) {
        nckv::set_error("append_rope_norm_at: write_slots is required");
        return NCKV_E_ARG;
    }
    return append_rope_norm_impl(q_in, k_in, v_in, q_out, k_cache, v_cache, positions, write_slots, nckv::KvSplit{0, 0, 0}, cos, sin, B, T_new,
                                 Hq, Hkv, D, T_max, cache_batch_stride, cache_token_stride, rope_len, qk_scale, eps,
                                 status, stream);
}

int nckv_append_rope_norm_split(const void *q_in, const void *k_in, const void *v_in, void *q_out,
                                void *k_cache, void *v_cache, const int32_t *cache_seqlens, const void *cos,
                                const void *sin, int B, int T_new, int Hq, int Hkv, int D, int T_local,
                                int64_t cache_batch_stride, int64_t cache_token_stride, int rope_len,
                                float qk_scale, float eps, int world, int rank, int block, int32_t *status,
                                void *stream) {
    if (world <= 0 || rank < 0 || rank >= world || block <= 0 || T_new != 1) {
        nckv::set_error("append_rope_norm_split: bad split (world=%d rank=%d block=%d) or T_new=%d != 1", world, rank,
                        block, T_new);
        return NCKV_E_ARG;
    }
    return append_rope_norm_impl(q_in, k_in, v_in, q_out, k_cache, v_cache, cache_seqlens, nullptr,
                                 nckv::KvSplit{world, rank, block}, cos, sin, B, T_new, Hq, Hkv, D, T_local,
                                 cache_batch_stride, cache_token_stride, rope_len, qk_scale, eps, status, stream);
}

int nckv_append_rope_norm_paged(const void *q_in, const void *k_in, const void *v_in, void *q_out, void *k_pool,
                                void *v_pool, const int32_t *block_table, const int32_t *cache_seqlens,
                                const void *cos, const void *sin, int B, int T_new, int Hq, int Hkv, int D,
                                int page_tokens, int max_pages, int n_pages, int64_t page_stride, int64_t token_stride,
                                int rope_len, float qk_scale, float eps, int32_t *status, void *stream) {
    if (!block_table || page_tokens <= 0 || max_pages <= 0 || n_pages <= 0 ||
        (long long)page_tokens * max_pages > 0x3fffffffLL) {
        nckv::set_error("append_rope_norm_paged: bad paging (page_tokens=%d max_pages=%d n_pages=%d)", page_tokens,
                        max_pages, n_pages);
        return NCKV_E_ARG;
    }
    return append_rope_norm_impl(q_in, k_in, v_in, q_out, k_pool, v_pool, cache_seqlens, nullptr, nckv::KvSplit{0, 0, 0},
                                 cos, sin, B, T_new, Hq, Hkv, D, page_tokens * max_pages, page_stride, token_stride,
                                 rope_len, qk_scale, eps, status, stream, block_table, page_tokens, max_pages, n_pages);
}

int nckv_append(const void *k_in, const void *v_in, void *k_cache, void *v_cache,
                const int32_t *cache_seqlens, int B, int T_new, int Hkv, int D, int T_max,
                int64_t cache_batch_stride, int64_t cache_token_stride, int32_t *status,
                void *stream) {
    using namespace nckv;
    int rc = check_common(k_in, v_in, k_cache, v_cache, cache_seqlens, B, T_new, Hkv, D, T_max,
                          cache_batch_stride, cache_token_stride, status);
    if (rc != NCKV_OK) return rc;
    AppendParams p;
    p.q_in = nullptr;
    p.k_in = static_cast<const uint4 *>(k_in);
    p.v_in = static_cast<const uint4 *>(v_in);
    p.q_out = nullptr;
    p.k_cache = static_cast<__nv_bfloat16 *>(k_cache);
    p.v_cache = static_cast<__nv_bfloat16 *>(v_cache);
    p.cache_seqlens = cache_seqlens;
    p.write_slots = nullptr;
    p.cos = nullptr;
    p.sin = nullptr;
    p.status = status;
    p.B = B; p.T_new = T_new; p.Hq = 0; p.Hkv = Hkv; p.T_max = T_max; p.rope_len = 0;
    p.cache_batch_stride = cache_batch_stride;
    p.cache_token_stride = cache_token_stride;
    p.qk_scale = 1.0f;
    p.eps = 0.0f;
    p.transform_k = 0;
    p.split = KvSplit{0, 0, 0};
    p.block_table = nullptr;
    p.page_tokens = p.max_pages = p.n_pages = 0;
    p.q_stride = 0;
    p.k_stride = p.v_stride = (long long)Hkv * 16;
    return launch_append(p, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
