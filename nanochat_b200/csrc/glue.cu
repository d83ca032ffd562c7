// Elementwise glue of the transformer trunk, fused per layer and bit-exact against the
// eager bf16 op sequence it replaces (every eager op computes in fp32 and rounds its result to bf16;
// the kernels round at the same points).
//
//   glue_row_kernel   one row (one token's residual vector, C channels) per CTA:
//                       a = x                      or  bf16(x + add)                  block residual (gpt.py:148-150)
//                       y = bf16(bf16(rl * a) + bf16(xl * x0))                        lambda mix     (gpt.py:457)
//                        or bf16(a - bf16(bl * xb))                                   backout        (gpt.py:466-467)
//                        or a
//                       n = bf16(y * rsqrt(mean_fp32(y^2) + eps))                     norm           (gpt.py:42-43)
//                     The fp32 sum of squares follows the order of torch's vectorised row kernel: a
//                     block of 32 x 4 threads, thread t accumulates the 4-element vectors t, t + 128,
//                     ... sequentially (fused multiply-add), then a shuffle-down tree inside each warp
//                     (offsets 16, 8, 4, 2, 1), then warps (0 += 2, 1 += 3), then 0 += 1.
//                     A row's operands are all loaded before anything is stored (NV vectors per thread,
//                     a template constant): stores that might alias kept each vector's loads behind the one before.
//   relu_sq_kernel    bf16(max(h, 0)^2)                                               MLP            (gpt.py:136)
//   ve_gate_kernel    bf16(v + bf16(bf16(3 * bf16(sigmoid(g))) * ve))                 value residual (gpt.py:92-95)
//   logit_cap_kernel  cap * tanh(float(z) * (1 / cap)), bf16 in, fp32 out               logits         (gpt.py:469-472)
//                     One pass over the logits (6 bytes each) where the eager ops take four (30 bytes each).
#include "vec_io.cuh"

namespace nckv {

constexpr int GLUE_THREADS = 128;  // 32 x 4, the block shape whose reduction order is reproduced
constexpr int GLUE_MAX_VEC = 16;   // vectors of 4 channels per thread: C <= 8192

struct GlueScalar {
    const void *at;  // on the device, fp32 or bf16, or null
    float value;     // without `at`
    bool f32;
};

struct GlueRowParams {
    const uint2 *x, *add, *x0, *xb;
    uint2 *out_sum, *out_x, *out_norm;
    GlueScalar rl, xl, bl;
    float eps;
    int C, mode;  // mode 0: y = a, 1: lambda mix, 2: backout
};

// A parameter on the device is read there by every launch, so that its owner may write or replace it between any two,
// replays of a graph included; rounded to bf16 as the eager multiply rounds it.
__device__ __forceinline__ float scalar_value(const GlueScalar &s) {
    if (!s.at) return s.value;
    return s.f32 ? round_bf16(*static_cast<const float *>(s.at)) : __bfloat162float(*static_cast<const __nv_bfloat16 *>(s.at));
}

__device__ __forceinline__ void unpack4(const uint2 &v, float (&f)[4]) {
    f[0] = bf16lo(v.x); f[1] = bf16hi(v.x);
    f[2] = bf16lo(v.y); f[3] = bf16hi(v.y);
}
__device__ __forceinline__ uint2 pack4(const float (&f)[4]) {
    uint2 v;
    v.x = pack_bf16x2(f[0], f[1]);
    v.y = pack_bf16x2(f[2], f[3]);
    return v;
}

// NV: vectors of 4 channels per thread
template <int NV>
__global__ void __launch_bounds__(GLUE_THREADS) glue_row_kernel(const GlueRowParams p) {
    __shared__ float s_buf[4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n_vec = p.C >> 2;
    const long long base = (long long)blockIdx.x * n_vec;
    const uint2 *second = p.mode == 1 ? p.x0 : p.xb;
    uint2 in[NV], in_add[NV], in_second[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = t + k * GLUE_THREADS;
        in[k] = in_add[k] = in_second[k] = make_uint2(0, 0);
        if (i < n_vec) {
            in[k] = p.x[base + i];
            if (p.add) in_add[k] = p.add[base + i];
            if (p.mode != 0) in_second[k] = second[base + i];
        }
    }
    const float rl = p.mode == 1 ? scalar_value(p.rl) : 0.f, second_l = p.mode == 1 ? scalar_value(p.xl) : p.mode == 2 ? scalar_value(p.bl) : 0.f;
    float y[NV][4];
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = t + k * GLUE_THREADS;
        if (i < n_vec) {
            float a[4];
            unpack4(in[k], a);
            if (p.add) {
                float b[4];
                unpack4(in_add[k], b);
#pragma unroll
                for (int e = 0; e < 4; ++e) a[e] = round_bf16(__fadd_rn(a[e], b[e]));
                if (p.out_sum) p.out_sum[base + i] = pack4(a);
            }
            if (p.mode != 0) {
                float z[4];
                unpack4(in_second[k], z);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    a[e] = p.mode == 1 ? round_bf16(__fadd_rn(round_bf16(__fmul_rn(rl, a[e])), round_bf16(__fmul_rn(second_l, z[e]))))
                                       : round_bf16(__fsub_rn(a[e], round_bf16(__fmul_rn(second_l, z[e]))));
            }
            if (p.out_x) p.out_x[base + i] = pack4(a);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                y[k][e] = a[e];
                acc = __fmaf_rn(a[e], a[e], acc);
            }
        }
    }
    if (!p.out_norm) return;  // uniform over the grid
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) acc = __fadd_rn(acc, __shfl_down_sync(0xffffffffu, acc, off));
    if (lane == 0 && warp >= 2) s_buf[warp - 2] = acc;
    __syncthreads();
    if (lane == 0 && warp < 2) acc = __fadd_rn(acc, s_buf[warp]);
    __syncthreads();
    if (lane == 0 && warp == 1) s_buf[0] = acc;
    __syncthreads();
    if (t == 0) s_buf[1] = __fadd_rn(acc, s_buf[0]);
    __syncthreads();
    const float rstd = rsqrtf(__fadd_rn(__fdiv_rn(s_buf[1], (float)p.C), p.eps));
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = t + k * GLUE_THREADS;
        if (i < n_vec) {
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = __fmul_rn(y[k][e], rstd);  // pack4 rounds to bf16
            p.out_norm[base + i] = pack4(o);
        }
    }
}

__global__ void __launch_bounds__(256) relu_sq_kernel(const uint4 *__restrict__ h, uint4 *__restrict__ out, long long n_vec) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_vec; i += (long long)gridDim.x * blockDim.x) {
        const uint4 v = h[i];
        uint4 o;
        const uint32_t in[4] = {v.x, v.y, v.z, v.w};
        uint32_t res[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float a = fmaxf(bf16lo(in[e]), 0.f), b = fmaxf(bf16hi(in[e]), 0.f);
            res[e] = pack_bf16x2(__fmul_rn(a, a), __fmul_rn(b, b));
        }
        o.x = res[0]; o.y = res[1]; o.z = res[2]; o.w = res[3];
        out[i] = o;
    }
}

// v, ve, v_out: (rows, Hkv, 128) bf16, v with its own row stride (it may be a column slice of a projection
// output); g: (rows, Hkv) bf16 (output of the gate's linear layer)
__global__ void __launch_bounds__(256) ve_gate_kernel(const uint4 *__restrict__ v, const __nv_bfloat16 *__restrict__ g,
                                                      const uint4 *__restrict__ ve, uint4 *__restrict__ v_out,
                                                      long long n_vec, int row_vecs, long long v_row_stride) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_vec; i += (long long)gridDim.x * blockDim.x) {
        const float lin = __bfloat162float(g[i >> 4]);  // 16 vectors of 8 channels per head
        const float sig = round_bf16(__fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-lin))));
        const float gate = round_bf16(__fmul_rn(3.0f, sig));
        const long long row = i / row_vecs;
        const uint4 a = v[row * v_row_stride + (i - row * row_vecs)], b = ve[i];
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
        uint32_t res[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float lo = __fadd_rn(bf16lo(av[e]), round_bf16(__fmul_rn(gate, bf16lo(bv[e]))));
            const float hi = __fadd_rn(bf16hi(av[e]), round_bf16(__fmul_rn(gate, bf16hi(bv[e]))));
            res[e] = pack_bf16x2(lo, hi);
        }
        uint4 o;
        o.x = res[0]; o.y = res[1]; o.z = res[2]; o.w = res[3];
        v_out[i] = o;
    }
}

// V elements at a time; rows of `cols` in an input of row stride `in_stride`
template <int V>
__global__ void __launch_bounds__(256) logit_cap_kernel(const __nv_bfloat16 *__restrict__ z, long long in_stride, float *__restrict__ out,
                                                        long long rows, int cols, float inv_cap, float cap) {
    const int per = cols / V;
    for (long long row = blockIdx.y; row < rows; row += gridDim.y) {
        const __nv_bfloat16 *src = z + row * in_stride;
        float *dst = out + row * cols;
        for (int i = blockIdx.x * 256 + threadIdx.x; i < per; i += gridDim.x * 256) {
            float v[V];
            get_v(src + (long long)i * V, v);
#pragma unroll
            for (int e = 0; e < V; ++e) v[e] = __fmul_rn(cap, tanhf(__fmul_rn(v[e], inv_cap)));
            put_v(dst + (long long)i * V, v);
        }
    }
}

}  // namespace nckv

extern "C" {

int nckv_glue_logit_cap(const void *z, int64_t z_row_stride, float *out, int64_t rows, int cols, float cap, void *stream) {
    using namespace nckv;
    if (!z || !out || rows <= 0 || cols <= 0 || z_row_stride < cols || !(cap > 0.f)) {
        set_error("glue_logit_cap: null pointer or bad size (rows=%lld cols=%d stride=%lld)", (long long)rows, cols, (long long)z_row_stride);
        return NCKV_E_ARG;
    }
    const bool vec = cols % 8 == 0 && z_row_stride % 8 == 0 && (((uintptr_t)z | (uintptr_t)out) & 15) == 0;
    const int per = vec ? cols / 8 : cols;
    const dim3 grid((unsigned)((per + 255) / 256), (unsigned)(rows < 65535 ? rows : 65535));
    const __nv_bfloat16 *in = static_cast<const __nv_bfloat16 *>(z);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (vec) logit_cap_kernel<8><<<grid, 256, 0, s>>>(in, z_row_stride, out, rows, cols, 1.f / cap, cap);
    else logit_cap_kernel<1><<<grid, 256, 0, s>>>(in, z_row_stride, out, rows, cols, 1.f / cap, cap);
    NCKV_CUDA_CHECK(cudaGetLastError());
    return NCKV_OK;
}

static int glue_mix_norm_impl(const void *x, const void *add, const void *x0, const void *x_backout, void *out_sum,
                              void *out_x, void *out_norm, int rows, int C, int mode, nckv::GlueScalar resid_lambda,
                              nckv::GlueScalar x0_lambda, nckv::GlueScalar backout_lambda, float eps, void *stream) {
    using namespace nckv;
    if (!x || rows <= 0 || (!out_x && !out_norm && !out_sum)) {
        set_error("glue_mix_norm: null pointer or non-positive row count");
        return NCKV_E_ARG;
    }
    if (C <= 0 || (C % 4) != 0 || C > 4 * GLUE_THREADS * GLUE_MAX_VEC) {
        set_error("glue_mix_norm: C=%d must be a multiple of 4 and at most %d", C, 4 * GLUE_THREADS * GLUE_MAX_VEC);
        return NCKV_E_UNSUPPORTED;
    }
    if (mode < 0 || mode > 2 || (mode == 1 && !x0) || (mode == 2 && !x_backout) || (out_sum && !add)) {
        set_error("glue_mix_norm: mode %d lacks its operand (1 needs x0, 2 needs x_backout; out_sum needs add)", mode);
        return NCKV_E_ARG;
    }
    const uintptr_t a = (uintptr_t)x | (uintptr_t)add | (uintptr_t)x0 | (uintptr_t)x_backout | (uintptr_t)out_sum |
                        (uintptr_t)out_x | (uintptr_t)out_norm;
    if ((a & 7) || ((C * 2) & 7)) {
        set_error("glue_mix_norm: rows must be 8-byte aligned");
        return NCKV_E_ARG;
    }
    GlueRowParams p;
    p.x = static_cast<const uint2 *>(x);
    p.add = static_cast<const uint2 *>(add);
    p.x0 = static_cast<const uint2 *>(x0);
    p.xb = static_cast<const uint2 *>(x_backout);
    p.out_sum = static_cast<uint2 *>(out_sum);
    p.out_x = static_cast<uint2 *>(out_x);
    p.out_norm = static_cast<uint2 *>(out_norm);
    p.rl = resid_lambda; p.xl = x0_lambda; p.bl = backout_lambda; p.eps = eps;
    p.C = C; p.mode = mode;
    const int nv = (C / 4 + GLUE_THREADS - 1) / GLUE_THREADS;
    const auto kernel = nv == 1 ? glue_row_kernel<1> : nv == 2 ? glue_row_kernel<2> : nv == 3 ? glue_row_kernel<3> : nv == 4 ? glue_row_kernel<4>
                        : nv <= 8 ? glue_row_kernel<8> : glue_row_kernel<GLUE_MAX_VEC>;
    kernel<<<rows, GLUE_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(p);
    NCKV_CUDA_CHECK(cudaGetLastError());
    return NCKV_OK;
}

int nckv_glue_mix_norm(const void *x, const void *add, const void *x0, const void *x_backout, void *out_sum,
                       void *out_x, void *out_norm, int rows, int C, int mode, float resid_lambda, float x0_lambda,
                       float backout_lambda, float eps, void *stream) {
    using nckv::GlueScalar;
    return glue_mix_norm_impl(x, add, x0, x_backout, out_sum, out_x, out_norm, rows, C, mode, GlueScalar{nullptr, resid_lambda, true},
                              GlueScalar{nullptr, x0_lambda, true}, GlueScalar{nullptr, backout_lambda, true}, eps, stream);
}

int nckv_glue_mix_norm_at(const void *x, const void *add, const void *x0, const void *x_backout, void *out_sum,
                          void *out_x, void *out_norm, int rows, int C, int mode, const void *resid_lambda,
                          const void *x0_lambda, const void *backout_lambda, int f32_mask, float eps, void *stream) {
    using nckv::GlueScalar;
    if ((mode == 1 && (!resid_lambda || !x0_lambda)) || (mode == 2 && !backout_lambda)) {
        nckv::set_error("glue_mix_norm: mode %d lacks a scalar", mode);
        return NCKV_E_ARG;
    }
    const void *at[3] = {resid_lambda, x0_lambda, backout_lambda};
    for (int i = 0; i < 3; ++i)
        if ((uintptr_t)at[i] & ((f32_mask >> i & 1) ? 3 : 1)) {
            nckv::set_error("glue_mix_norm: misaligned scalar");
            return NCKV_E_ARG;
        }
    return glue_mix_norm_impl(x, add, x0, x_backout, out_sum, out_x, out_norm, rows, C, mode, GlueScalar{resid_lambda, 0.f, (f32_mask & 1) != 0},
                              GlueScalar{x0_lambda, 0.f, (f32_mask & 2) != 0}, GlueScalar{backout_lambda, 0.f, (f32_mask & 4) != 0}, eps, stream);
}

int nckv_glue_relu_sq(const void *h, void *out, int64_t n, void *stream) {
    using namespace nckv;
    if (!h || !out || n <= 0 || (n % 8) != 0 || (((uintptr_t)h | (uintptr_t)out) & 15)) {
        set_error("glue_relu_sq: null/misaligned pointer or element count %lld not a positive multiple of 8", (long long)n);
        return NCKV_E_ARG;
    }
    const long long n_vec = n / 8;
    long long blocks = (n_vec + 255) / 256;
    const long long cap = (long long)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    relu_sq_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4 *>(h), static_cast<uint4 *>(out), n_vec);
    NCKV_CUDA_CHECK(cudaGetLastError());
    return NCKV_OK;
}

int nckv_glue_ve_gate(const void *v, int64_t v_row_stride, const void *gate_lin, const void *ve, void *v_out, int rows,
                      int Hkv, int D, void *stream) {
    using namespace nckv;
    if (!v || !gate_lin || !ve || !v_out || rows <= 0 || Hkv <= 0) {
        set_error("glue_ve_gate: null pointer or non-positive size");
        return NCKV_E_ARG;
    }
    if (D != NCKV_D) {
        set_error("glue_ve_gate: head_dim %d unsupported (kernels are built for 128)", D);
        return NCKV_E_UNSUPPORTED;
    }
    if (v_row_stride == 0) v_row_stride = (int64_t)Hkv * D;
    if (v_row_stride % 8 || v_row_stride < (int64_t)Hkv * D) {
        set_error("glue_ve_gate: v_row_stride must be a multiple of 8 elements and span a row's heads");
        return NCKV_E_ARG;
    }
    if (((uintptr_t)v | (uintptr_t)ve | (uintptr_t)v_out) & 15) {
        set_error("glue_ve_gate: tensors must be 16-byte aligned");
        return NCKV_E_ARG;
    }
    const long long n_vec = (long long)rows * Hkv * (NCKV_D / 8);
    long long blocks = (n_vec + 255) / 256;
    const long long cap = (long long)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    ve_gate_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4 *>(v), static_cast<const __nv_bfloat16 *>(gate_lin), static_cast<const uint4 *>(ve),
        static_cast<uint4 *>(v_out), n_vec, Hkv * (NCKV_D / 8), (long long)(v_row_stride / 8));
    NCKV_CUDA_CHECK(cudaGetLastError());
    return NCKV_OK;
}

}  // extern "C"
