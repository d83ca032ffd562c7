// The calls a decode step repeats most, from torch tensors to libnckv's C entry points without the interpreter in
// between: the checks, the outputs' allocation and the launches of one kv_attention cost about 40 us as Python
// statements over ctypes and a few as C++, beside 13 us of kernels on the smallest shapes.
//
// Every function here takes the plain case only and returns None for anything else (other dtypes, strides or devices, a
// missing workspace, sizes that do not fit, a call that the library refused); the caller then takes the general Python
// path, which decides what is wrong and says so.  The interpreter lock is given up once the arguments have been looked at: an
// allocation or a launch may wait for the device, and other threads run meanwhile.  Nothing is kept between calls but the table of workspaces, which mirrors the caller's.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <map>
#include <optional>
#include <utility>

#include "../../include/nckv.h"

namespace {

using at::Tensor;
constexpr int64_t D = 128;

// (device, stream) -> scratch, as registered by the caller; guarded by the interpreter lock.  Never destroyed: the
// tensors must not outlive the CUDA context at exit.
std::map<std::pair<int, uintptr_t>, Tensor> &workspaces() {
    static auto *m = new std::map<std::pair<int, uintptr_t>, Tensor>();
    return *m;
}

void set_workspace(int device, uintptr_t stream, const Tensor &ws) { workspaces()[{device, stream}] = ws; }

bool bf16_on(const Tensor &t, const c10::Device &dev) { return t.scalar_type() == at::kBFloat16 && t.device() == dev; }

// Token stride of (B, T, H, D) activations with packed heads, or -1.
int64_t token_stride(const Tensor &t) {
    const int64_t T = t.size(1);
    if (t.stride(3) != 1 || t.stride(2) != D || (T > 1 && t.stride(0) != T * t.stride(1))) return -1;
    const int64_t s = T > 1 ? t.stride(1) : t.stride(0);
    return s % 8 == 0 && s >= t.size(2) * D && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0 ? s : -1;
}

struct Launch {
    cudaStream_t stream;
    Tensor ws;
};

std::optional<Launch> launch_on(const c10::Device &dev, int B, int Hq, int Hkv) {
    const cudaStream_t s = at::cuda::getCurrentCUDAStream(dev.index()).stream();
    const auto it = workspaces().find({dev.index(), reinterpret_cast<uintptr_t>(s)});
    if (it == workspaces().end()) return std::nullopt;
    const size_t need = nckv_workspace_bytes(B, Hq, Hkv, (int)D);
    if (need == 0 || (size_t)it->second.numel() < need) return std::nullopt;
    return Launch{s, it->second};
}

// Append and attention of one layer, dense cache: nckv_append_rope_norm, then nckv_decode_attn (one new token per row; few rows and short
// caches: nckv_decode_small alone) or nckv_prefill_attn.  block_table: the caches are page pools (one new token per row).
std::optional<Tensor> kv_attention(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &k_cache, const Tensor &v_cache,
                                   const std::optional<Tensor> &block_table, const Tensor &seqlens, const Tensor &cos, const Tensor &sin,
                                   int64_t window_left, double qk_scale, double eps) {
    if (!q.is_cuda() || q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || k_cache.dim() != 4 || v_cache.dim() != 4 || seqlens.dim() != 1)
        return std::nullopt;
    const c10::Device dev = q.device();
    for (const Tensor *t : {&q, &k, &v, &k_cache, &v_cache, &cos, &sin})
        if (!bf16_on(*t, dev)) return std::nullopt;
    const int64_t B = q.size(0), T = q.size(1), Hq = q.size(2), Hkv = k.size(2);
    if (B <= 0 || T <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || q.size(3) != D || k.size(0) != B || k.size(1) != T || k.size(3) != D ||
        v.sizes() != k.sizes() || seqlens.scalar_type() != at::kInt || seqlens.device() != dev || seqlens.numel() != B ||
        !seqlens.is_contiguous() || window_left < -1 || window_left > INT_MAX)
        return std::nullopt;
    const bool paged = block_table.has_value();
    if (paged && (T != 1 || block_table->scalar_type() != at::kInt || block_table->device() != dev || block_table->dim() != 2 ||
                  block_table->size(0) != B || !block_table->is_contiguous() || k_cache.size(1) % nckv_paged_tile_tokens()))
        return std::nullopt;
    if (k_cache.sizes() != v_cache.sizes() || k_cache.strides() != v_cache.strides() || (!paged && k_cache.size(0) != B) ||
        k_cache.size(2) != Hkv || k_cache.size(3) != D || k_cache.stride(3) != 1 || k_cache.stride(2) != D)
        return std::nullopt;
    if (!cos.is_contiguous() || !sin.is_contiguous() || cos.numel() != sin.numel() || cos.numel() % (D / 2) || cos.numel() == 0)
        return std::nullopt;
    const int64_t rope_len = cos.numel() / (D / 2);
    const bool packed = q.is_contiguous() && k.is_contiguous() && v.is_contiguous();
    const int64_t sq = packed ? 0 : token_stride(q), sk = packed ? 0 : token_stride(k), sv = packed ? 0 : token_stride(v);
    if (!packed && (paged || sq < 0 || sk < 0 || sv < 0)) return std::nullopt;
    if (B > INT_MAX || T > INT_MAX || k_cache.size(1) > INT_MAX || rope_len > INT_MAX) return std::nullopt;
    const auto on = launch_on(dev, (int)B, (int)Hq, (int)Hkv);
    if (!on) return std::nullopt;

    const pybind11::gil_scoped_release unlocked;
    const c10::cuda::CUDAGuard guard(dev);
    const auto opt = q.options();
    const int64_t pages = paged ? block_table->size(1) : 1;
    if (T == 1 && nckv_decode_small_fits((int)B, (int)Hq, (int)Hkv, k_cache.size(1) * pages, (int)window_left)) {
        Tensor y = at::empty({B, T, Hq, D}, opt);
        if (nckv_decode_small(q.data_ptr(), k.data_ptr(), v.data_ptr(), sq, sk, sv, k_cache.data_ptr(), v_cache.data_ptr(),
                              paged ? static_cast<const int32_t *>(block_table->data_ptr()) : nullptr, static_cast<const int32_t *>(seqlens.data_ptr()),
                              cos.data_ptr(), sin.data_ptr(), y.data_ptr(), (int)B, (int)Hq, (int)Hkv, (int)D, (int)k_cache.size(1), (int)pages,
                              (int)k_cache.size(0), k_cache.stride(0), k_cache.stride(1), (int)rope_len, (int)window_left, (float)qk_scale, (float)eps,
                              static_cast<int32_t *>(on->ws.data_ptr()), on->stream) < 0)
            return std::nullopt;
        return y;
    }
    Tensor q_rot = at::empty({B, T, Hq, D}, opt);
    int32_t *status = static_cast<int32_t *>(on->ws.data_ptr());
    const size_t ws_bytes = (size_t)on->ws.numel();
    const int32_t *lens = static_cast<const int32_t *>(seqlens.data_ptr());
    const int b = (int)B, t = (int)T, hq = (int)Hq, hk = (int)Hkv, d = (int)D, cap = (int)k_cache.size(1), rl = (int)rope_len;
    const int64_t s0 = k_cache.stride(0), s1 = k_cache.stride(1);
    const float scale = (float)qk_scale, e = (float)eps;
    if (paged) {
        const int32_t *table = static_cast<const int32_t *>(block_table->data_ptr());
        const int max_pages = (int)block_table->size(1), n_pages = (int)k_cache.size(0);
        if (nckv_append_rope_norm_paged(q.data_ptr(), k.data_ptr(), v.data_ptr(), q_rot.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), table,
                                        lens, cos.data_ptr(), sin.data_ptr(), b, t, hq, hk, d, cap, max_pages, n_pages, s0, s1, rl, scale, e,
                                        status, on->stream) < 0)
            return std::nullopt;
        Tensor y = at::empty({B, T, Hq, D}, opt);
        if (nckv_decode_attn_paged(q_rot.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), table, lens, y.data_ptr(), nullptr, nullptr, b, hq, hk,
                                   d, cap, max_pages, n_pages, s0, s1, 1, (int)window_left, status, ws_bytes, on->stream) < 0)
            return std::nullopt;
        return y;
    }
    // strides of 0: packed
    if (nckv_append_rope_norm_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), sq, sk, sv, q_rot.data_ptr(), k_cache.data_ptr(),
                                      v_cache.data_ptr(), lens, cos.data_ptr(), sin.data_ptr(), b, t, hq, hk, d, cap, s0, s1, rl, scale, e,
                                      status, on->stream) < 0)
        return std::nullopt;
    Tensor y = at::empty({B, T, Hq, D}, opt);
    const int rc = t == 1 ? nckv_decode_attn(q_rot.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), lens, y.data_ptr(), nullptr, nullptr, b, hq,
                                             hk, d, cap, s0, s1, 1, (int)window_left, 0, 0, status, ws_bytes, on->stream)
                          : nckv_prefill_attn(q_rot.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), lens, y.data_ptr(), b, t, hq, hk, d, cap,
                                              s0, s1, (int)window_left, status, on->stream);
    if (rc < 0) return std::nullopt;
    return y;
}

// Rows of the trunk's elementwise kernels: contiguous bf16 on one device.
bool row_tensor(const Tensor &t, const Tensor &like) {
    return bf16_on(t, like.device()) && t.is_contiguous() && t.sizes() == like.sizes();
}

using Three = std::tuple<std::optional<Tensor>, std::optional<Tensor>, std::optional<Tensor>>;

// launch(pointers of x, add, x0, x_backout, sum, y, norm, rows, channels, mode, stream) does the rest
template <typename Launch>
std::optional<Three> mix_norm(const Tensor &x, const std::optional<Tensor> &add, const std::optional<Tensor> &x0,
                              const std::optional<Tensor> &x_backout, bool want_sum, bool want_x, bool want_norm, const Launch &launch) {
    if (!x.is_cuda() || x.dim() == 0 || x.numel() == 0 || !row_tensor(x, x)) return std::nullopt;
    for (const std::optional<Tensor> *t : {&add, &x0, &x_backout})
        if (*t && !row_tensor(**t, x)) return std::nullopt;
    const int64_t C = x.size(-1), rows = x.numel() / C;
    if (rows > INT_MAX || C > INT_MAX) return std::nullopt;
    const pybind11::gil_scoped_release unlocked;
    const c10::cuda::CUDAGuard guard(x.device());
    Three out;
    auto &[sum, y, norm] = out;
    if (want_sum && add) sum = at::empty_like(x);
    if (want_x) y = at::empty_like(x);
    if (want_norm) norm = at::empty_like(x);
    auto ptr = [](const std::optional<Tensor> &t) { return t ? t->data_ptr() : nullptr; };
    const cudaStream_t s = at::cuda::getCurrentCUDAStream(x.device().index()).stream();
    if (launch(x.data_ptr(), ptr(add), ptr(x0), ptr(x_backout), ptr(sum), ptr(y), ptr(norm), (int)rows, (int)C, x0 ? 1 : (x_backout ? 2 : 0), s) < 0)
        return std::nullopt;
    return out;
}

std::optional<Three> glue_mix_norm(const Tensor &x, const std::optional<Tensor> &add, const std::optional<Tensor> &x0,
                                   const std::optional<Tensor> &x_backout, double resid_lambda, double x0_lambda, double backout_lambda,
                                   bool want_sum, bool want_x, bool want_norm, double eps) {
    return mix_norm(x, add, x0, x_backout, want_sum, want_x, want_norm,
                    [&](void *px, void *pa, void *p0, void *pb, void *ps, void *py, void *pn, int rows, int C, int mode, cudaStream_t s) {
                        return nckv_glue_mix_norm(px, pa, p0, pb, ps, py, pn, rows, C, mode, (float)resid_lambda, (float)x0_lambda,
                                                  (float)backout_lambda, (float)eps, s);
                    });
}

// The same with the scalars (those of the mix that is asked for) in vectors on the rows' device: element `layer` of the
// first two, the only one of the third.
std::optional<Three> glue_mix_norm_at(const Tensor &x, const std::optional<Tensor> &add, const std::optional<Tensor> &x0,
                                      const std::optional<Tensor> &x_backout, const std::optional<Tensor> &resid_lambdas,
                                      const std::optional<Tensor> &x0_lambdas, const std::optional<Tensor> &backout_lambda, int64_t layer,
                                      bool want_sum, bool want_x, bool want_norm, double eps) {
    const void *at[3] = {};
    int f32_mask = 0, i = 0;
    for (const std::optional<Tensor> *t : {&resid_lambdas, &x0_lambdas, &backout_lambda}) {
        if (*t) {
            const int64_t n = (*t)->numel(), e = i < 2 ? layer : 0;
            const bool f32 = (*t)->scalar_type() == at::kFloat;
            if (e < 0 || e >= n || (i == 2 && n != 1) || !(*t)->is_contiguous() || (*t)->device() != x.device() ||
                (!f32 && (*t)->scalar_type() != at::kBFloat16))
                return std::nullopt;
            at[i] = static_cast<const char *>((*t)->data_ptr()) + e * (f32 ? 4 : 2);
            f32_mask |= (int)f32 << i;
        }
        ++i;
    }
    return mix_norm(x, add, x0, x_backout, want_sum, want_x, want_norm,
                    [&](void *px, void *pa, void *p0, void *pb, void *ps, void *py, void *pn, int rows, int C, int mode, cudaStream_t s) {
                        return nckv_glue_mix_norm_at(px, pa, p0, pb, ps, py, pn, rows, C, mode, at[0], at[1], at[2], f32_mask, (float)eps, s);
                    });
}

std::optional<Tensor> glue_relu_sq(const Tensor &h) {
    if (!h.is_cuda() || !row_tensor(h, h)) return std::nullopt;
    const pybind11::gil_scoped_release unlocked;
    const c10::cuda::CUDAGuard guard(h.device());
    Tensor out = at::empty_like(h);
    if (nckv_glue_relu_sq(h.data_ptr(), out.data_ptr(), h.numel(), at::cuda::getCurrentCUDAStream(h.device().index()).stream()) < 0)
        return std::nullopt;
    return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("set_workspace", &set_workspace);
    m.def("kv_attention", &kv_attention);
    m.def("glue_mix_norm", &glue_mix_norm);
    m.def("glue_mix_norm_at", &glue_mix_norm_at);
    m.def("glue_relu_sq", &glue_relu_sq);
}
