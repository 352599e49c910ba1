// Native host path of the operator and of the module: argument blocks, allocation and autograd in C++.
//
// The kernels sit behind the C ABI of libsa2.so (include/sa2.h); this file turns at::Tensors into its argument
// blocks, as attention.py and headnorm.py do through ctypes.  In Python a forward + backward pair of the operator
// cost the host 280 us and a generation step of the module 520 us, more than the kernels of short sequences take.
//
// Every function returns None when the tensors are not what the kernels take, or when torch is recording or
// transforming the computation; the Python caller then runs its own checks, which raise the documented exceptions, and
// its general path.
#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <ATen/TracerMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include "sa2.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// entry points of the loaded library (it may be another build than the one beside this file)
struct Lib {
    int (*fwd)(const sa2_fwd_args *) = nullptr;
    int (*bwd)(const sa2_bwd_args *) = nullptr;
    size_t (*workspace)(const sa2_shape *) = nullptr;
    int (*norm_fwd)(const sa2_headnorm_args *) = nullptr;
    int (*norm_bwd)(const sa2_headnorm_args *) = nullptr;
    size_t (*partial_bytes)(int64_t, int32_t) = nullptr;
    int (*qkv_fwd)(const sa2_qkvnorm_args *) = nullptr;
    int (*qkv_bwd)(const sa2_qkvnorm_args *) = nullptr;
    int (*append)(const sa2_qkvnorm_args *, const sa2_append_set *, int32_t, int32_t) = nullptr;
    int (*norm_linear)(const void *, const void *, int32_t, float, const void *, void *, int32_t, int32_t, int32_t, void *) = nullptr;
    int (*step_attn)(const sa2_qkvnorm_args *, const sa2_append_set *, void *, int32_t, int32_t, int32_t, float) = nullptr;
} L;

void bind(const std::map<std::string, uintptr_t> &f) {
    auto set = [&](auto &slot, const char *name) { slot = reinterpret_cast<std::decay_t<decltype(slot)>>(f.at(name)); };
    set(L.fwd, "sa2_fwd"); set(L.bwd, "sa2_bwd"); set(L.workspace, "sa2_bwd_workspace_bytes");
    set(L.norm_fwd, "sa2_headnorm_fwd"); set(L.norm_bwd, "sa2_headnorm_bwd"); set(L.partial_bytes, "sa2_headnorm_partial_bytes");
    set(L.qkv_fwd, "sa2_qkvnorm_fwd"); set(L.qkv_bwd, "sa2_qkvnorm_bwd"); set(L.append, "sa2_qkv_append");
    set(L.norm_linear, "sa2_norm_linear"); set(L.step_attn, "sa2_step_attn");
}

// raises _lib.Sa2Error, also from the autograd engine's threads
void check(int status, const char *where) {
    if (status == SA2_OK) return;
    pybind11::gil_scoped_acquire gil;
    try {
        pybind11::module_::import("simplicial_attention_b200._lib").attr("check")(status, where);
    } catch (pybind11::error_already_set &e) {
        e.restore();
        python_error err;
        err.persist();
        throw err;
    }
}

int dtype_of(const Tensor &t) {
    return t.scalar_type() == at::kBFloat16 ? SA2_BF16 : t.scalar_type() == at::kFloat ? SA2_F32 : -1;
}
bool aligned(const Tensor &t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }

// The kernels may read t's memory as it stands: t is on `where`, and neither a subclass nor a functorch transform stands
// between it and its values, nor does it carry a forward-mode tangent that a raw launch would drop.  The general paths
// run into torch's own errors, or its dispatch, for everything else.
bool plain(const Tensor &t, c10::Device where) {
    static const c10::DispatchKeySet wrappers({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper});
    return t.device() == where && t.is_cuda() && t.layout() == at::kStrided && !t.is_neg() && !t.key_set().has_any(wrappers) && !t._fw_grad(0).defined();
}
// torch.jit.trace is recording: it sees the allocations of the nodes below but not their launches, so that a replay
// would return uninitialised memory
bool tracing() { return at::tracer::impl::is_dispatch_enabled(); }

// the tensor itself if the kernels can address it in place, else a contiguous copy
Tensor usable(const Tensor &t) {
    const bool ok = t.stride(3) == 1 && t.stride(0) % 4 == 0 && t.stride(1) % 4 == 0 && t.stride(2) % 4 == 0 && aligned(t);
    return ok ? t : t.contiguous();
}
// keys and values, which the bf16 kernels load with TMA: it cannot repeat a dimension (an expanded tensor)
Tensor usable_kv(const Tensor &t) {
    if (t.scalar_type() == at::kBFloat16)
        for (int x = 0; x < 3; ++x)
            if (t.stride(x) == 0 && t.size(x) > 1) return t.contiguous();
    return usable(t);
}
sa2_strides strides(const Tensor &t) { return sa2_strides{t.stride(0), t.stride(1), t.stride(2)}; }

struct Cfg {
    int64_t w1, w2, kernel;
    double scale;
};

sa2_shape shape_of(const Tensor &q, const Tensor &k1, const Tensor &k2, const Cfg &c) {
    sa2_shape s;
    s.b = (int32_t)q.size(0); s.n = (int32_t)q.size(1); s.hq = (int32_t)q.size(2); s.hk = (int32_t)k1.size(2);
    s.d = (int32_t)q.size(3); s.w1 = (int32_t)c.w1; s.w2 = (int32_t)c.w2;
    s.off1 = (int32_t)(k1.size(1) - q.size(1)); s.off2 = (int32_t)(k2.size(1) - q.size(1));
    s.dtype = dtype_of(q); s.kernel = (int32_t)c.kernel; s.scale = (float)c.scale;
    return s;
}

bool inputs_ok(const Tensor &q, const Tensor &k1, const Tensor &k2, const Tensor &v1, const Tensor &v2) {
    if (tracing()) return false;
    for (const Tensor *t : {&q, &k1, &k2, &v1, &v2})
        if (!plain(*t, q.device()) || t->dim() != 4 || t->scalar_type() != q.scalar_type()) return false;
    const auto n = q.size(1), d = q.size(3), hk = k1.size(2);
    if (dtype_of(q) < 0 || (d != 32 && d != 64 && d != 128) || hk <= 0 || q.size(2) % hk != 0) return false;
    if (k1.sizes() != v1.sizes() || k2.sizes() != v2.sizes()) return false;
    for (const Tensor *t : {&k1, &k2})
        if (t->size(0) != q.size(0) || t->size(2) != hk || t->size(3) != d || t->size(1) < n) return false;
    return true;
}

// out [b][n][hq][d] and lse [b][hq][n]; the inputs are usable
void run_forward(const Tensor &q, const Tensor &k1, const Tensor &k2, const Tensor &v1, const Tensor &v2, const Cfg &c, Tensor &out, Tensor &lse) {
    sa2_fwd_args a;
    a.shape = shape_of(q, k1, k2, c);
    out = at::empty({q.size(0), q.size(1), q.size(2), q.size(3)}, q.options());
    lse = at::empty({q.size(0), q.size(2), q.size(1)}, q.options().dtype(at::kFloat));
    a.q = q.data_ptr(); a.k1 = k1.data_ptr(); a.k2 = k2.data_ptr(); a.v1 = v1.data_ptr(); a.v2 = v2.data_ptr();
    a.out = out.data_ptr(); a.lse = lse.data_ptr<float>();
    a.sq = strides(q); a.sk1 = strides(k1); a.sk2 = strides(k2); a.sv1 = strides(v1); a.sv2 = strides(v2); a.sout = strides(out);
    a.stream = c10::cuda::getCurrentCUDAStream(q.get_device()).stream();
    check(L.fwd(&a), "sa2_fwd");
}

void run_backward(const Tensor &q, const Tensor &k1, const Tensor &k2, const Tensor &v1, const Tensor &v2, const Tensor &out, const Tensor &lse,
                  const Tensor &dout, const Cfg &c, const Tensor (&g)[5]) {
    sa2_bwd_args a;
    a.shape = shape_of(q, k1, k2, c);
    const size_t bytes = L.workspace(&a.shape);
    const Tensor ws = at::empty({(int64_t)std::max<size_t>(bytes, 256)}, q.options().dtype(at::kByte));
    a.q = q.data_ptr(); a.k1 = k1.data_ptr(); a.k2 = k2.data_ptr(); a.v1 = v1.data_ptr(); a.v2 = v2.data_ptr();
    a.out = out.data_ptr(); a.dout = dout.data_ptr(); a.lse = lse.data_ptr<float>();
    a.dq = g[0].data_ptr(); a.dk1 = g[1].data_ptr(); a.dk2 = g[2].data_ptr(); a.dv1 = g[3].data_ptr(); a.dv2 = g[4].data_ptr();
    a.sq = strides(q); a.sk1 = strides(k1); a.sk2 = strides(k2); a.sv1 = strides(v1); a.sv2 = strides(v2);
    a.sout = strides(out); a.sdout = strides(dout);
    a.sdq = strides(g[0]); a.sdk1 = strides(g[1]); a.sdk2 = strides(g[2]); a.sdv1 = strides(g[3]); a.sdv2 = strides(g[4]);
    a.grad_dtype = dtype_of(g[0]);
    a.phases = 0;
    a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
    a.stream = c10::cuda::getCurrentCUDAStream(q.get_device()).stream();
    check(L.bwd(&a), "sa2_bwd");
}

// ------------------------------------------------------------------ the operator
struct Attn : torch::autograd::Function<Attn> {
    static variable_list forward(AutogradContext *ctx, const Tensor &q, const Tensor &k1, const Tensor &k2, const Tensor &v1, const Tensor &v2,
                                 int64_t w1, int64_t w2, double scale, int64_t kernel) {
        const c10::cuda::CUDAGuard guard(q.device());
        const Cfg c{w1, w2, kernel, scale};
        Tensor out, lse;
        run_forward(usable(q), usable_kv(k1), usable_kv(k2), usable_kv(v1), usable_kv(v2), c, out, lse);
        ctx->save_for_backward({q, k1, k2, v1, v2, out, lse});
        ctx->saved_data["w1"] = w1;
        ctx->saved_data["w2"] = w2;
        ctx->saved_data["scale"] = scale;
        ctx->saved_data["kernel"] = kernel;
        ctx->mark_non_differentiable({lse});
        ctx->set_materialize_grads(false);      // no zeros for the gradient of lse
        return {out, lse};
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto s = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard guard(s[0].device());
        const Cfg c{ctx->saved_data["w1"].toInt(), ctx->saved_data["w2"].toInt(), ctx->saved_data["kernel"].toInt(), ctx->saved_data["scale"].toDouble()};
        Tensor dout = grads[0].defined() ? usable(grads[0]) : at::zeros_like(s[5]);
        if (dout.scalar_type() != s[0].scalar_type()) dout = dout.to(s[0].scalar_type());
        Tensor g[5];
        for (int x = 0; x < 5; ++x) g[x] = at::empty(s[x].sizes(), s[x].options());
        run_backward(usable(s[0]), usable_kv(s[1]), usable_kv(s[2]), usable_kv(s[3]), usable_kv(s[4]), s[5], s[6], dout, c, g);
        return {g[0], g[1], g[2], g[3], g[4], Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

pybind11::object attn(const Tensor &q, const Tensor &k1, const Tensor &k2, const Tensor &v1, const Tensor &v2, int64_t w1, int64_t w2,
                      std::optional<double> scale, int64_t kernel, bool return_lse) {
    if (!inputs_ok(q, k1, k2, v1, v2)) return pybind11::none();
    auto r = Attn::apply(q, k1, k2, v1, v2, w1, w2, scale ? *scale : 1. / std::sqrt((double)q.size(3)), kernel);
    if (return_lse) return pybind11::make_tuple(r[0], r[1]);
    return pybind11::cast(r[0]);
}

// ------------------------------------------------------------------ RMSNorm with one gain per channel
struct HeadNorm : torch::autograd::Function<HeadNorm> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &weight, int64_t d, double eps, at::ScalarType out_dtype) {
        const c10::cuda::CUDAGuard guard(x.device());
        const int64_t ch = x.size(-1);
        Tensor x2 = x.reshape({-1, ch});
        if (x2.stride(1) != 1) x2 = x2.contiguous();
        const Tensor w = weight.detach().to(at::kFloat).contiguous();
        const int64_t rows = x2.size(0);
        Tensor y = at::empty({rows, ch}, x.options().dtype(out_dtype));
        Tensor rstd = at::empty({rows, ch / d}, x.options().dtype(at::kFloat));
        sa2_headnorm_args a{};
        a.x = x2.data_ptr(); a.weight = w.data_ptr<float>(); a.y = y.data_ptr(); a.rstd = rstd.data_ptr<float>();
        a.rows = rows; a.x_stride = x2.stride(0); a.y_stride = ch; a.channels = (int32_t)ch; a.d = (int32_t)d;
        a.x_dtype = dtype_of(x2); a.y_dtype = dtype_of(y); a.eps = (float)eps;
        a.stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
        check(L.norm_fwd(&a), "sa2_headnorm_fwd");
        ctx->save_for_backward({x2, w, rstd});
        ctx->saved_data["d"] = d;
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["shape"] = x.sizes().vec();
        ctx->saved_data["wdtype"] = (int64_t)weight.scalar_type();
        return y.view(x.sizes());
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto s = ctx->get_saved_variables();
        const Tensor &x2 = s[0];
        const c10::cuda::CUDAGuard guard(x2.device());
        const int64_t rows = x2.size(0), ch = x2.size(1);
        Tensor dy = grads[0].reshape({rows, ch});
        if (dy.stride(1) != 1 || dtype_of(dy) < 0) dy = dy.contiguous().to(dtype_of(dy) < 0 ? at::kFloat : dy.scalar_type());
        Tensor dx = at::empty({rows, ch}, x2.options()), dw = at::empty({ch}, x2.options().dtype(at::kFloat));
        const size_t bytes = L.partial_bytes(rows, (int32_t)ch);
        const Tensor partial = at::empty({(int64_t)std::max<size_t>(bytes, 256)}, x2.options().dtype(at::kByte));
        sa2_headnorm_args a{};
        a.x = x2.data_ptr(); a.dy = dy.data_ptr(); a.weight = s[1].data_ptr<float>(); a.y = dx.data_ptr(); a.rstd = s[2].data_ptr<float>();
        a.dweight = dw.data_ptr<float>(); a.partial = partial.data_ptr(); a.partial_bytes = (size_t)partial.numel();
        a.rows = rows; a.x_stride = x2.stride(0); a.y_stride = ch; a.dy_stride = dy.stride(0); a.channels = (int32_t)ch;
        a.d = (int32_t)ctx->saved_data["d"].toInt();
        a.x_dtype = dtype_of(x2); a.y_dtype = dtype_of(dy); a.eps = (float)ctx->saved_data["eps"].toDouble();
        a.stream = c10::cuda::getCurrentCUDAStream(x2.get_device()).stream();
        check(L.norm_bwd(&a), "sa2_headnorm_bwd");
        return {dx.view(ctx->saved_data["shape"].toIntVector()), dw.to((at::ScalarType)ctx->saved_data["wdtype"].toInt()), Tensor(), Tensor(), Tensor()};
    }
};
pybind11::object headnorm(const Tensor &x, const Tensor &weight, int64_t d, double eps, at::ScalarType out_dtype) {
    if (tracing() || !plain(x, x.device()) || !plain(weight, x.device())) return pybind11::none();
    return pybind11::cast(HeadNorm::apply(x, weight, d, eps, out_dtype));
}

// ------------------------------------------------------------------ the module: packed projection -> attention
struct Heads {
    int64_t hq, hk, d;
    int64_t channels() const { return d * (hq + 4 * hk); }
};

// the five operands inside a packed [b][n][channels] tensor, read (or written) in place
void split(const Tensor &y, const Heads &h, Tensor (&t)[5]) {
    const int64_t b = y.size(0), n = y.size(1), sb = y.stride(0), sn = y.stride(1), o = y.storage_offset();
    const int64_t k = o + h.hq * h.d, v = k + 2 * h.hk * h.d;
    t[0] = y.as_strided({b, n, h.hq, h.d}, {sb, sn, h.d, 1}, o);
    t[1] = y.as_strided({b, n, h.hk, h.d}, {sb, sn, 2 * h.d, 1}, k);
    t[2] = y.as_strided({b, n, h.hk, h.d}, {sb, sn, 2 * h.d, 1}, k + h.d);
    t[3] = y.as_strided({b, n, h.hk, h.d}, {sb, sn, 2 * h.d, 1}, v);
    t[4] = y.as_strided({b, n, h.hk, h.d}, {sb, sn, 2 * h.d, 1}, v + h.d);
}

void fill_norm(sa2_qkvnorm_args &a, const Tensor &x, const Tensor (&gain)[5], const Heads &h, double eps) {
    a.x = x.data_ptr(); a.rows = x.size(0) * x.size(1); a.x_stride = x.stride(1);
    for (int g = 0; g < 5; ++g) a.gain[g] = gain[g].data_ptr();
    a.hq = (int32_t)h.hq; a.hk = (int32_t)h.hk; a.d = (int32_t)h.d;
    a.x_dtype = dtype_of(x); a.gain_dtype = dtype_of(gain[0]); a.eps = (float)eps;
    a.stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
}

struct QkvAttn : torch::autograd::Function<QkvAttn> {
    static Tensor forward(AutogradContext *ctx, const Tensor &proj, const Tensor &g0, const Tensor &g1, const Tensor &g2, const Tensor &g3,
                          const Tensor &g4, int64_t hq, int64_t hk, int64_t d, double eps, at::ScalarType dt, int64_t w1, int64_t w2, int64_t kernel) {
        const c10::cuda::CUDAGuard guard(proj.device());
        const Heads h{hq, hk, d};
        const Tensor gain[5] = {g0, g1, g2, g3, g4};
        Tensor y = at::empty(proj.sizes(), proj.options().dtype(dt));
        Tensor rstd = at::empty({proj.size(0) * proj.size(1), hq + 4 * hk}, proj.options().dtype(at::kFloat));
        sa2_qkvnorm_args a{};
        fill_norm(a, proj, gain, h, eps);
        a.y = y.data_ptr(); a.rstd = rstd.data_ptr<float>(); a.y_stride = y.stride(1); a.y_dtype = dtype_of(y);
        check(L.qkv_fwd(&a), "sa2_qkvnorm_fwd");
        Tensor t[5], out, lse;
        split(y, h, t);
        run_forward(t[0], t[1], t[2], t[3], t[4], Cfg{w1, w2, kernel, 1. / std::sqrt((double)d)}, out, lse);
        ctx->save_for_backward({proj, g0, g1, g2, g3, g4, rstd, y, out, lse});
        ctx->saved_data["i"] = std::vector<int64_t>{hq, hk, d, w1, w2, kernel};
        ctx->saved_data["eps"] = eps;
        return out;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto s = ctx->get_saved_variables();
        const Tensor &proj = s[0], &rstd = s[6], &y = s[7], &out = s[8], &lse = s[9];
        const c10::cuda::CUDAGuard guard(proj.device());
        const auto i = ctx->saved_data["i"].toIntVector();
        const Heads h{i[0], i[1], i[2]};
        const Tensor gain[5] = {s[1], s[2], s[3], s[4], s[5]};
        Tensor dout = usable(grads[0]);
        if (dout.scalar_type() != y.scalar_type()) dout = dout.to(y.scalar_type());
        // the gradients of the five operands land side by side where the norm's backward reads them
        Tensor dy = at::empty(y.sizes(), y.options()), t[5], g[5];
        split(y, h, t);
        split(dy, h, g);
        run_backward(t[0], t[1], t[2], t[3], t[4], out, lse, dout, Cfg{i[3], i[4], i[5], 1. / std::sqrt((double)h.d)}, g);
        sa2_qkvnorm_args a{};
        fill_norm(a, proj, gain, h, ctx->saved_data["eps"].toDouble());
        Tensor dx = at::empty(proj.sizes(), proj.options().memory_format(at::MemoryFormat::Contiguous)), dg[5];
        for (int x = 0; x < 5; ++x) {
            dg[x] = at::empty({h.d}, gain[x].options());
            a.dgain[x] = dg[x].data_ptr();
        }
        const size_t bytes = L.partial_bytes(a.rows, (int32_t)h.channels());
        const Tensor partial = at::empty({(int64_t)bytes}, proj.options().dtype(at::kByte));
        a.dy = dy.data_ptr(); a.y = dx.data_ptr(); a.rstd = rstd.data_ptr<float>(); a.partial = partial.data_ptr(); a.partial_bytes = bytes;
        a.dy_stride = dy.stride(1); a.y_stride = dx.stride(1); a.y_dtype = dtype_of(dy);
        check(L.qkv_bwd(&a), "sa2_qkvnorm_bwd");
        variable_list r(14);
        r[0] = dx;
        for (int x = 0; x < 5; ++x) r[1 + x] = dg[x];
        return r;
    }
};

bool gains_ok(const std::vector<Tensor> &gain, const Heads &h, c10::Device where) {
    if (gain.size() != 5) return false;
    for (const Tensor &g : gain)
        if (!plain(g, where) || g.scalar_type() != gain[0].scalar_type() || dtype_of(g) < 0 || g.dim() != 1 || g.size(0) != h.d || g.stride(0) != 1 || !aligned(g))
            return false;
    return true;
}
bool projection_ok(const Tensor &proj, const std::vector<Tensor> &gain, const Heads &h, at::ScalarType dt) {
    if (tracing() || !plain(proj, proj.device()) || proj.dim() != 3 || dtype_of(proj) < 0 || (dt != at::kFloat && dt != at::kBFloat16)) return false;
    if (proj.size(2) != h.channels() || proj.numel() == 0 || proj.stride(2) != 1 || proj.stride(0) != proj.size(1) * proj.stride(1)) return false;
    return gains_ok(gain, h, proj.device()) && (h.d == 32 || h.d == 64 || h.d == 128);
}

// [b][n][hq][d], or None
pybind11::object qkv_attn(const Tensor &proj, const std::vector<Tensor> &gain, int64_t hq, int64_t hk, int64_t d, double eps, at::ScalarType dt,
                          int64_t w1, int64_t w2, int64_t kernel) {
    if (!projection_ok(proj, gain, Heads{hq, hk, d}, dt) || hq + 4 * hk > 6400 / d) return pybind11::none();
    return pybind11::cast(QkvAttn::apply(proj, gain[0], gain[1], gain[2], gain[3], gain[4], hq, hk, d, eps, dt, w1, w2, kernel));
}

bool cache_ok(const std::vector<Tensor> &cache, const Heads &h, const Tensor &x) {
    if (cache.size() != 4) return false;
    const int64_t piece = x.scalar_type() == at::kBFloat16 ? 8 : 4;
    for (const Tensor &t : cache)
        if (!plain(t, x.device()) || t.dim() != 4 || t.scalar_type() != x.scalar_type() || t.size(0) != x.size(0) || t.size(2) != h.hk || t.size(3) != h.d || t.stride(3) != 1 ||
            t.stride(0) % piece || t.stride(1) % piece || t.stride(2) % piece || !aligned(t)) return false;
    return cache[0].size(1) == cache[2].size(1) && cache[1].size(1) == cache[3].size(1);
}

// out [b][n][hq][d], and set = [k, k', v, v'] with the new rows behind the cached ones, cut to what later rows can see
void attend_cached(const Tensor &proj, const std::vector<Tensor> &gain, const std::vector<Tensor> &cache, const Heads &h, double eps, int64_t w1,
                   int64_t w2, int64_t kernel, Tensor &out, Tensor (&set)[4]) {
    const int64_t b = proj.size(0), n = proj.size(1);
    const Tensor g5[5] = {gain[0], gain[1], gain[2], gain[3], gain[4]};
    Tensor q = at::empty({b, n, h.hq, h.d}, proj.options()), lse;
    sa2_append_set as[4];
    for (int s = 0; s < 4; ++s) {
        const int64_t keep = cache[s].size(1);
        set[s] = at::empty({b, keep + n, h.hk, h.d}, proj.options());
        as[s] = sa2_append_set{cache[s].data_ptr(), strides(cache[s]), set[s].data_ptr(), (int32_t)keep};
    }
    sa2_qkvnorm_args a{};
    fill_norm(a, proj, g5, h, eps);
    a.y = q.data_ptr(); a.y_dtype = dtype_of(q);
    check(L.append(&a, as, (int32_t)b, (int32_t)n), "sa2_qkv_append");
    run_forward(q, set[0], set[1], set[2], set[3], Cfg{w1, w2, kernel, 1. / std::sqrt((double)h.d)}, out, lse);
    for (int s = 0; s < 4; ++s) {
        const int64_t rows = set[s].size(1), keep = std::min(rows, (s & 1 ? w2 : w1) - 1);
        if (keep < rows) set[s] = set[s].narrow(1, rows - keep, keep);
    }
}

// One new row per sequence: the same in one launch, with set = [k, k', v, v'] cut to what later rows can see as it is made.
// False where sa2_step_attn does not take the shape.
bool attend_one(const Tensor &proj, const std::vector<Tensor> &gain, const std::vector<Tensor> &cache, const Heads &h, double eps, int64_t w1,
                int64_t w2, Tensor &out, Tensor (&set)[4]) {
    const int64_t b = proj.size(0);
    const Tensor g5[5] = {gain[0], gain[1], gain[2], gain[3], gain[4]};
    sa2_append_set as[4];
    for (int s = 0; s < 4; ++s) {
        const int64_t keep = cache[s].size(1);
        set[s] = at::empty({b, std::min(keep + 1, (s & 1 ? w2 : w1) - 1), h.hk, h.d}, proj.options());
        as[s] = sa2_append_set{cache[s].data_ptr(), strides(cache[s]), set[s].data_ptr(), (int32_t)keep};
    }
    sa2_qkvnorm_args a{};
    fill_norm(a, proj, g5, h, eps);
    out = at::empty({b, 1, h.hq, h.d}, proj.options());
    const int rc = L.step_attn(&a, as, out.data_ptr(), (int32_t)b, (int32_t)w1, (int32_t)w2, (float)(1. / std::sqrt((double)h.d)));
    if (rc == SA2_ERR_UNSUPPORTED) return false;
    check(rc, "sa2_step_attn");
    return true;
}

// Generation: (out [b][n][hq][d], [k, k', v, v']), or None.  cache: [k, k', v, v'] of the rows before; no gradients.
pybind11::object qkv_attn_cached(const Tensor &proj, const std::vector<Tensor> &gain, const std::vector<Tensor> &cache, int64_t hq, int64_t hk,
                                 int64_t d, double eps, int64_t w1, int64_t w2, int64_t kernel) {
    const Heads h{hq, hk, d};
    if (!projection_ok(proj, gain, h, proj.scalar_type()) || !cache_ok(cache, h, proj)) return pybind11::none();
    const c10::cuda::CUDAGuard guard(proj.device());
    const at::AutoDispatchBelowADInplaceOrView below;
    Tensor out, set[4];
    attend_cached(proj, gain, cache, h, eps, w1, w2, kernel, out, set);
    return pybind11::make_tuple(out, set[0], set[1], set[2], set[3]);
}

bool row_norm_ok(const std::optional<Tensor> &w, const Tensor &x) {
    return !w || (w->dim() == 1 && w->numel() == x.size(2) && plain(*w, x.device()) && dtype_of(*w) >= 0 && w->stride(0) == 1 && aligned(*w));
}
// RMSNorm over the last dimension, the gain read in its own type; the row scale is not kept.  Widths that the kernel
// does not take go where headnorm.py's RMSNorm sends them.
Tensor row_norm(const Tensor &x, const Tensor &w, double eps) {
    const int64_t d = w.numel();
    if (d != 32 && d != 64 && d != 128 && d != 256 && d != 512) return at::rms_norm(x, {d}, w, eps);
    const Tensor x2 = x.is_contiguous() ? x : x.contiguous();
    Tensor y = at::empty(x2.sizes(), x2.options());
    sa2_qkvnorm_args a{};
    a.x = x2.data_ptr(); a.y = y.data_ptr(); a.gain[0] = w.data_ptr();
    a.rows = x2.numel() / d; a.x_stride = a.y_stride = d; a.hq = 1; a.hk = 0; a.d = (int32_t)d;
    a.x_dtype = a.y_dtype = dtype_of(x2); a.gain_dtype = dtype_of(w); a.eps = (float)eps;
    a.stream = c10::cuda::getCurrentCUDAStream(x2.get_device()).stream();
    check(L.qkv_fwd(&a), "sa2_qkvnorm_fwd");
    return y;
}

// Does the kernel for few rows take x W^T?  Up to 16 rows always: it is the faster one on the device too.  Up to 64 with a W of at most
// 2^20 entries: on the device it takes longer there (with the norm, 512 -> 1536: 4.9 us at 32 rows and 7.5 at 64, against 3.0 and the norm's
// own 2.0), but its two calls cost the host 16 to 20 us less.  Whole steps back to back, with the library's kernel / with this one (in
// brackets the same as a graph, which the host does not bound): W of 0.75 and 0.25 M entries, 17 rows 48 / 30 us (16.6 / 16.9), 32 rows 48 /
// 30 (17.2 / 18.4), 64 rows 47 / 31 (17.5 / 24.5).  Above the line the gap closes and turns: 1.25 and 0.25 M, 64 rows 48 / 43 (25.6 / 37.8);
// 5 and 1 M, 64 rows 52 / 82 (44 / 75); 20 and 4 M, 17 rows 54 / 69 (35 / 63).
bool few_rows(const Tensor &x, const Tensor &w) {
    const int64_t rows = x.size(0) * x.size(1), k = w.size(1), outs = w.size(0);
    return rows <= (k * outs <= 1 << 20 ? 64 : 16) && k % 32 == 0 && outs % 16 == 0 && x.scalar_type() == at::kBFloat16 && x.is_contiguous() &&
           w.is_contiguous() && aligned(x) && aligned(w);
}
// x W^T over the last dimension, and the same behind an RMSNorm
Tensor few_rows_linear(const Tensor &x, const Tensor *gain, double eps, const Tensor &w) {
    Tensor y = at::empty({x.size(0), x.size(1), w.size(0)}, x.options());
    check(L.norm_linear(x.data_ptr(), gain ? gain->data_ptr() : nullptr, gain ? dtype_of(*gain) : SA2_F32, (float)eps, w.data_ptr(), y.data_ptr(),
                        (int32_t)(x.size(0) * x.size(1)), (int32_t)w.size(1), (int32_t)w.size(0),
                        c10::cuda::getCurrentCUDAStream(x.get_device()).stream()), "sa2_norm_linear");
    return y;
}
Tensor step_linear(const Tensor &x, const Tensor &w) { return few_rows(x, w) ? few_rows_linear(x, nullptr, 0., w) : at::linear(x, w); }
Tensor step_norm_linear(const Tensor &x, const Tensor &gain, double eps, const Tensor &w) {
    return few_rows(x, w) ? few_rows_linear(x, &gain, eps, w) : at::linear(row_norm(x, gain, eps), w);
}

// A whole generation step: (out [b][n][dim], [k, k', v, v']), or None.  norms: gain and eps of the prenorm and of
// the postnorm, where there are any.  From Python, the module calls and autograd nodes around its five kernels
// cost the host twice what the kernels of a small batch take.
pybind11::object step(const Tensor &x, const std::optional<Tensor> &pre, double pre_eps, const Tensor &w_qkv, const std::vector<Tensor> &gain,
                      const std::vector<Tensor> &cache, int64_t hq, int64_t hk, int64_t d, double eps, int64_t w1, int64_t w2, int64_t kernel,
                      const Tensor &w_out, const std::optional<Tensor> &post, double post_eps) {
    const Heads h{hq, hk, d};
    // (a dispatch mode wants to see the projections, which the kernel for few rows hides)
    if (tracing() || c10::impl::TorchDispatchModeTLS::any_modes_set()) return pybind11::none();
    if (!plain(x, x.device()) || x.dim() != 3 || x.numel() == 0 || dtype_of(x) < 0 || !row_norm_ok(pre, x)) return pybind11::none();
    for (const Tensor *w : {&w_qkv, &w_out})
        if (!plain(*w, x.device()) || w->dim() != 2 || w->scalar_type() != x.scalar_type()) return pybind11::none();
    if (w_qkv.size(1) != x.size(2) || w_qkv.size(0) != h.channels() || w_out.size(1) != hq * d || w_out.size(0) != x.size(2) || !row_norm_ok(post, x))
        return pybind11::none();
    if (!cache_ok(cache, h, x) || !gains_ok(gain, h, x.device())) return pybind11::none();
    const c10::cuda::CUDAGuard guard(x.device());
    const at::AutoDispatchBelowADInplaceOrView below;
    const Tensor proj = pre ? step_norm_linear(x, *pre, pre_eps, w_qkv) : step_linear(x, w_qkv);
    if (!projection_ok(proj, gain, h, x.scalar_type())) return pybind11::none();
    Tensor out, set[4];
    const bool one = x.size(1) == 1 && x.scalar_type() == at::kBFloat16 && (d == 64 || d == 128) && w2 <= 64 && kernel == SA2_KERNEL_AUTO;
    if (!one || !attend_one(proj, gain, cache, h, eps, w1, w2, out, set)) attend_cached(proj, gain, cache, h, eps, w1, w2, kernel, out, set);
    out = step_linear(out.view({x.size(0), x.size(1), hq * d}), w_out);
    if (post) out = row_norm(out, *post, post_eps);
    return pybind11::make_tuple(out, set[0], set[1], set[2], set[3]);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", &bind);
    m.def("attn", &attn);
    m.def("headnorm", &headnorm);
    m.def("qkv_attn", &qkv_attn);
    m.def("qkv_attn_cached", &qkv_attn_cached);
    m.def("step", &step);
}
