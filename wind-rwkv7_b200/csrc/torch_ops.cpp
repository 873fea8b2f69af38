// Host path of the Python entry points, eager mode: argument checks, allocation, launches and autograd nodes in C++, on top of
// the C ABI of libwkv7_sm100.so.  The Python form of the same (ctypes calls of 17 to 35 arguments, autograd functions run by the
// interpreter) costs 25 us for a decode step, 240 us for an attn forward + backward and 2.1 ms for a time-mixer layer, which is what
// small calls then take; torch.compile still traces that form.
//
// A function here that returns None (nothing launched) leaves the call to the Python path: other dtypes, devices, shapes or layouts than the
// ones below, with their conversions and error messages.
#include <ATen/TracerMode.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/extension.h>

#include "../../include/wkv7_sm100.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

constexpr int64_t N = 64;
constexpr double LN_EPS = 64e-5;

void check(int rc, const char* what) {
    if (rc != 0)
        throw std::runtime_error(std::string(what) + " failed: " + wkv7_status_string(rc) + " (status " + std::to_string(rc) + ")");
    const int dev = wkv7_peek_status();
    if (dev != 0)
        throw std::runtime_error(std::string("an earlier wkv7 kernel reported: ") + wkv7_status_string(dev) + " (status " + std::to_string(dev) +
                                 "); its results are invalid.  wkv7_device_status() reads and clears the error.");
}
void* stream() { return (void*)at::cuda::getCurrentCUDAStream().stream(); }
float* f32(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
Tensor scratch(const Tensor& like) {
    static const int64_t bytes = (int64_t)wkv7_workspace_bytes();
    return at::empty({bytes}, like.options().dtype(at::kByte));
}
// Scratch of a backward call; undefined where the tiles of a walked state gradient, up to 512 MB, cannot be had: the kernels then take the form
// that needs none.
Tensor bwd_scratch(int64_t bytes, const Tensor& like) {
    try {
        return at::empty({bytes}, like.options().dtype(at::kByte));
    } catch (const c10::OutOfMemoryError&) {
        if (bytes <= (int64_t)wkv7_workspace_bytes()) throw;
        return Tensor();
    }
}
bool grad_wanted(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}
// a dense CUDA tensor of its own: no transform wrapper, whose meaning only the Python path's operators see
bool plain(const Tensor& t) {
    using c10::DispatchKey;
    const auto keys = t.key_set();
    return t.is_cuda() && t.layout() == at::kStrided && !t.is_neg() && !keys.has(DispatchKey::Python) && !keys.has(DispatchKey::FuncTorchGradWrapper) &&
           !keys.has(DispatchKey::FuncTorchBatched);
}

// What an entry point asks first, with the GIL held (it looks at the Python objects).  The Python path has to run for Python subclasses
// of Tensor, which see its operators; for forward-mode duals, for which its autograd functions raise; and under torch.jit.trace, which
// records those functions but would see nothing here besides allocations.
struct Eager {
    const bool duals;  // whether there can be any: asked tensor by tensor, it costs a decode step 0.2 of its 6 us
    explicit Eager(bool autograd) : duals(autograd && torch::autograd::ForwardADLevel::try_get_by_idx(0) != nullptr) {}
    bool operator()(const Tensor& t) const {
        PyObject* o = t.defined() ? t.unsafeGetTensorImpl()->pyobj_slot()->load_pyobj() : nullptr;
        return !o || (THPVariable_CheckExact(o) && !(duals && t._fw_grad(0).defined()));
    }
};
bool eager(std::initializer_list<const Tensor*> ts, bool autograd = true) {  // autograd: the Python form has an autograd function
    const Eager ok(autograd);
    for (const Tensor* t : ts)
        if (!ok(*t)) return false;
    return !at::tracer::impl::is_dispatch_enabled();
}
bool eager(const variable_list& ts) {
    const Eager ok(true);
    for (const Tensor& t : ts)
        if (!ok(t)) return false;
    return !at::tracer::impl::is_dispatch_enabled();
}

// A tensor whose elements lie back to back from a 16-byte boundary on.  Backward nodes ask it of what they have saved: hooks on
// saved tensors hand back the same values, but in a layout of their own.
Tensor dense(const Tensor& t) {
    if (!t.defined() || (t.is_contiguous() && !(reinterpret_cast<uintptr_t>(t.data_ptr()) & 15))) return t;
    return t.clone(at::MemoryFormat::Contiguous);
}

// F::apply on the first sizeof...(I) tensors of a list: autograd sees tensors that are arguments of their own, not those in a list
template <typename F, size_t... I>
auto apply_list(const variable_list& in, std::index_sequence<I...>) { return F::apply(in[I]...); }

// ---- WKV7 ------------------------------------------------------------------------------------------
// [B,T,H*64] tensors with one layout whose rows are whole, 16-byte aligned and apart: outputs and gradients take the same layout, and
// rows of windows or expanded batches that share memory would be written over one another
struct Rows { int64_t B, T, H, sb, st; int io; };
Rows rows(const Tensor& w) {
    return Rows{w.size(0), w.size(1), w.size(2) / N, w.stride(0), w.stride(1), w.scalar_type() == at::kBFloat16 ? WKV7_BF16 : WKV7_F32};
}
bool rows_of(std::initializer_list<const Tensor*> ts, Rows& r) {
    const Tensor& w = **ts.begin();
    if (!plain(w) || w.dim() != 3) return false;
    const auto dt = w.scalar_type();
    if (dt != at::kBFloat16 && dt != at::kFloat) return false;
    const int64_t per16 = dt == at::kBFloat16 ? 8 : 4;
    if (w.size(2) % N != 0 || w.size(0) == 0 || w.size(1) == 0 || w.size(2) == 0) return false;
    r = rows(w);
    if (w.stride(2) != 1 || r.sb % per16 || r.st % per16 || r.st < w.size(2)) return false;
    const int64_t row = w.size(2);
    if (r.B > 1 && r.sb < (r.T - 1) * r.st + row && (r.sb < row || r.st < (r.B - 1) * r.sb + row)) return false;  // [B][T] or [T][B] order
    for (const Tensor* t : ts)
        if (!plain(*t) || t->scalar_type() != dt || t->sizes() != w.sizes() || t->strides() != w.strides() || t->device() != w.device() ||
            (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15))
            return false;
    return true;
}
bool state_ok(const OptTensor& s, const Rows& r, const Tensor& like) {
    if (!s || !s->defined()) return true;
    return plain(*s) && s->scalar_type() == at::kFloat && s->is_contiguous() && s->device() == like.device() && s->dim() == 4 && s->size(0) == r.B &&
           s->size(1) == r.H && s->size(2) == N && s->size(3) == N;
}
Tensor like_rows(const Tensor& t) { return at::empty_strided(t.sizes(), t.strides(), t.options()); }
Tensor states(const Tensor& like, const Rows& r) { return at::empty({r.B, r.H, N, N}, like.options().dtype(at::kFloat)); }

// forward; g, params defined: attn_ln.  Returns y, sT, checkpoints (undefined without save)
variable_list wkv_forward(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b, const Tensor& g,
                          const Tensor& params, const Tensor& s0, bool save) {
    const Rows q = rows(w);
    Tensor y = like_rows(v), sT = states(w, q), ck;
    if (save) ck = at::empty({wkv7_checkpoint_bytes(q.B, q.T, q.H, N) / 4}, sT.options());
    Tensor ws = scratch(w);
    if (g.defined())
        check(wkv7_attn_ln_fwd_ws(r.data_ptr(), w.data_ptr(), k.data_ptr(), v.data_ptr(), a.data_ptr(), b.data_ptr(), g.data_ptr(), f32(params), f32(s0),
                                  y.data_ptr(), f32(sT), f32(ck), LN_EPS, q.B, q.T, q.H, N, q.sb, q.st, N, q.io, ws.data_ptr(), stream()), "wkv7_attn_ln_fwd_ws");
    else
        check(wkv7_fwd_ws(r.data_ptr(), w.data_ptr(), k.data_ptr(), v.data_ptr(), a.data_ptr(), b.data_ptr(), f32(s0), y.data_ptr(), f32(sT), f32(ck),
                          q.B, q.T, q.H, N, q.sb, q.st, N, q.io, ws.data_ptr(), stream()), "wkv7_fwd_ws");
    return {y, sT, ck};
}
// backward.  Returns dr, dw, dk, dv, da, db, ds0 (, dg, dparams)
variable_list wkv_backward(Tensor r, Tensor w, Tensor k, Tensor v, Tensor a, Tensor b, Tensor g, Tensor params, Tensor ck, Tensor sT, Tensor dy, Tensor dsT) {
    Rows q;
    if (!rows_of({&w, &r, &k, &v, &a, &b}, q) || (g.defined() && !rows_of({&w, &g}, q))) {
        for (Tensor* t : {&r, &w, &k, &v, &a, &b, &g}) *t = dense(*t);
        q = rows(w);
    }
    for (Tensor* t : {&params, &ck, &sT}) *t = dense(*t);
    if (!dy.defined()) dy = at::zeros_like(v);
    if (dy.scalar_type() != w.scalar_type()) dy = dy.to(w.scalar_type());
    if (dy.strides() != w.strides() || (reinterpret_cast<uintptr_t>(dy.data_ptr()) & 15)) {
        Tensor d = like_rows(w);
        d.copy_(dy);
        dy = d;
    }
    if (dsT.defined()) dsT = dsT.to(at::kFloat).contiguous();
    Tensor dr = like_rows(w), dw = like_rows(w), dk = like_rows(w), dv = like_rows(w), da = like_rows(w), db = like_rows(w), ds0 = states(w, q);
    const Tensor ws = bwd_scratch((g.defined() ? wkv7_attn_ln_bwd_ws_bytes : wkv7_bwd_ws_bytes)(q.B, q.T, q.H, N, q.io), w);
    void* const wsp = ws.defined() ? ws.data_ptr() : nullptr;
    const float* sTp = dsT.defined() ? f32(sT) : nullptr;
    if (!g.defined()) {
        check(wkv7_bwd_ws(r.data_ptr(), w.data_ptr(), k.data_ptr(), v.data_ptr(), a.data_ptr(), b.data_ptr(), dy.data_ptr(), f32(ck), f32(dsT), sTp,
                          dr.data_ptr(), dw.data_ptr(), dk.data_ptr(), dv.data_ptr(), da.data_ptr(), db.data_ptr(), f32(ds0), q.B, q.T, q.H, N, q.sb, q.st, N,
                          q.io, wsp, stream()), "wkv7_bwd_ws");
        return {dr, dw, dk, dv, da, db, ds0};
    }
    Tensor dg = like_rows(w), dp = at::empty({3, q.H * N}, ds0.options()), part = at::empty({q.B, 3, q.H * N}, ds0.options());
    check(wkv7_attn_ln_bwd_ws(r.data_ptr(), w.data_ptr(), k.data_ptr(), v.data_ptr(), a.data_ptr(), b.data_ptr(), g.data_ptr(), f32(params), dy.data_ptr(),
                              f32(ck), f32(dsT), sTp, dr.data_ptr(), dw.data_ptr(), dk.data_ptr(), dv.data_ptr(), da.data_ptr(), db.data_ptr(), dg.data_ptr(),
                              f32(dp), f32(part), f32(ds0), LN_EPS, q.B, q.T, q.H, N, q.sb, q.st, N, q.io, wsp, stream()), "wkv7_attn_ln_bwd_ws");
    return {dr, dw, dk, dv, da, db, ds0, dg, dp};
}

// r, w, k, v, a, b (, g, params), s0 -> y, sT
struct WkvFn : public Function<WkvFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b,
                                 const OptTensor& g_, const OptTensor& params_, const OptTensor& s0_) {
        const Tensor g = g_.value_or(Tensor()), params = params_.value_or(Tensor()), s0 = s0_.value_or(Tensor());
        const variable_list o = wkv_forward(r, w, k, v, a, b, g, params, s0, true);
        ctx->save_for_backward({r, w, k, v, a, b, g, params, o[2], o[1]});
        ctx->set_materialize_grads(false);
        ctx->saved_data["s0"] = s0.defined();
        return {o[0], o[1]};
    }
    static variable_list backward(AutogradContext* ctx, variable_list go) {
        const variable_list s = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard guard(s[1].device());
        at::NoGradGuard ng;
        const variable_list d = wkv_backward(s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8], s[9], go[0], go[1]);
        return {d[0], d[1], d[2], d[3], d[4], d[5], d.size() > 7 ? d[7] : Tensor(), d.size() > 7 ? d[8] : Tensor(),
                ctx->saved_data["s0"].toBool() ? d[6] : Tensor()};
    }
};

py::object wkv(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b, const Tensor& g, const Tensor& params,
               const OptTensor& s0, bool return_state) {
    Rows q;
    const Tensor st = s0.value_or(Tensor());
    if (!eager({&r, &w, &k, &v, &a, &b, &g, &params, &st}) || !rows_of({&w, &r, &k, &v, &a, &b}, q) || !state_ok(s0, q, w)) return py::none();
    if (g.defined()) {
        if (!rows_of({&w, &g}, q)) return py::none();
        if (!plain(params) || params.scalar_type() != at::kFloat || !params.is_contiguous() || params.device() != w.device() || params.dim() != 2 ||
            params.size(0) != 3 || params.size(1) != q.H * N)
            return py::none();
    }
    Tensor y, sT;
    {
        py::gil_scoped_release nogil;
        const c10::cuda::CUDAGuard guard(w.device());
        variable_list o;
        if (grad_wanted({&r, &w, &k, &v, &a, &b, &g, &params, &st})) {
            const auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
            o = WkvFn::apply(r, w, k, v, a, b, opt(g), opt(params), opt(st));
        } else {
            at::NoGradGuard ng;
            o = wkv_forward(r, w, k, v, a, b, g, params, st, false);
        }
        y = o[0];
        sT = o[1];
    }
    if (return_state) return py::make_tuple(y, sT);
    return py::cast(y);
}
py::object attn(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b, const OptTensor& s0, bool return_state) {
    return wkv(r, w, k, v, a, b, Tensor(), Tensor(), s0, return_state);
}
py::object attn_ln(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b, const Tensor& g, const Tensor& params,
                   const OptTensor& s0, bool return_state) {
    return wkv(r, w, k, v, a, b, g, params, s0, return_state);
}

// decode: (y, state)
py::object attn_step(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b, const OptTensor& state, bool inplace) {
    Rows q;
    const Tensor st = state.value_or(Tensor());
    if (!eager({&r, &w, &k, &v, &a, &b, &st}, false) || !rows_of({&w, &r, &k, &v, &a, &b}, q) || !state_ok(state, q, w)) return py::none();
    Tensor y, sT;
    {
        py::gil_scoped_release nogil;
        const c10::cuda::CUDAGuard guard(w.device());
        at::NoGradGuard ng;
        y = like_rows(v);
        sT = inplace && st.defined() ? st : states(w, q);
        check(wkv7_step(r.data_ptr(), w.data_ptr(), k.data_ptr(), v.data_ptr(), a.data_ptr(), b.data_ptr(), f32(st),
                        y.data_ptr(), f32(sT), q.B, q.T, q.H, N, q.sb, q.st, N, q.io, stream()), "wkv7_step");
    }
    return py::make_tuple(y, sT);
}

// ---- several tensors converted in one launch ---------------------------------------------------------
struct Casts {
    const void* src[WKV7_CAST_MAX];
    void* dst[WKV7_CAST_MAX];
    int64_t numel[WKV7_CAST_MAX];
    int kind[WKV7_CAST_MAX], count = 0;
    void add(const Tensor& s, void* d, int k) { src[count] = s.data_ptr(); dst[count] = d; numel[count] = s.numel(); kind[count++] = k; }
    void run() { if (count) check(wkv7_cast(src, dst, numel, kind, count, stream()), "wkv7_cast"); }
};
bool castable(const Tensor& p, at::Device dev) {  // a parameter the conversion kernel takes
    return plain(p) && p.device() == dev && p.scalar_type() == at::kFloat && p.is_contiguous() && p.numel() % 8 == 0 && !(reinterpret_cast<uintptr_t>(p.data_ptr()) & 15);
}
// bf16 copies of fp32 parameters, back to back in one buffer
Tensor cast_params(const variable_list& ps, std::vector<Tensor>& out) {
    int64_t n = 0;
    for (const Tensor& p : ps) n += p.numel();
    Tensor buf = at::empty({n}, ps[0].options().dtype(at::kBFloat16));
    Casts c;
    n = 0;
    for (const Tensor& p : ps) {
        out.push_back(buf.narrow(0, n, p.numel()).view(p.sizes()));
        c.add(p, out.back().data_ptr(), 0);
        n += p.numel();
    }
    c.run();
    return buf;
}
bool bf16_dense(const Tensor& t) { return plain(t) && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && !(reinterpret_cast<uintptr_t>(t.data_ptr()) & 15); }
Tensor dense_bf16(const Tensor& t, const Tensor& like) {  // a gradient as its kernel wants it
    if (!t.defined()) return at::zeros_like(like);
    Tensor u = t.to(at::kBFloat16).contiguous();
    return reinterpret_cast<uintptr_t>(u.data_ptr()) & 15 ? u.clone() : u;
}

// ---- ddlerp -------------------------------------------------------------------------------------------
void ddlerp_forward(const Tensor& x, const std::vector<Tensor>& p, Tensor& m, Tensor& y) {  // p: alpha, L, R, beta in bf16
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), D = p[2].size(2);
    m = at::empty({B, T, 4 * D}, x.options());
    y = at::empty({4, B, T, C}, x.options());
    Tensor ws = at::empty({(int64_t)wkv7_ddlerp_fwd_tc_workspace_bytes(C, D)}, x.options().dtype(at::kByte));
    check(wkv7_ddlerp_fwd_tc(x.data_ptr(), p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), p[3].data_ptr(), m.data_ptr(), y.data_ptr(), ws.data_ptr(),
                             B, T, C, D, stream()), "wkv7_ddlerp_fwd_tc");
}
// dx, dalpha, dL, dR, dbeta (parameter gradients fp32)
variable_list ddlerp_backward(const Tensor& x, const std::vector<Tensor>& p, const Tensor& m, const Tensor& d0, const Tensor& d1, const Tensor& d2, const Tensor& d3) {
    const int64_t B = x.size(0), T = x.size(1), C = x.size(2), D = p[2].size(2);
    const auto f = x.options().dtype(at::kFloat);
    Tensor dpre = at::empty({B, T, 4 * D}, x.options()), dx = at::empty_like(x), dalpha = at::empty({C}, f), dL = at::empty({4 * D, C}, f),
           dR = at::empty({4, C, D}, f), dbeta = at::empty({4, 1, 1, C}, f);
    Tensor ws = at::empty({(int64_t)wkv7_ddlerp_bwd_tc_workspace_bytes(C, D)}, x.options().dtype(at::kByte));
    check(wkv7_ddlerp_bwd_tc(x.data_ptr(), p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), p[3].data_ptr(), m.data_ptr(), d0.data_ptr(), d1.data_ptr(),
                             d2.data_ptr(), d3.data_ptr(), dpre.data_ptr(), dx.data_ptr(), f32(dalpha), f32(dL), f32(dR), f32(dbeta), ws.data_ptr(),
                             B, T, C, D, stream()), "wkv7_ddlerp_bwd_tc");
    return {dx, dalpha, dL, dR, dbeta};
}
struct DdlerpFn : public Function<DdlerpFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& alpha, const Tensor& L, const Tensor& R, const Tensor& beta) {
        std::vector<Tensor> p;
        cast_params({alpha, L, R, beta}, p);
        Tensor m, y;
        ddlerp_forward(x, p, m, y);
        ctx->save_for_backward({x, p[0], p[1], p[2], p[3], m});
        ctx->set_materialize_grads(false);
        return y.unbind(0);
    }
    static variable_list backward(AutogradContext* ctx, variable_list go) {
        variable_list s = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard guard(s[0].device());
        at::NoGradGuard ng;
        for (Tensor& t : s) t = dense(t);
        return ddlerp_backward(s[0], {s[1], s[2], s[3], s[4]}, s[5], dense_bf16(go[0], s[0]), dense_bf16(go[1], s[0]), dense_bf16(go[2], s[0]), dense_bf16(go[3], s[0]));
    }
};
py::object ddlerp(const Tensor& x, const Tensor& alpha, const Tensor& L, const Tensor& R, const Tensor& beta) {
    if (!eager({&x, &alpha, &L, &R, &beta}) || !bf16_dense(x) || x.dim() != 3 || x.numel() == 0 || x.size(2) % 64 != 0) return py::none();
    const int64_t C = x.size(2);
    for (const Tensor* t : {&alpha, &L, &R, &beta})
        if (!castable(*t, x.device())) return py::none();
    if (R.dim() != 3 || R.size(0) != 4 || R.size(1) != C || alpha.dim() != 1 || alpha.size(0) != C || L.dim() != 2 || L.size(0) != 4 * R.size(2) || L.size(1) != C ||
        beta.dim() != 4 || beta.size(0) != 4 || beta.size(3) != C || beta.numel() != 4 * C)
        return py::none();
    variable_list y;
    {
        py::gil_scoped_release nogil;
        const c10::cuda::CUDAGuard guard(x.device());
        if (grad_wanted({&x, &alpha, &L, &R, &beta})) {
            y = DdlerpFn::apply(x, alpha, L, R, beta);
        } else {
            at::NoGradGuard ng;
            std::vector<Tensor> p;
            cast_params({alpha, L, R, beta}, p);
            Tensor m, z;
            ddlerp_forward(x, p, m, z);
            y = z.unbind(0);
        }
    }
    return py::make_tuple(y[0], y[1], y[2], y[3]);
}

// ---- expand_loras -----------------------------------------------------------------------------------------
// a [B,T,D] tensor whose rows (pitch ld) the kernels can read as they lie
bool pitched(const Tensor& t, int64_t B, int64_t T, int64_t D, int64_t* ld) {
    if (!plain(t) || t.scalar_type() != at::kBFloat16 || t.dim() != 3 || t.size(0) != B || t.size(1) != T || t.size(2) != D || t.stride(2) != 1) return false;
    *ld = T > 1 ? t.stride(1) : B > 1 ? t.stride(0) : D;
    return *ld >= D && *ld % 8 == 0 && (B == 1 || t.stride(0) == T * *ld) && !(reinterpret_cast<uintptr_t>(t.data_ptr()) & 15);
}
// acts: w_in, k_in, z_in, a_in, ma_in, mk_in; p: Wz, Wa, Wma, Wmk, w_bias, a_bias, ma_bias, mk_bias in bf16.  Returns w, k, kk, b
variable_list loras_forward(const variable_list& a, const int64_t* ld, const std::vector<Tensor>& p) {
    const int64_t B = a[0].size(0), T = a[0].size(1), C = a[0].size(2), D = p[0].size(1);
    variable_list o;
    for (int i = 0; i < 4; ++i) o.push_back(at::empty({B, T, C}, a[0].options()));
    check(wkv7_expand_loras_fwd_ld(a[0].data_ptr(), a[1].data_ptr(), a[2].data_ptr(), a[3].data_ptr(), a[4].data_ptr(), a[5].data_ptr(), ld, p[0].data_ptr(),
                                   p[1].data_ptr(), p[2].data_ptr(), p[3].data_ptr(), p[4].data_ptr(), p[5].data_ptr(), p[6].data_ptr(), p[7].data_ptr(),
                                   o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), o[3].data_ptr(), B, T, C, D, stream()), "wkv7_expand_loras_fwd");
    return o;
}
// d: dw, dk, dkk, db.  Writes the rank-D input gradients to da[0..3] (pitches ldg); returns dw_in, dk_in, 4 weight, 4 bias gradients (fp32, one buffer)
variable_list loras_backward(const variable_list& a, const int64_t* ld, const std::vector<Tensor>& p, const variable_list& d, const variable_list& da, const int64_t* ldg) {
    const int64_t B = a[0].size(0), T = a[0].size(1), C = a[0].size(2), D = p[0].size(1);
    Tensor dw = at::empty({B, T, C}, a[0].options()), dk = at::empty({B, T, C}, a[0].options());
    Tensor buf = at::empty({4 * C * D + 4 * C}, a[0].options().dtype(at::kFloat));
    variable_list o{dw, dk};
    for (int i = 0; i < 4; ++i) o.push_back(buf.narrow(0, i * C * D, C * D).view({C, D}));
    for (int i = 0; i < 4; ++i) o.push_back(buf.narrow(0, 4 * C * D + i * C, C));
    Tensor ws = at::empty({std::max<int64_t>(16, wkv7_expand_loras_bwd_workspace_bytes(B, T, C, D))}, a[0].options().dtype(at::kByte));
    check(wkv7_expand_loras_bwd_ld(a[0].data_ptr(), a[1].data_ptr(), a[2].data_ptr(), a[3].data_ptr(), a[4].data_ptr(), a[5].data_ptr(), ld, p[0].data_ptr(),
                                   p[1].data_ptr(), p[2].data_ptr(), p[3].data_ptr(), p[4].data_ptr(), p[5].data_ptr(), p[6].data_ptr(), p[7].data_ptr(),
                                   d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(), dw.data_ptr(), dk.data_ptr(), da[0].data_ptr(),
                                   da[1].data_ptr(), da[2].data_ptr(), da[3].data_ptr(), ldg, f32(o[2]), f32(o[3]), f32(o[4]), f32(o[5]), f32(o[6]), f32(o[7]),
                                   f32(o[8]), f32(o[9]), ws.data_ptr(), B, T, C, D, stream()), "wkv7_expand_loras_bwd");
    return o;
}
struct LorasFn : public Function<LorasFn> {
    // in: six activations, eight parameters
    template <typename... Ts>
    static variable_list forward(AutogradContext* ctx, const Ts&... args) {
        const variable_list in{args...}, a(in.begin(), in.begin() + 6);
        std::vector<Tensor> p;
        cast_params(variable_list(in.begin() + 6, in.end()), p);
        int64_t ld[4];
        for (int i = 0; i < 4; ++i) pitched(a[2 + i], a[0].size(0), a[0].size(1), p[0].size(1), ld + i);
        variable_list s = a;
        s.insert(s.end(), p.begin(), p.end());
        ctx->save_for_backward(s);
        ctx->set_materialize_grads(false);
        return loras_forward(a, ld, p);
    }
    static variable_list backward(AutogradContext* ctx, variable_list go) {
        const variable_list s = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard guard(s[0].device());
        at::NoGradGuard ng;
        variable_list a(s.begin(), s.begin() + 6);
        std::vector<Tensor> p(s.begin() + 6, s.end());
        for (Tensor& t : p) t = dense(t);
        a[0] = dense(a[0]);
        a[1] = dense(a[1]);
        const int64_t B = a[0].size(0), T = a[0].size(1), D = p[0].size(1);
        int64_t ld[4];
        variable_list d, da;
        for (int i = 0; i < 4; ++i) {
            if (!pitched(a[2 + i], B, T, D, ld + i)) {
                a[2 + i] = dense(a[2 + i]);
                ld[i] = D;
            }
            d.push_back(dense_bf16(go[i], a[0]));
            da.push_back(at::empty({B, T, D}, a[0].options()));
        }
        const variable_list o = loras_backward(a, ld, p, d, da, nullptr);
        return {o[0], o[1], da[0], da[1], da[2], da[3], o[2], o[3], o[4], o[5], o[6], o[7], o[8], o[9]};
    }
};
py::object expand_loras(const variable_list& in) {
    const Tensor& w = in[0];
    if (!eager(in) || !bf16_dense(w) || w.dim() != 3 || w.numel() == 0 || w.size(2) % 64 != 0 || !bf16_dense(in[1]) || in[1].sizes() != w.sizes() || in[6].dim() != 2) return py::none();
    const int64_t C = w.size(2), D = in[6].size(1);
    int64_t ld[4];
    for (int i = 0; i < 4; ++i)
        if (!pitched(in[2 + i], w.size(0), w.size(1), D, ld + i) || in[2 + i].device() != w.device()) return py::none();
    for (int i = 6; i < 14; ++i) {
        if (!castable(in[i], w.device())) return py::none();
        if (i < 10 ? (in[i].dim() != 2 || in[i].size(0) != C || in[i].size(1) != D) : (in[i].dim() != 1 || in[i].size(0) != C)) return py::none();
    }
    if (in[1].device() != w.device() || (D != 16 && D != 32 && D != 64 && D != 128)) return py::none();
    variable_list o;
    {
        py::gil_scoped_release nogil;
        const c10::cuda::CUDAGuard guard(w.device());
        bool grad = false;
        for (const Tensor& t : in) grad = grad || grad_wanted({&t});
        if (grad) {
            o = apply_list<LorasFn>(in, std::make_index_sequence<14>{});
        } else {
            at::NoGradGuard ng;
            std::vector<Tensor> p;
            cast_params(variable_list(in.begin() + 6, in.end()), p);
            o = loras_forward(variable_list(in.begin(), in.begin() + 6), ld, p);
        }
    }
    return py::make_tuple(o[0], o[1], o[2], o[3]);
}


// ---- TimeMixer --------------------------------------------------------------------------------------------
// One autograd node for the whole layer: the ops above, the projection kernel and plain matrix products, in the order of
// time_mixer.py.  All parameters are converted by one launch, and first-stage weights that share an input lie next to each other
// there, so they need no concatenation; the backward sums into its products (beta = 1), writes the rank-D gradients into the
// columns where the next product reads them, and takes weight gradients straight in fp32.
enum { WR, WK, WV, WO, GATE1, GATE2, KKK1, MK1, DECAY1, AAA1, MA1, DECAY2, MAAX, MAA1, MAA2, MAA, KKK2, AAA2, MA2, MK2, DECAY, AAAAA, MISCA, MISCK, NBF,
       LNW = NBF, LNB, FAAAA, NPAR };
constexpr int64_t MIX = 32, DEC = 64, SMALL = 16, GATE = 128, WAM = DEC + 2 * SMALL;

// rows of x may be columns of a wider tensor; tanh on the first `to` columns of the result
struct Proj { Tensor x; const Tensor& w; int64_t to; Tensor* out; };
void proj(std::initializer_list<Proj> ps) {
    constexpr int MAX = WKV7_PROJ_LD_MAX;
    const void *a[MAX], *b[MAX];
    void* c[MAX];
    int64_t n[MAX], k[MAX], lda[MAX], from[MAX] = {}, to[MAX];
    int i = 0;
    for (const Proj& p : ps) {
        *p.out = at::empty({p.x.size(0), p.w.size(0)}, p.x.options());
        a[i] = p.x.data_ptr(); b[i] = p.w.data_ptr(); c[i] = p.out->data_ptr(); n[i] = p.w.size(0); k[i] = p.x.size(1); lda[i] = p.x.stride(0); to[i++] = p.to;
    }
    check(wkv7_proj_gemm_group_ld(i, a, b, c, n, k, lda, from, to, ps.begin()->x.size(0), stream()), "wkv7_proj_gemm_group_ld");
}
// Tiles of 128 x 128 an SM, times two, in one launch of all the mixer's first-stage products, three C x C ones among them: with few rows (M = B T)
// at::mm, the better kernel with many, leaves half of the SMs idle, one product after the other, and its calls cost the host 10 us
// each.  Up to four tiles an SM this library's kernel takes the first stages in one launch; up to one and a half, where the host is
// what the layer waits for, the second stages (one launch) and the output projection, too.  Layer in us, all at::mm -> first -> all:
//   C = 512, 256 rows (0.2 tiles an SM)  157 -> 130 -> 111      C = 768, 1280 rows (1.4)   159 -> 131 -> 119
//   C = 2048, 515 rows (1.7)             174 -> 153 -> 155      C = 2048, 1280 rows (3.5)  201 -> 191 -> 198
//   C = 2048, 1792 rows (4.8)            297 -> 296             C = 2048, 2400 rows (6.6)  277 -> 287
int64_t half_tiles(int64_t M, int64_t C) {
    const int64_t tiles = (M + 127) / 128 * (3 * ((C + 127) / 128) + 3), sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    return (2 * tiles + sms - 1) / sms;
}
struct Mixer {
    int64_t B, T, C;
    std::vector<Tensor> p;                   // bf16 copies, in the order of the enum
    Tensor params, kkmk_w, wam_w;            // [3,C] fp32; kkk_w1 | mk_w1; decay_w1 | aaa_w1 | ma_w1
    Tensor m, y4, r, g1, g, k0, kkmk, v, wam, w2, w, k, kk, b, y, sT, ck;

    void convert(const variable_list& in) {
        int64_t n = 0;
        for (int i = 0; i < NBF; ++i) n += in[i].numel();
        Tensor buf = at::empty({n}, in[0].options().dtype(at::kBFloat16));
        params = at::empty({3, C}, in[0].options());
        Casts c;
        int64_t at_kk = 0, at_wam = 0;
        n = 0;
        for (int i = 0; i < NBF; ++i) {
            if (i == KKK1) at_kk = n;
            if (i == DECAY1) at_wam = n;
            p.push_back(buf.narrow(0, n, in[i].numel()).view(in[i].sizes()));
            c.add(in[i], p.back().data_ptr(), 0);
            n += in[i].numel();
        }
        kkmk_w = buf.narrow(0, at_kk, 2 * SMALL * C).view({2 * SMALL, C});
        wam_w = buf.narrow(0, at_wam, WAM * C).view({WAM, C});
        for (int i = 0; i < 3; ++i) c.add(in[LNW + i], params.data_ptr<float>() + i * C, 2);
        c.run();
    }
    Tensor rows(const Tensor& t) const { return t.view({B * T, t.size(-1)}); }
    Tensor seq(const Tensor& t) const { return t.view({B, T, t.size(-1)}); }
    Tensor in4(int i) const { return rows(y4.select(0, i)); }
    variable_list loras_in() const {
        const Tensor a = seq(kkmk), c = seq(wam);
        return {w2, k0, a.narrow(2, 0, SMALL), c.narrow(2, DEC, SMALL), c.narrow(2, DEC + SMALL, SMALL), a.narrow(2, SMALL, SMALL)};
    }
    std::vector<Tensor> loras_par() const { return {p.begin() + KKK2, p.begin() + NBF}; }
    std::vector<Tensor> ddlerp_par() const { return {p.begin() + MAAX, p.begin() + MAA + 1}; }

    Tensor forward(const Tensor& x, const variable_list& in, bool save) {
        B = x.size(0); T = x.size(1); C = x.size(2);
        convert(in);
        ddlerp_forward(x, ddlerp_par(), m, y4);
        const Tensor xrg = in4(0), xwa = in4(1), xk = in4(2), xv = in4(3);
        const int64_t load = half_tiles(B * T, C);
        Tensor r2, k2, v2, g2, w22, out;
        if (load <= 8) {
            proj({{xrg, p[WR], 0, &r2}, {xk, p[WK], 0, &k2}, {xv, p[WV], 0, &v2}, {xrg, p[GATE1], GATE, &g1}, {xk, kkmk_w, 0, &kkmk}, {xwa, wam_w, DEC, &wam}});
        } else {
            r2 = at::mm(xrg, p[WR].t());
            proj({{xrg, p[GATE1], GATE, &g1}, {xk, kkmk_w, 0, &kkmk}, {xwa, wam_w, DEC, &wam}});
            k2 = at::mm(xk, p[WK].t());
            v2 = at::mm(xv, p[WV].t());
        }
        if (load <= 3) {
            proj({{g1, p[GATE2], 0, &g2}, {wam.narrow(1, 0, DEC), p[DECAY2], 0, &w22}});
        } else {
            g2 = at::mm(g1, p[GATE2].t());
            w22 = at::mm(wam.narrow(1, 0, DEC), p[DECAY2].t());
        }
        r = seq(r2); k0 = seq(k2); v = seq(v2); g = seq(g2); w2 = seq(w22);
        if (!save) y4 = m = Tensor();
        const int64_t ld[4] = {2 * SMALL, WAM, WAM, 2 * SMALL};
        const variable_list o = loras_forward(loras_in(), ld, loras_par());
        w = o[0]; k = o[1]; kk = o[2]; b = o[3];
        if (!save) k0 = w2 = Tensor();
        const variable_list a = wkv_forward(r, w, k, v, kk, b, g, params, Tensor(), save);
        y = a[0]; sT = a[1]; ck = a[2];
        if (load > 3) return seq(at::mm(rows(y), p[WO].t()));
        proj({{rows(y), p[WO], 0, &out}});
        return seq(out);
    }
    variable_list saved() const {
        variable_list s{params, kkmk_w, wam_w, m, y4, r, g1, g, k0, kkmk, v, wam, w2, w, k, kk, b, y, sT, ck};
        s.insert(s.end(), p.begin(), p.end());
        return s;
    }
    explicit Mixer(const variable_list& s) {
        Tensor* f[] = {&params, &kkmk_w, &wam_w, &m, &y4, &r, &g1, &g, &k0, &kkmk, &v, &wam, &w2, &w, &k, &kk, &b, &y, &sT, &ck};
        size_t i = 0;
        for (Tensor* t : f) *t = dense(s[i++]);
        for (; i < s.size(); ++i) p.push_back(dense(s[i]));
        B = r.size(0); T = r.size(1); C = r.size(2);
    }
    Mixer() = default;

    // the parameters' gradients, then dx; `want(i)`: parameter i has a use for its gradient
    template <typename Want>
    variable_list backward(const Tensor& x, Tensor dout, Want want) {
        variable_list d(NPAR + 1);
        auto grad = [&](int i, const Tensor& dpre, const Tensor& in) { if (want(i)) d[i] = at::mm(dpre.t(), in, at::kFloat); };
        // a group of weights with one input: rows of one product
        auto group = [&](std::initializer_list<int> is, const Tensor& dpre, const Tensor& in) {
            bool any = false;
            for (int i : is) any = any || want(i);
            if (!any) return;
            const Tensor all = at::mm(dpre.t(), in, at::kFloat);
            int64_t at_row = 0;
            for (int i : is) {
                const int64_t n = p[i].size(0);
                d[i] = all.narrow(0, at_row, n);
                at_row += n;
            }
        };
        dout = rows(dout);
        grad(WO, dout, rows(y));
        variable_list a = wkv_backward(r, w, k, v, kk, b, g, params, ck, sT, seq(at::mm(dout, p[WO])), Tensor());
        const Tensor dr = rows(a[0]), dv = rows(a[3]), dg = rows(a[7]);
        for (int i = 0; i < 3; ++i) d[LNW + i] = a[8].select(0, i);

        Tensor dkkmk = at::empty_like(kkmk), dwam = at::empty_like(wam);
        const int64_t ld[4] = {2 * SMALL, WAM, WAM, 2 * SMALL};
        const Tensor sk = seq(dkkmk), sw = seq(dwam);
        const variable_list l = loras_backward(loras_in(), ld, loras_par(), {a[1], a[2], a[4], a[5]},
                                               {sk.narrow(2, 0, SMALL), sw.narrow(2, DEC, SMALL), sw.narrow(2, DEC + SMALL, SMALL), sk.narrow(2, SMALL, SMALL)}, ld);
        a.clear();
        for (int i = 0; i < 8; ++i) d[KKK2 + i] = l[2 + i];
        const Tensor dw2 = rows(l[0]), dk0 = rows(l[1]);

        const Tensor t = wam.narrow(1, 0, DEC);
        Tensor dt = dwam.narrow(1, 0, DEC);
        grad(DECAY2, dw2, t);
        at::mm_out(dt, dw2, p[DECAY2]);
        at::tanh_backward_out(dt, dt, t);
        grad(GATE2, dg, g1);
        Tensor dg1 = at::mm(dg, p[GATE2]);
        at::tanh_backward_out(dg1, dg1, g1);

        const Tensor xrg = in4(0), xwa = in4(1), xk = in4(2), xv = in4(3);
        group({DECAY1, AAA1, MA1}, dwam, xwa);
        const Tensor dxwa = at::mm(dwam, wam_w);
        grad(WK, dk0, xk);
        group({KKK1, MK1}, dkkmk, xk);
        const Tensor dxk = at::mm(dk0, p[WK]).addmm_(dkkmk, kkmk_w);
        grad(WV, dv, xv);
        const Tensor dxv = at::mm(dv, p[WV]);
        grad(WR, dr, xrg);
        grad(GATE1, dg1, xrg);
        const Tensor dxrg = at::mm(dr, p[WR]).addmm_(dg1, p[GATE1]);
        const variable_list q = ddlerp_backward(x, ddlerp_par(), m, dxrg, dxwa, dxk, dxv);
        d[NPAR] = q[0];
        for (int i = 0; i < 4; ++i) d[MAAX + i] = q[1 + i];
        return d;
    }
};
struct MixerFn : public Function<MixerFn> {
    // in: the parameters in the order of the enum, then x
    template <typename... Ts>
    static Tensor forward(AutogradContext* ctx, const Ts&... args) {
        const variable_list in{args...};
        const Tensor x = in.back();
        Mixer mx;
        const Tensor out = mx.forward(x, in, true);
        variable_list s = mx.saved();
        s.push_back(x);
        ctx->save_for_backward(s);
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list go) {
        variable_list s = ctx->get_saved_variables();
        const Tensor x = dense(s.back());
        s.pop_back();
        const c10::cuda::CUDAGuard guard(x.device());
        at::NoGradGuard ng;
        return Mixer(s).backward(x, dense_bf16(go[0], x), [&](int i) { return ctx->needs_input_grad(i); });
    }
};
py::object mixer(Tensor x, const variable_list& in) {
    if (!eager({&x}) || !eager(in) || !plain(x) || x.dim() != 3 || x.numel() == 0 || x.size(2) % N != 0 || (int)in.size() != NPAR || at::autocast::is_autocast_enabled(at::kCUDA)) return py::none();
    if (x.scalar_type() != at::kBFloat16 && x.scalar_type() != at::kFloat) return py::none();
    const int64_t C = x.size(2);
    const std::array<std::vector<int64_t>, NPAR> shape{{{C, C}, {C, C}, {C, C}, {C, C}, {GATE, C}, {C, GATE}, {SMALL, C}, {SMALL, C}, {DEC, C}, {SMALL, C}, {SMALL, C},
        {C, DEC}, {C}, {4 * MIX, C}, {4, C, MIX}, {4, 1, 1, C}, {C, SMALL}, {C, SMALL}, {C, SMALL}, {C, SMALL}, {C}, {C}, {C}, {C}, {C}, {C}, {C}}};
    bool grad = x.requires_grad();
    for (int i = 0; i < NPAR; ++i) {
        if (!castable(in[i], x.device()) || in[i].sizes() != at::IntArrayRef(shape[i])) return py::none();
        grad = grad || in[i].requires_grad();
    }
    Tensor out;
    {
        py::gil_scoped_release nogil;
        const c10::cuda::CUDAGuard guard(x.device());
        x = x.to(at::kBFloat16).contiguous();
        if (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) x = x.clone();
        if (grad && at::GradMode::is_enabled()) {
            variable_list all = in;
            all.push_back(x);
            out = apply_list<MixerFn>(all, std::make_index_sequence<NPAR + 1>{});
        } else {
            at::NoGradGuard ng;
            out = Mixer().forward(x, in, false);
        }
    }
    return py::cast(out);
}
}  // namespace

PYBIND11_MODULE(_wkv7_torch, mod) {
    mod.def("attn", attn);
    mod.def("attn_ln", attn_ln);
    mod.def("attn_step", attn_step);
    mod.def("ddlerp", ddlerp);
    mod.def("expand_loras", expand_loras);
    mod.def("mixer", mixer);
}
