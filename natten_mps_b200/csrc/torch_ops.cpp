// PyTorch side of the library: the CUDA and autograd kernels of torch.ops.natten_b200.* (the schemas and the Meta
// kernels are in _torch_ops.py) and the argument parsing of the functional API, all in native code.
//
// A call of na2d() used to spend 60 (forward) to 330 (with backward) microseconds in Python: argument checks, a
// Python-implemented operator and autograd formula, ctypes marshalling and a status copy per launch.  The smaller
// half of the sizes this library is used at takes less than that on the GPU.  Here the same call is one C function:
// parse, check, dispatch (so that autograd, fake tensors and tracing see the operator as before), allocate, launch.
//
// Anything the parser does not like (a wrong shape, a bad value, a tensor subclass) makes it return
// NotImplemented; functional.py then takes its own path, which raises the errors and serves the rare forms.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/autocast_mode.h>
#include <torch/library.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <optional>
#include <tuple>
#include <vector>

#include "../../include/natten_b200.h"

namespace {

using at::IntArrayRef;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using Bools = c10::List<bool>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

std::atomic<int> g_flags{0};                 // NATTEN_FLAG_* for every call (testing aid)

// ----------------------------------------------------------------------------- C ABI helpers
int dtype_code(at::ScalarType t)
{
    switch (t) {
        case at::kFloat: return NATTEN_F32;
        case at::kHalf: return NATTEN_F16;
        case at::kBFloat16: return NATTEN_BF16;
        case at::kDouble: return NATTEN_F64;
        default: break;
    }
    TORCH_CHECK_VALUE(false, "unsupported dtype ", t, "; expected float32, float16, bfloat16 or float64");
}

at::ScalarType acc_type(at::ScalarType t) { return t == at::kDouble ? at::kDouble : at::kFloat; }

void check(int code, const char* what)
{
    if (code == 0) return;
    const char* text = natten_strerror(code);
    TORCH_CHECK_VALUE(code != NATTEN_E_INVALID, what, ": ", text, " (code ", code, ")");
    TORCH_CHECK_NOT_IMPLEMENTED(code != NATTEN_E_UNSUPPORTED, what, ": ", text, " (code ", code, ")");
    TORCH_CHECK(false, what, ": ", text, " (code ", code, ")");
}

// A kernel that gave up on a bounded wait has raised the device's word in host memory by itself: reading it costs
// nothing on the stream.  It is looked at before every launch.
void poll_status(const Tensor& t)
{
    TORCH_CHECK(natten_host_status(t.device().index()) == 0,
                "natten_b200: a tensor-core kernel gave up on a bounded wait (results since then are invalid); call "
                "natten_mps_b200._cabi.clear_status() to re-arm the device");
}

void require_cuda(std::initializer_list<const Tensor*> tensors, const Tensor& first)
{
    for (const Tensor* t : tensors) {
        if (!t || !t->defined()) continue;
        TORCH_CHECK(t->is_cuda(), "natten_mps_b200 runs on CUDA tensors only (there is no CPU fallback); got a tensor on ",
                    t->device());
        TORCH_CHECK(t->device() == first.device(), "natten_mps_b200: tensors on ", first.device(), " and ", t->device());
    }
}

// (batch, token, head) strides in elements, if the spatial axes collapse into one token axis and the channels are
// adjacent.
bool token_strides(const Tensor& t, int rank, int64_t (&s)[3])
{
    const IntArrayRef st = t.strides(), sz = t.sizes();
    const int n = rank + 3;
    if (sz[n - 1] != 1 && st[n - 1] != 1) return false;
    for (int a = rank - 1; a > 0; --a)
        if (sz[a + 1] != 1 && st[a] != st[a + 1] * sz[a + 1]) return false;
    s[0] = st[0];
    s[1] = st[rank];
    s[2] = st[n - 2];
    return true;
}

Tensor strided_input(const Tensor& t, int rank, int64_t (&s)[3])
{
    if (token_strides(t, rank, s)) return t;
    Tensor c = t.contiguous();
    token_strides(c, rank, s);
    return c;
}

struct Call {
    natten_params_t p;
    std::vector<int64_t> shape;              // scratch for output shapes
    int rank;

    // spatial extents from `t` [B, *L, ., .]; kernel geometry per axis
    Call(const Tensor& t, int64_t heads_q, int64_t heads_kv, int64_t dim, int64_t dim_v, IntArrayRef ks, IntArrayRef st,
         IntArrayRef dil, const Bools& causal)
    {
        rank = (int)t.dim() - 3;
        TORCH_CHECK_VALUE(rank >= 1 && rank <= 3 && (int)ks.size() == rank && (int)st.size() == rank &&
                              (int)dil.size() == rank && (int)causal.size() == rank,
                          "natten_b200: tensors of rank ", t.dim(), " do not match the kernel geometry");
        p = natten_params_t{};
        p.rank = rank;
        p.dtype = dtype_code(t.scalar_type());
        p.batch = (int)t.size(0);
        p.heads_q = (int)heads_q;
        p.heads_kv = (int)heads_kv;
        p.dim = (int)dim;
        p.dim_v = (int)dim_v;
        for (int a = 0; a < 3; ++a) {
            const bool on = a < rank;
            p.extent[a] = on ? (int)t.size(1 + a) : 1;
            p.kernel[a] = on ? (int)ks[a] : 1;
            p.dilation[a] = on ? (int)dil[a] : 1;
            p.stride[a] = on ? (int)st[a] : 1;
            p.causal[a] = on ? (causal[a] ? 1 : 0) : 0;
        }
        p.has_scale = 0;
        p.scale = 1.0;
        p.flags = g_flags.load(std::memory_order_relaxed);
    }
    void scale(double s) { p.has_scale = 1; p.scale = s; }

    // [B, *ceil(L / stride), heads, last...]
    IntArrayRef out_shape(int64_t heads, int64_t last)
    {
        shape.clear();
        shape.push_back(p.batch);
        for (int a = 0; a < rank; ++a) shape.push_back((p.extent[a] + p.stride[a] - 1) / p.stride[a]);
        shape.push_back(heads);
        if (last >= 0) shape.push_back(last);
        return shape;
    }
    int64_t slots() const { return (int64_t)p.kernel[0] * p.kernel[1] * p.kernel[2]; }
};

Tensor fresh(IntArrayRef shape, at::ScalarType dtype, const Tensor& like)
{
    return at::detail::empty_cuda(shape, dtype, like.device(), std::nullopt);
}
const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* out_ptr(const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
void* stream_of(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

Tensor as(const Tensor& t, at::ScalarType dtype)
{
    return (t.scalar_type() == dtype ? t : t.to(dtype)).contiguous();
}

void set_extents(natten_params_t& p, const OptTensor& extents, const Tensor& q, Tensor& held)
{
    if (!extents || !extents->defined()) return;
    held = extents->to(q.device(), at::kInt).reshape({-1, p.rank}).contiguous();
    p.extents = held.const_data_ptr<int32_t>();
}

void same_dtype(const Tensor& q, std::initializer_list<const Tensor*> others)
{
    for (const Tensor* t : others)
        TORCH_CHECK_VALUE(!t->defined() || t->scalar_type() == q.scalar_type(), "natten_b200: tensors of dtype ",
                          q.scalar_type(), " and ", t->scalar_type());
}

// ----------------------------------------------------------------------------- CUDA kernels of the operators
std::tuple<Tensor, Tensor> fused_cuda(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const OptTensor& ek_in,
                                      const OptTensor& ev_in, const OptTensor& extents, IntArrayRef ks, IntArrayRef st,
                                      IntArrayRef dil, Bools causal, double scale)
{
    Tensor ek = ek_in.value_or(Tensor()), ev = ev_in.value_or(Tensor());
    require_cuda({&q_in, &k_in, &v_in, &ek, &ev}, q_in);
    same_dtype(q_in, {&k_in, &v_in, &ek, &ev});
    Call c(q_in, q_in.size(-2), k_in.size(-2), q_in.size(-1), v_in.size(-1), ks, st, dil, causal);
    const Tensor q = strided_input(q_in, c.rank, c.p.q_stride), k = strided_input(k_in, c.rank, c.p.k_stride),
                 v = strided_input(v_in, c.rank, c.p.v_stride);
    if (ek.defined()) {
        ek = ek.contiguous();
        ev = ev.contiguous();
        c.p.n_extra = (int)ek.size(1);
    }
    c.scale(scale);
    const c10::cuda::CUDAGuard guard(q.device());
    Tensor held;
    set_extents(c.p, extents, q, held);
    Tensor out = fresh(c.out_shape(c.p.heads_q, c.p.dim_v), q.scalar_type(), q);
    Tensor lse = fresh(c.out_shape(c.p.heads_q, -1), acc_type(q.scalar_type()), q);
    poll_status(q);
    check(natten_fused_fwd(&c.p, ptr(q), ptr(k), ptr(v), ptr(ek), ptr(ev), out_ptr(out), out_ptr(lse), stream_of(q)),
          "natten_fused_fwd");
    return {out, lse};
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> fused_bwd_cuda(
    const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const OptTensor& ek_in, const OptTensor& ev_in,
    const OptTensor& extents, const Tensor& out_in, const Tensor& lse_in, const Tensor& dout_in, const OptTensor& dlse_in,
    IntArrayRef ks, IntArrayRef st, IntArrayRef dil, Bools causal, double scale)
{
    Tensor ek = ek_in.value_or(Tensor()), ev = ev_in.value_or(Tensor()), dlse = dlse_in.value_or(Tensor());
    require_cuda({&q_in, &k_in, &v_in, &ek, &ev, &out_in, &lse_in, &dout_in, &dlse}, q_in);
    same_dtype(q_in, {&k_in, &v_in, &ek, &ev, &out_in});
    Call c(q_in, q_in.size(-2), k_in.size(-2), q_in.size(-1), v_in.size(-1), ks, st, dil, causal);
    const Tensor q = strided_input(q_in, c.rank, c.p.q_stride), k = strided_input(k_in, c.rank, c.p.k_stride),
                 v = strided_input(v_in, c.rank, c.p.v_stride);
    c.scale(scale);
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor out = out_in.contiguous(), lse = lse_in.contiguous(), dout = as(dout_in, q.scalar_type());
    if (dlse.defined()) dlse = as(dlse, lse.scalar_type());
    Tensor dek, dev;
    if (ek.defined()) {
        ek = ek.contiguous();
        ev = ev.contiguous();
        c.p.n_extra = (int)ek.size(1);
        dek = fresh(ek.sizes(), ek.scalar_type(), q);
        dev = fresh(ev.sizes(), ev.scalar_type(), q);
    }
    Tensor held;
    set_extents(c.p, extents, q, held);
    Tensor dq = fresh(q.sizes(), q.scalar_type(), q), dk = fresh(k.sizes(), k.scalar_type(), q),
           dv = fresh(v.sizes(), v.scalar_type(), q);
    const size_t ws_bytes = std::max<size_t>(natten_workspace_bytes(&c.p, NATTEN_OP_FUSED_BWD), 256);
    Tensor ws = fresh({(int64_t)ws_bytes}, at::kByte, q);
    poll_status(q);
    check(natten_fused_bwd(&c.p, ptr(q), ptr(k), ptr(v), ptr(ek), ptr(ev), ptr(out), ptr(lse), ptr(dout), ptr(dlse),
                           out_ptr(dq), out_ptr(dk), out_ptr(dv), out_ptr(dek), out_ptr(dev), out_ptr(ws), ws_bytes,
                           stream_of(q)),
          "natten_fused_bwd");
    if (!dek.defined()) {
        dek = fresh({0}, q.scalar_type(), q);
        dev = fresh({0}, q.scalar_type(), q);
    }
    return {dq, dk, dv, dek, dev};
}

Tensor qk_cuda(const Tensor& q_in, const Tensor& k_in, IntArrayRef ks, IntArrayRef dil, IntArrayRef st, Bools causal,
               std::optional<double> scale)
{
    require_cuda({&q_in, &k_in}, q_in);
    same_dtype(q_in, {&k_in});
    Call c(q_in, q_in.size(-2), k_in.size(-2), q_in.size(-1), q_in.size(-1), ks, st, dil, causal);
    const Tensor q = strided_input(q_in, c.rank, c.p.q_stride), k = strided_input(k_in, c.rank, c.p.k_stride);
    std::copy(c.p.k_stride, c.p.k_stride + 3, c.p.v_stride);
    if (scale) c.scale(*scale);
    const c10::cuda::CUDAGuard guard(q.device());
    Tensor logits = fresh(c.out_shape(c.p.heads_q, c.slots()), q.scalar_type(), q);
    poll_status(q);
    check(natten_qk_fwd(&c.p, ptr(q), ptr(k), out_ptr(logits), stream_of(q)), "natten_qk_fwd");
    return logits;
}

std::tuple<Tensor, Tensor> qk_bwd_cuda(const Tensor& dlogits_in, const Tensor& q_in, const Tensor& k_in, IntArrayRef ks,
                                       IntArrayRef dil, IntArrayRef st, Bools causal, std::optional<double> scale)
{
    require_cuda({&q_in, &k_in, &dlogits_in}, q_in);
    same_dtype(q_in, {&k_in});
    Call c(q_in, q_in.size(-2), k_in.size(-2), q_in.size(-1), q_in.size(-1), ks, st, dil, causal);
    const Tensor q = strided_input(q_in, c.rank, c.p.q_stride), k = strided_input(k_in, c.rank, c.p.k_stride);
    std::copy(c.p.k_stride, c.p.k_stride + 3, c.p.v_stride);
    if (scale) c.scale(*scale);
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor dlogits = as(dlogits_in, q.scalar_type());
    Tensor dq = fresh(q.sizes(), q.scalar_type(), q), dk = fresh(k.sizes(), k.scalar_type(), q);
    poll_status(q);
    check(natten_qk_bwd(&c.p, ptr(q), ptr(k), ptr(dlogits), out_ptr(dq), out_ptr(dk), stream_of(q)), "natten_qk_bwd");
    return {dq, dk};
}

struct Unit {                                // unit stride, no causal axis: what the bias operators cover
    std::vector<int64_t> ones;
    Bools no;
    explicit Unit(size_t rank) : ones(rank, 1) { for (size_t i = 0; i < rank; ++i) no.push_back(false); }
};

Tensor qk_rpb_cuda(const Tensor& q_in, const Tensor& k_in, const Tensor& rpb_in, IntArrayRef ks, IntArrayRef dil,
                   std::optional<double> scale)
{
    require_cuda({&q_in, &k_in, &rpb_in}, q_in);
    same_dtype(q_in, {&k_in});
    const Unit u(ks.size());
    Call c(q_in, q_in.size(-2), k_in.size(-2), q_in.size(-1), q_in.size(-1), ks, u.ones, dil, u.no);
    const Tensor q = strided_input(q_in, c.rank, c.p.q_stride), k = strided_input(k_in, c.rank, c.p.k_stride);
    std::copy(c.p.k_stride, c.p.k_stride + 3, c.p.v_stride);
    if (scale) c.scale(*scale);
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor rpb = as(rpb_in, q.scalar_type());
    Tensor logits = fresh(c.out_shape(c.p.heads_q, c.slots()), q.scalar_type(), q);
    poll_status(q);
    check(natten_qk_rpb_fwd(&c.p, ptr(q), ptr(k), ptr(rpb), out_ptr(logits), stream_of(q)), "natten_qk_rpb_fwd");
    return logits;
}

std::tuple<Tensor, Tensor, Tensor> qk_rpb_bwd_cuda(const Tensor& dlogits_in, const Tensor& q_in, const Tensor& k_in,
                                                   IntArrayRef rpb_shape, IntArrayRef ks, IntArrayRef dil,
                                                   std::optional<double> scale)
{
    require_cuda({&q_in, &k_in, &dlogits_in}, q_in);
    same_dtype(q_in, {&k_in});
    const Unit u(ks.size());
    Call c(q_in, q_in.size(-2), k_in.size(-2), q_in.size(-1), q_in.size(-1), ks, u.ones, dil, u.no);
    const Tensor q = strided_input(q_in, c.rank, c.p.q_stride), k = strided_input(k_in, c.rank, c.p.k_stride);
    std::copy(c.p.k_stride, c.p.k_stride + 3, c.p.v_stride);
    if (scale) c.scale(*scale);
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor dlogits = as(dlogits_in, q.scalar_type());
    Tensor dq = fresh(q.sizes(), q.scalar_type(), q), dk = fresh(k.sizes(), k.scalar_type(), q),
           drpb = fresh(rpb_shape, q.scalar_type(), q);
    poll_status(q);
    check(natten_qk_rpb_bwd(&c.p, ptr(q), ptr(k), ptr(dlogits), out_ptr(dq), out_ptr(dk), out_ptr(drpb), stream_of(q)),
          "natten_qk_rpb_bwd");
    return {dq, dk, drpb};
}

Tensor av_cuda(const Tensor& attn_in, const Tensor& v_in, IntArrayRef ks, IntArrayRef dil, IntArrayRef st, Bools causal)
{
    require_cuda({&v_in, &attn_in}, v_in);
    Call c(v_in, attn_in.size(-2), v_in.size(-2), v_in.size(-1), v_in.size(-1), ks, st, dil, causal);
    const Tensor v = strided_input(v_in, c.rank, c.p.v_stride);
    std::copy(c.p.v_stride, c.p.v_stride + 3, c.p.q_stride);
    std::copy(c.p.v_stride, c.p.v_stride + 3, c.p.k_stride);
    const c10::cuda::CUDAGuard guard(v.device());
    const Tensor attn = as(attn_in, v.scalar_type());
    c.shape = attn.sizes().vec();
    c.shape.back() = v.size(-1);
    Tensor out = fresh(c.shape, v.scalar_type(), v);
    poll_status(v);
    check(natten_av_fwd(&c.p, ptr(attn), ptr(v), out_ptr(out), stream_of(v)), "natten_av_fwd");
    return out;
}

std::tuple<Tensor, Tensor> av_bwd_cuda(const Tensor& dout_in, const Tensor& attn_in, const Tensor& v_in, IntArrayRef ks,
                                       IntArrayRef dil, IntArrayRef st, Bools causal)
{
    require_cuda({&v_in, &attn_in, &dout_in}, v_in);
    Call c(v_in, attn_in.size(-2), v_in.size(-2), v_in.size(-1), v_in.size(-1), ks, st, dil, causal);
    const Tensor v = strided_input(v_in, c.rank, c.p.v_stride);
    std::copy(c.p.v_stride, c.p.v_stride + 3, c.p.q_stride);
    std::copy(c.p.v_stride, c.p.v_stride + 3, c.p.k_stride);
    const c10::cuda::CUDAGuard guard(v.device());
    const Tensor attn = as(attn_in, v.scalar_type()), dout = as(dout_in, v.scalar_type());
    Tensor dattn = fresh(attn.sizes(), v.scalar_type(), v), dv = fresh(v.sizes(), v.scalar_type(), v);
    poll_status(v);
    check(natten_av_bwd(&c.p, ptr(attn), ptr(v), ptr(dout), out_ptr(dattn), out_ptr(dv), stream_of(v)), "natten_av_bwd");
    return {dattn, dv};
}

// ----------------------------------------------------------------------------- dispatcher handles
template <typename Sig> auto handle(const char* name)
{
    return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}
std::tuple<Tensor, Tensor> call_fused(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& ek, const OptTensor& ev,
                                      const OptTensor& extents, IntArrayRef ks, IntArrayRef st, IntArrayRef dil, Bools causal,
                                      double scale)
{
    static const auto op = handle<decltype(fused_cuda)>("natten_b200::na_fused");
    return op.call(q, k, v, ek, ev, extents, ks, st, dil, std::move(causal), scale);
}
Tensor call_qk(const Tensor& q, const Tensor& k, IntArrayRef ks, IntArrayRef dil, IntArrayRef st, Bools causal,
               std::optional<double> scale)
{
    static const auto op = handle<decltype(qk_cuda)>("natten_b200::na_qk");
    return op.call(q, k, ks, dil, st, std::move(causal), scale);
}
Tensor call_av(const Tensor& attn, const Tensor& v, IntArrayRef ks, IntArrayRef dil, IntArrayRef st, Bools causal)
{
    static const auto op = handle<decltype(av_cuda)>("natten_b200::na_av");
    return op.call(attn, v, ks, dil, st, std::move(causal));
}
Tensor call_qk_rpb(const Tensor& q, const Tensor& k, const Tensor& rpb, IntArrayRef ks, IntArrayRef dil, std::optional<double> scale)
{
    static const auto op = handle<decltype(qk_rpb_cuda)>("natten_b200::na_qk_rpb");
    return op.call(q, k, rpb, ks, dil, scale);
}

// ----------------------------------------------------------------------------- autograd
// Kernel geometry in one saved integer list: [lists..., causal flags], each list `rank` long.
std::vector<int64_t> pack(std::initializer_list<IntArrayRef> lists, const Bools& causal)
{
    std::vector<int64_t> g;
    g.reserve(12);
    for (const IntArrayRef& l : lists) g.insert(g.end(), l.begin(), l.end());
    for (size_t i = 0; i < causal.size(); ++i) g.push_back(causal[i] ? 1 : 0);
    return g;
}
struct Unpacked {
    std::vector<int64_t> g;
    size_t rank;
    Unpacked(const AutogradContext* ctx, size_t lists, bool causal = true)
        : g(ctx->saved_data.at("g").toIntVector()), rank(g.size() / (lists + (causal ? 1 : 0))) {}
    IntArrayRef list(size_t i) const { return IntArrayRef(g.data() + i * rank, rank); }
    Bools flags(size_t i) const
    {
        Bools b;
        b.reserve(rank);
        for (size_t a = 0; a < rank; ++a) b.push_back(g[i * rank + a] != 0);
        return b;
    }
};
std::optional<double> saved_scale(const AutogradContext* ctx)
{
    const c10::IValue& s = ctx->saved_data.at("s");
    return s.isNone() ? std::nullopt : std::optional<double>(s.toDouble());
}
bool wants_grad(std::initializer_list<const Tensor*> tensors)
{
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : tensors)
        if (t && t->defined() && t->requires_grad()) return true;
    return false;
}
const Tensor* opt_ptr(const OptTensor& t) { return t ? &*t : nullptr; }

struct FusedFn : public torch::autograd::Function<FusedFn> {
    static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& ek,
                                 const OptTensor& ev, const OptTensor& extents, IntArrayRef ks, IntArrayRef st,
                                 IntArrayRef dil, const Bools& causal, double scale)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        auto [out, lse] = call_fused(q, k, v, ek, ev, extents, ks, st, dil, causal, scale);
        ctx->saved_data["g"] = pack({ks, st, dil}, causal);
        ctx->saved_data["s"] = scale;
        ctx->save_for_backward({q, k, v, ek.value_or(Tensor()), ev.value_or(Tensor()), extents.value_or(Tensor()), out, lse});
        ctx->set_materialize_grads(false);       // no zero-filled gradient for an unused log-sum-exp
        return {out, lse};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        static const auto op = handle<decltype(fused_bwd_cuda)>("natten_b200::na_fused_bwd");
        const auto s = ctx->get_saved_variables();
        const Unpacked u(ctx, 3);
        auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
        const Tensor dout = grads[0].defined() ? grads[0] : at::zeros_like(s[6]);
        auto [dq, dk, dv, dek, dev] = op.call(s[0], s[1], s[2], opt(s[3]), opt(s[4]), opt(s[5]), s[6], s[7], dout,
                                              opt(grads[1]), u.list(0), u.list(1), u.list(2), u.flags(3), *saved_scale(ctx));
        const bool extra = s[3].defined();
        return {dq, dk, dv, extra ? dek : Tensor(), extra ? dev : Tensor(), {}, {}, {}, {}, {}, {}};
    }
};
std::tuple<Tensor, Tensor> fused_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& ek,
                                          const OptTensor& ev, const OptTensor& extents, IntArrayRef ks, IntArrayRef st,
                                          IntArrayRef dil, Bools causal, double scale)
{
    if (!wants_grad({&q, &k, &v, opt_ptr(ek), opt_ptr(ev)})) {
        at::AutoDispatchBelowADInplaceOrView below;
        return call_fused(q, k, v, ek, ev, extents, ks, st, dil, std::move(causal), scale);
    }
    const variable_list r = FusedFn::apply(q, k, v, ek, ev, extents, ks, st, dil, causal, scale);
    return {r[0], r[1]};
}

struct QkFn : public torch::autograd::Function<QkFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, IntArrayRef ks, IntArrayRef dil,
                          IntArrayRef st, const Bools& causal, std::optional<double> scale)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Tensor logits = call_qk(q, k, ks, dil, st, causal, scale);
        ctx->saved_data["g"] = pack({ks, dil, st}, causal);
        ctx->saved_data["s"] = scale;
        ctx->save_for_backward({q, k});
        return logits;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        static const auto op = handle<decltype(qk_bwd_cuda)>("natten_b200::na_qk_bwd");
        const auto s = ctx->get_saved_variables();
        const Unpacked u(ctx, 3);
        auto [dq, dk] = op.call(grads[0], s[0], s[1], u.list(0), u.list(1), u.list(2), u.flags(3), saved_scale(ctx));
        return {dq, dk, {}, {}, {}, {}, {}};
    }
};
Tensor qk_autograd(const Tensor& q, const Tensor& k, IntArrayRef ks, IntArrayRef dil, IntArrayRef st, Bools causal,
                   std::optional<double> scale)
{
    if (!wants_grad({&q, &k})) {
        at::AutoDispatchBelowADInplaceOrView below;
        return call_qk(q, k, ks, dil, st, std::move(causal), scale);
    }
    return QkFn::apply(q, k, ks, dil, st, causal, scale);
}

struct AvFn : public torch::autograd::Function<AvFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& attn, const Tensor& v, IntArrayRef ks, IntArrayRef dil,
                          IntArrayRef st, const Bools& causal)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Tensor out = call_av(attn, v, ks, dil, st, causal);
        ctx->saved_data["g"] = pack({ks, dil, st}, causal);
        ctx->save_for_backward({attn, v});
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        static const auto op = handle<decltype(av_bwd_cuda)>("natten_b200::na_av_bwd");
        const auto s = ctx->get_saved_variables();
        const Unpacked u(ctx, 3);
        auto [dattn, dv] = op.call(grads[0], s[0], s[1], u.list(0), u.list(1), u.list(2), u.flags(3));
        return {dattn.to(s[0].scalar_type()), dv, {}, {}, {}, {}};
    }
};
Tensor av_autograd(const Tensor& attn, const Tensor& v, IntArrayRef ks, IntArrayRef dil, IntArrayRef st, Bools causal)
{
    if (!wants_grad({&attn, &v})) {
        at::AutoDispatchBelowADInplaceOrView below;
        return call_av(attn, v, ks, dil, st, std::move(causal));
    }
    return AvFn::apply(attn, v, ks, dil, st, causal);
}

struct QkRpbFn : public torch::autograd::Function<QkRpbFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& rpb, IntArrayRef ks,
                          IntArrayRef dil, std::optional<double> scale)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        Tensor logits = call_qk_rpb(q, k, rpb, ks, dil, scale);
        ctx->saved_data["g"] = pack({ks, dil}, Bools());
        ctx->saved_data["s"] = scale;
        ctx->saved_data["t"] = rpb.scalar_type();
        ctx->save_for_backward({q, k});
        return logits;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        static const auto op = handle<decltype(qk_rpb_bwd_cuda)>("natten_b200::na_qk_rpb_bwd");
        const auto s = ctx->get_saved_variables();
        const Unpacked u(ctx, 2, /*causal=*/false);
        std::vector<int64_t> shape{s[0].size(-2)};
        for (int64_t k : u.list(0)) shape.push_back(2 * k - 1);
        auto [dq, dk, drpb] = op.call(grads[0], s[0], s[1], shape, u.list(0), u.list(1), saved_scale(ctx));
        return {dq, dk, drpb.to(ctx->saved_data.at("t").toScalarType()), {}, {}, {}};
    }
};
Tensor qk_rpb_autograd(const Tensor& q, const Tensor& k, const Tensor& rpb, IntArrayRef ks, IntArrayRef dil,
                       std::optional<double> scale)
{
    if (!wants_grad({&q, &k, &rpb})) {
        at::AutoDispatchBelowADInplaceOrView below;
        return call_qk_rpb(q, k, rpb, ks, dil, scale);
    }
    return QkRpbFn::apply(q, k, rpb, ks, dil, scale);
}

// The whole module, projections included, as one node of the autograd graph.  Built from the separate operators a training
// pass of it took 330 us on the host (projections, views, unbind and their thirty backward operators) where the kernels
// take 165: most of the host time goes into dispatching and into the engine's bookkeeping between small operators.  The
// products are the ones the separate operators run; the three gradients of the packed projection are put side by side by
// one copy instead of three.
struct Projected { Tensor y1, y2, q, k, v; };
Projected project(const Tensor& x, const Tensor& w1, const OptTensor& b1, const Tensor& w2, const OptTensor& b2, int64_t heads, int64_t kv)
{
    auto split = [&](const Tensor& y, int64_t n, int64_t h) {
        std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 1);
        if (n > 1) shape.push_back(n);
        shape.push_back(h);
        shape.push_back(y.size(-1) / (n * h));
        return y.view(shape);
    };
    Projected r;
    r.y1 = at::linear(x, w1, b1);
    if (w2.defined()) {
        r.y2 = at::linear(x, w2, b2);
        r.q = split(r.y1, 1, heads);
        const Tensor t = split(r.y2, 2, kv);
        r.k = t.select(-3, 0);
        r.v = t.select(-3, 1);
    } else {
        const Tensor t = split(r.y1, 3, heads);
        r.q = t.select(-3, 0);
        r.k = t.select(-3, 1);
        r.v = t.select(-3, 2);
    }
    return r;
}
Tensor rows_of(const Tensor& t) { return t.reshape({-1, t.size(-1)}); }
Tensor joined_heads(const Tensor& out)
{
    std::vector<int64_t> shape(out.sizes().begin(), out.sizes().end() - 1);
    shape.back() *= out.size(-1);
    return out.reshape(shape);
}

struct ModuleFn : public torch::autograd::Function<ModuleFn> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const OptTensor& b1, const OptTensor& w2,
                          const OptTensor& b2, const Tensor& wp, const OptTensor& bp, int64_t heads, int64_t kv, IntArrayRef ks, IntArrayRef st,
                          IntArrayRef dil, const Bools& causal, double scale)
    {
        at::AutoDispatchBelowADInplaceOrView below;
        const Projected r = project(x, w1, b1, w2.value_or(Tensor()), b2, heads, kv);
        auto [out, lse] = call_fused(r.q, r.k, r.v, std::nullopt, std::nullopt, std::nullopt, ks, st, dil, causal, scale);
        ctx->saved_data["g"] = pack({ks, st, dil}, causal);
        ctx->saved_data["s"] = scale;
        ctx->saved_data["m"] = (int64_t)((b1 ? 4 : 0) | (w2 ? 8 : 0) | (b2 ? 16 : 0) | (bp ? 64 : 0) | 35);     // arguments that are there
        ctx->save_for_backward({x, w1, w2.value_or(Tensor()), wp, r.q, r.k, r.v, out, lse});
        ctx->saved_data["h"] = std::vector<int64_t>{heads, kv, version_of(b1), version_of(b2)};
        ctx->saved_data["b1"] = b1;              // for differentiable() alone: a plain backward does not look at them, and
        ctx->saved_data["b2"] = b2;              // does not mind if they have been written to since
        return at::linear(joined_heads(out), wp, bp);
    }
    static int64_t version_of(const OptTensor& t) { return t && !t->is_inference() ? t->_version() : 0; }
    // The gradients with a graph of their own (create_graph): from the separate operators, run again.  `stand_in` keeps the
    // arguments apart where one was computed from another (a weight shared between layers).
    static variable_list differentiable(AutogradContext* ctx, const variable_list& s, const Tensor& grad, const bool (&needs)[7])
    {
        auto stand_in = [](const Tensor& t) { return t.defined() ? t.view_as(t) : t; };
        auto bias = [&](const char* name, int64_t version) {
            const OptTensor b = ctx->saved_data.at(name).toOptional<Tensor>();
            TORCH_CHECK(version_of(b) == version, "natten_b200: a projection's bias was modified in place since the forward pass; "
                        "its gradients can't be given a graph");
            return b ? OptTensor(stand_in(*b)) : b;
        };
        const c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);     // as in the forward pass
        const auto h = ctx->saved_data.at("h").toIntVector();
        const Unpacked u(ctx, 3);
        const Tensor x = stand_in(s[0]), w1 = stand_in(s[1]), w2 = stand_in(s[2]), wp = stand_in(s[3]);
        const OptTensor b1 = bias("b1", h[2]), b2 = bias("b2", h[3]);
        const Projected r = project(x, w1, b1, w2, b2, h[0], h[1]);
        const Tensor out = std::get<0>(call_fused(r.q, r.k, r.v, std::nullopt, std::nullopt, std::nullopt, u.list(0), u.list(1),
                                                  u.list(2), u.flags(3), *saved_scale(ctx)));
        const Tensor y = at::linear(joined_heads(out), wp);
        const Tensor args[6] = {x, w1, b1.value_or(Tensor()), w2, b2.value_or(Tensor()), wp};
        variable_list wanted, result(14);
        for (int i = 0; i < 6; ++i)
            if (needs[i]) wanted.push_back(args[i]);
        if (!wanted.empty()) {
            const variable_list got = torch::autograd::grad({y}, wanted, {grad}, /*retain_graph=*/true, /*create_graph=*/true,
                                                            /*allow_unused=*/true);
            for (int i = 0, n = 0; i < 6; ++i)
                if (needs[i]) result[i] = got[n++];
        }
        if (needs[6]) result[6] = rows_of(grad).sum(0);
        return result;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads)
    {
        static const auto op = handle<decltype(fused_bwd_cuda)>("natten_b200::na_fused_bwd");
        const auto s = ctx->get_saved_variables();
        const Tensor &x = s[0], &w1 = s[1], &w2 = s[2], &wp = s[3];
        const Unpacked u(ctx, 3);
        variable_list r(14);
        const int64_t there = ctx->saved_data.at("m").toInt();
        bool needs[7];
        for (int i = 0, edge = 0; i < 7; ++i) needs[i] = ((there >> i) & 1) && ctx->needs_input_grad(edge++);
        if (at::GradMode::is_enabled()) return differentiable(ctx, s, grads[0], needs);
        const Tensor g = rows_of(grads[0]), x2 = rows_of(x);
        if (needs[6]) r[6] = g.sum(0);           // (a kernel first: it makes the device's context current on the engine's thread)
        if (needs[5]) r[5] = g.t().mm(rows_of(joined_heads(s[7])));
        bool inner = false;
        for (int i = 0; i < 5; ++i) inner = inner || needs[i];
        if (!inner) return r;
        auto [dq, dk, dv, dek, dev] = op.call(s[4], s[5], s[6], std::nullopt, std::nullopt, std::nullopt, s[7], s[8],
                                              g.mm(wp).view(s[7].sizes()), std::nullopt, u.list(0), u.list(1), u.list(2), u.flags(3),
                                              *saved_scale(ctx));
        auto flat = [&](const Tensor& t) { return t.reshape({x2.size(0), -1}); };
        const Tensor d1 = w2.defined() ? flat(dq) : at::cat({flat(dq), flat(dk), flat(dv)}, 1);
        const Tensor d2 = w2.defined() ? at::cat({flat(dk), flat(dv)}, 1) : Tensor();
        if (needs[0]) r[0] = (w2.defined() ? at::addmm(d1.mm(w1), d2, w2) : d1.mm(w1)).view(x.sizes());
        if (needs[1]) r[1] = d1.t().mm(x2);
        if (needs[2]) r[2] = d1.sum(0);
        if (needs[3]) r[3] = d2.t().mm(x2);
        if (needs[4]) r[4] = d2.sum(0);
        return r;
    }
};

// ----------------------------------------------------------------------------- argument parsing for functional.py
// An integer per axis from an int or a tuple / list of ints; every value positive (bools are not integers here).
bool ints(PyObject* o, int rank, int64_t (&out)[3])
{
    auto one = [](PyObject* x, int64_t& v) {
        if (!PyLong_CheckExact(x)) return false;
        int overflow = 0;
        v = PyLong_AsLongLongAndOverflow(x, &overflow);
        return overflow == 0 && v > 0 && v < (1 << 30);
    };
    if (PyLong_CheckExact(o)) {
        if (!one(o, out[0])) return false;
        for (int a = 1; a < rank; ++a) out[a] = out[0];
        return true;
    }
    const bool tuple = PyTuple_CheckExact(o);
    if (!tuple && !PyList_CheckExact(o)) return false;
    if ((tuple ? PyTuple_GET_SIZE(o) : PyList_GET_SIZE(o)) != rank) return false;
    for (int a = 0; a < rank; ++a)
        if (!one(tuple ? PyTuple_GET_ITEM(o, a) : PyList_GET_ITEM(o, a), out[a])) return false;
    return true;
}
// The same for flags: a bool or a tuple / list of bools.
bool flags(PyObject* o, int rank, Bools& out, bool& any)
{
    out.reserve(rank);
    any = false;
    const bool tuple = PyTuple_CheckExact(o), list = PyList_CheckExact(o);
    if ((tuple && PyTuple_GET_SIZE(o) != rank) || (list && PyList_GET_SIZE(o) != rank)) return false;
    for (int a = 0; a < rank; ++a) {
        PyObject* x = tuple ? PyTuple_GET_ITEM(o, a) : list ? PyList_GET_ITEM(o, a) : o;
        if (x != Py_True && x != Py_False) return false;
        out.push_back(x == Py_True);
        any = any || x == Py_True;
    }
    return true;
}
// None or a number
bool number(PyObject* o, std::optional<double>& out)
{
    if (o == Py_None) { out = std::nullopt; return true; }
    if (PyFloat_CheckExact(o)) { out = PyFloat_AS_DOUBLE(o); return true; }
    if (PyLong_CheckExact(o)) {
        out = PyLong_AsDouble(o);
        if (PyErr_Occurred()) { PyErr_Clear(); return false; }
        return true;
    }
    return false;
}
// A plain tensor (or parameter) of `dims` dimensions.
const Tensor* tensor(PyObject* o, int dims)
{
    if (!THPVariable_CheckExact(o)) return nullptr;
    const Tensor& t = THPVariable_Unpack(o);
    return t.dim() == dims && !t.unsafeGetTensorImpl()->has_symbolic_sizes_strides() ? &t : nullptr;
}

PyObject* not_handled() { Py_RETURN_NOTIMPLEMENTED; }
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }

bool spatial_equal(const Tensor& a, const Tensor& b, int rank)
{
    for (int i = 0; i <= rank; ++i)
        if (a.size(i) != b.size(i)) return false;
    return true;
}
bool kernel_fits(const Tensor& t, int rank, const int64_t (&ks)[3], const int64_t (&dil)[3])
{
    for (int a = 0; a < rank; ++a)
        if (ks[a] * dil[a] > t.size(1 + a)) return false;
    return true;
}
// query / key / value of a fused call agree (grouped heads allowed); additional tokens, when given, fit them
bool fused_shapes(const Tensor& q, const Tensor& k, const Tensor& v, int rank)
{
    return spatial_equal(q, k, rank) && spatial_equal(q, v, rank) && q.size(-1) == k.size(-1) && k.size(-2) == v.size(-2) &&
           k.size(-2) > 0 && q.size(-2) % k.size(-2) == 0;
}
bool extra_tokens(PyObject* ko, PyObject* vo, const Tensor& q, const Tensor& k, OptTensor& ek, OptTensor& ev)
{
    if (ko == Py_None && vo == Py_None) return true;
    const Tensor *a = tensor(ko, 4), *b = tensor(vo, 4);
    if (!a || !b || a->sizes() != b->sizes() || a->size(0) != q.size(0) || a->size(-1) != q.size(-1) || a->size(-2) != k.size(-2))
        return false;
    ek = *a;
    ev = *b;
    return true;
}

struct NoGil {                               // kernels are launched (and may block on a full queue) without the GIL
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

// na(rank, query, key, value, kernel_size, stride, dilation, is_causal, scale, return_lse, extra_k, extra_v)
PyObject* py_na(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    const int rank = n == 12 ? (int)PyLong_AsLong(args[0]) : 0;
    if (rank < 1 || rank > 3 || at::impl::torch_function_mode_enabled()) return not_handled();
    const Tensor *q = tensor(args[1], rank + 3), *k = tensor(args[2], rank + 3), *v = tensor(args[3], rank + 3);
    if (!q || !k || !v || !fused_shapes(*q, *k, *v, rank)) return not_handled();
    int64_t ks[3], st[3], dil[3];
    Bools causal;
    bool any_causal = false;
    std::optional<double> scale;
    OptTensor ek, ev;
    if (!ints(args[4], rank, ks) || !ints(args[5], rank, st) || !ints(args[6], rank, dil) ||
        !flags(args[7], rank, causal, any_causal) || !number(args[8], scale) || (args[9] != Py_True && args[9] != Py_False) ||
        !extra_tokens(args[10], args[11], *q, *k, ek, ev) || !kernel_fits(*q, rank, ks, dil))
        return not_handled();
    bool covers = !any_causal;               // the window is the whole input: global attention, not ours
    for (int a = 0; a < rank; ++a) {
        if (st[a] > ks[a]) return not_handled();
        covers = covers && ks[a] >= q->size(1 + a) && st[a] == 1;
    }
    if (covers) return not_handled();
    if (!scale) scale = std::pow((double)q->size(-1), -0.5);
    const bool want_lse = args[9] == Py_True;
    Tensor out, lse;
    {
        NoGil nogil;
        std::tie(out, lse) = call_fused(*q, *k, *v, ek, ev, std::nullopt, {ks, (size_t)rank}, {st, (size_t)rank},
                                        {dil, (size_t)rank}, std::move(causal), *scale);
        if (want_lse && !ek) lse = lse.to(q->scalar_type());
    }
    if (!want_lse) return wrap(std::move(out));
    PyObject* both = PyTuple_New(2);
    if (!both) return nullptr;
    PyTuple_SET_ITEM(both, 0, wrap(std::move(out)));
    PyTuple_SET_ITEM(both, 1, wrap(std::move(lse)));
    return both;
    END_HANDLE_TH_ERRORS
}

// na_module(rank, x, w1, b1 | None, w2 | None, b2 | None, proj weight, proj bias | None, heads, kv heads, kernel_size, stride,
// dilation, is_causal, scale): the packed (w1) or separate (w1, w2) projections, attention and the output projection
PyObject* py_module(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    const int rank = n == 15 ? (int)PyLong_AsLong(args[0]) : 0;
    if (rank < 1 || rank > 3 || at::impl::torch_function_mode_enabled() || c10::impl::dispatch_mode_enabled() ||
        at::autocast::is_autocast_enabled(at::kCUDA) || PyLong_AsLong(args[8]) < 1 || PyLong_AsLong(args[9]) < 1)
        return not_handled();
    // anything that wraps tensors or records them (functorch, functionalisation, subclasses) takes the separate operators
    const c10::DispatchKeySet plain({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                                     c10::DispatchKey::AutocastCUDA});
    const c10::DispatchKeySet modes({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode,
                                     c10::DispatchKey::Functionalize, c10::DispatchKey::Python});
    if (!(c10::impl::tls_local_dispatch_key_set().included_ & modes).empty()) return not_handled();
    const int64_t heads = PyLong_AsLong(args[8]), kv = PyLong_AsLong(args[9]);
    Tensor t[7];
    for (int i = 0; i < 7; ++i) {
        if (args[1 + i] == Py_None) continue;
        const Tensor* p = tensor(args[1 + i], i == 0 ? rank + 2 : i % 2 ? 2 : 1);
        if (!p || (p->key_set() - plain).highestFunctionalityKey() != c10::DispatchKey::Undefined || p->layout() != at::kStrided || p->numel() == 0) return not_handled();
        t[i] = *p;
        if (!t[0].defined() || p->scalar_type() != t[0].scalar_type() || p->device() != t[0].device()) return not_handled();
    }
    const Tensor &x = t[0], &w1 = t[1], &b1 = t[2], &w2 = t[3], &b2 = t[4], &wp = t[5], &bp = t[6];
    if (!x.defined() || !w1.defined() || !wp.defined() || !x.is_cuda() || (b2.defined() && !w2.defined())) return not_handled();
    const int64_t C = x.size(-1), D = C / heads;
    if (D * heads != C || heads % kv != 0 || w1.size(0) != (w2.defined() ? C : 3 * C) || w1.size(1) != C || wp.size(0) != C ||
        wp.size(1) != C || (w2.defined() ? w2.size(0) != 2 * kv * D || w2.size(1) != C : kv != heads) ||
        (b1.defined() && b1.size(0) != w1.size(0)) || (b2.defined() && b2.size(0) != w2.size(0)) || (bp.defined() && bp.size(0) != C))
        return not_handled();
    int64_t ks[3], st[3], dil[3];
    Bools causal;
    bool any_causal = false;
    std::optional<double> scale;
    if (!ints(args[10], rank, ks) || !ints(args[11], rank, st) || !ints(args[12], rank, dil) || !flags(args[13], rank, causal, any_causal) ||
        !number(args[14], scale) || !scale || !kernel_fits(x, rank, ks, dil))
        return not_handled();
    bool covers = !any_causal;               // global attention, not ours
    for (int a = 0; a < rank; ++a) {
        if (st[a] > ks[a]) return not_handled();
        covers = covers && ks[a] >= x.size(1 + a) && st[a] == 1;
    }
    if (covers) return not_handled();
    Tensor out;
    {
        NoGil nogil;
        const IntArrayRef ksr(ks, rank), str(st, rank), dilr(dil, rank);
        auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
        if (wants_grad({&x, &w1, &b1, &w2, &b2, &wp, &bp})) {
            out = ModuleFn::apply(x, w1, opt(b1), opt(w2), opt(b2), wp, opt(bp), heads, kv, ksr, str, dilr, causal, *scale);
        } else {
            at::AutoDispatchBelowADInplaceOrView below;
            const Projected r = project(x, w1, opt(b1), w2, opt(b2), heads, kv);
            out = at::linear(joined_heads(std::get<0>(call_fused(r.q, r.k, r.v, std::nullopt, std::nullopt, std::nullopt, ksr, str, dilr,
                                                                 std::move(causal), *scale))), wp, opt(bp));
        }
    }
    return wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// na_varlen(rank, query, key, value, sizes, kernel_size, dilation, scale, extra_k, extra_v)
PyObject* py_varlen(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    const int rank = n == 10 ? (int)PyLong_AsLong(args[0]) : 0;
    if (rank < 1 || rank > 3 || at::impl::torch_function_mode_enabled()) return not_handled();
    const Tensor *q = tensor(args[1], rank + 3), *k = tensor(args[2], rank + 3), *v = tensor(args[3], rank + 3);
    const Tensor* sizes = tensor(args[4], rank == 1 ? 1 : 2);
    if (!q || !k || !v || !sizes || !fused_shapes(*q, *k, *v, rank) || k->size(-1) != v->size(-1) || !q->is_cuda())
        return not_handled();
    int64_t ks[3], dil[3];
    std::optional<double> scale;
    OptTensor ek, ev;
    if (!ints(args[5], rank, ks) || !ints(args[6], rank, dil) || !number(args[7], scale) ||
        !extra_tokens(args[8], args[9], *q, *k, ek, ev))
        return not_handled();
    if (sizes->size(0) != q->size(0) || (rank > 1 && sizes->size(1) != rank) ||
        (sizes->scalar_type() != at::kInt && sizes->scalar_type() != at::kLong) || sizes->layout() != at::kStrided)
        return not_handled();
    if (!scale) scale = std::pow((double)q->size(-1), -0.5);
    Tensor out;
    bool in_range = true;
    {
        NoGil nogil;
        // the one host read that the range check needs (the kernels use the tensor where it is)
        const Tensor host = sizes->detach().cpu().to(at::kLong).contiguous();
        const int64_t* x = host.const_data_ptr<int64_t>();
        for (int64_t i = 0; i < host.numel(); ++i) {
            const int a = (int)(i % rank);
            in_range = in_range && x[i] >= ks[a] && x[i] <= q->size(1 + a);
        }
        if (in_range) {
            Bools no;
            for (int a = 0; a < rank; ++a) no.push_back(false);
            const int64_t one[3] = {1, 1, 1};
            const Tensor table = sizes->reshape({sizes->size(0), rank}).to(at::kInt);
            out = std::get<0>(call_fused(*q, *k, *v, ek, ev, table, {ks, (size_t)rank}, {one, (size_t)rank},
                                         {dil, (size_t)rank}, std::move(no), *scale));
        }
    }
    return in_range ? wrap(std::move(out)) : not_handled();
    END_HANDLE_TH_ERRORS
}

// na_qk(rank, query, key, rpb | None, kernel_size, dilation, stride, is_causal, scale)
PyObject* py_qk(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    const int rank = n == 9 ? (int)PyLong_AsLong(args[0]) : 0;
    if (rank < 1 || rank > 3 || at::impl::torch_function_mode_enabled()) return not_handled();
    const Tensor *q = tensor(args[1], rank + 3), *k = tensor(args[2], rank + 3);
    if (!q || !k || q->sizes() != k->sizes()) return not_handled();
    int64_t ks[3], st[3], dil[3];
    Bools causal;
    bool any_causal = false;
    std::optional<double> scale;
    if (!ints(args[4], rank, ks) || !ints(args[5], rank, dil) || !ints(args[6], rank, st) ||
        !flags(args[7], rank, causal, any_causal) || !number(args[8], scale) || !kernel_fits(*q, rank, ks, dil))
        return not_handled();
    const Tensor* rpb = nullptr;
    if (args[3] != Py_None) {
        rpb = tensor(args[3], rank + 1);
        if (!rpb || rpb->size(0) != q->size(-2)) return not_handled();
        for (int a = 0; a < rank; ++a)
            if (ks[a] % 2 == 0 || rpb->size(1 + a) != 2 * ks[a] - 1 || st[a] != 1) return not_handled();
    }
    Tensor logits;
    {
        NoGil nogil;
        const IntArrayRef ksr(ks, rank), dilr(dil, rank), str(st, rank);
        logits = rpb ? call_qk_rpb(*q, *k, *rpb, ksr, dilr, scale) : call_qk(*q, *k, ksr, dilr, str, std::move(causal), scale);
    }
    return wrap(std::move(logits));
    END_HANDLE_TH_ERRORS
}

// na_av(rank, attn, value, kernel_size, dilation, stride, is_causal)
PyObject* py_av(PyObject*, PyObject* const* args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    const int rank = n == 7 ? (int)PyLong_AsLong(args[0]) : 0;
    if (rank < 1 || rank > 3 || at::impl::torch_function_mode_enabled()) return not_handled();
    const Tensor *attn = tensor(args[1], rank + 3), *v = tensor(args[2], rank + 3);
    if (!attn || !v) return not_handled();
    int64_t ks[3], st[3], dil[3], slots = 1;
    Bools causal;
    bool any_causal = false;
    if (!ints(args[3], rank, ks) || !ints(args[4], rank, dil) || !ints(args[5], rank, st) ||
        !flags(args[6], rank, causal, any_causal) || !kernel_fits(*v, rank, ks, dil))
        return not_handled();
    if (attn->size(0) != v->size(0) || attn->size(-2) != v->size(-2)) return not_handled();
    for (int a = 0; a < rank; ++a) {
        slots *= ks[a];
        if (attn->size(1 + a) != (v->size(1 + a) + st[a] - 1) / st[a]) return not_handled();
    }
    if (attn->size(-1) != slots) return not_handled();
    Tensor out;
    {
        NoGil nogil;
        out = call_av(*attn, *v, {ks, (size_t)rank}, {dil, (size_t)rank}, {st, (size_t)rank}, std::move(causal));
    }
    return wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

PyObject* py_set_flags(PyObject*, PyObject* o)
{
    g_flags.store((int)PyLong_AsLong(o));
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"na", (PyCFunction)(void (*)(void))py_na, METH_FASTCALL, nullptr},
    {"na_module", (PyCFunction)(void (*)(void))py_module, METH_FASTCALL, nullptr},
    {"na_varlen", (PyCFunction)(void (*)(void))py_varlen, METH_FASTCALL, nullptr},
    {"na_qk", (PyCFunction)(void (*)(void))py_qk, METH_FASTCALL, nullptr},
    {"na_av", (PyCFunction)(void (*)(void))py_av, METH_FASTCALL, nullptr},
    {"set_flags", py_set_flags, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Native host path of natten_mps_b200.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

} // namespace

TORCH_LIBRARY_IMPL(natten_b200, CUDA, m)
{
    m.impl("na_fused", fused_cuda);
    m.impl("na_fused_bwd", fused_bwd_cuda);
    m.impl("na_qk", qk_cuda);
    m.impl("na_qk_bwd", qk_bwd_cuda);
    m.impl("na_qk_rpb", qk_rpb_cuda);
    m.impl("na_qk_rpb_bwd", qk_rpb_bwd_cuda);
    m.impl("na_av", av_cuda);
    m.impl("na_av_bwd", av_bwd_cuda);
}

TORCH_LIBRARY_IMPL(natten_b200, Autograd, m)
{
    m.impl("na_fused", fused_autograd);
    m.impl("na_qk", qk_autograd);
    m.impl("na_qk_rpb", qk_rpb_autograd);
    m.impl("na_av", av_autograd);
}

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
