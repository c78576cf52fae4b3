// The six libtorch_tp_jit::jit_* operators registered from C++ on top of the C ABI of liboeq_b200.so.
//
// Counterpart of the reference's op layer (extension/torch_core.hpp:274-644: op bodies, check_tensor, output
// allocation, TORCH_LIBRARY schemas at :626-644; extension/libtorch_tp_jit.cpp:17-108: stream and registration glue).
// Same schemas, same argument checks with the same messages, outputs allocated with the inputs' options, launches on
// the current CUDA stream of the tensors' device.  Being registered in C++, the operators exist in any process that
// loads this library (an AOTInductor package run from C++ included) and a call costs a few microseconds of host time;
// the autograd chain forward -> backward -> double backward is registered here too, so that recording and running a
// gradient never enters Python.  The Python module openequivariance_b200/_torch/ops.py adds the fake and autocast
// registrations and the third order on top and carries an equivalent Python implementation for installations where this
// file was not built.
//
// Built by openequivariance_b200/build_native.py (g++ against the installed torch; links liboeq_b200.so).

#include <ATen/ATen.h>
#include <c10/core/Event.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <memory>
#include <mutex>
#include <string>
#include <tuple>
#include <unordered_map>
#include <vector>

#include "../../include/oeq_b200.h"

namespace {

[[noreturn]] void refuse(const std::string& message) { TORCH_CHECK(false, message); }

struct Problem {
    std::string desc;
    oeqb_kernel_prop prop;
};

std::mutex g_mutex;
std::unordered_map<int64_t, std::shared_ptr<Problem>> g_problems;

// key -> descriptor text and properties; the tensor -> bytes copy happens once per key
std::shared_ptr<Problem> problem(const at::Tensor& json_bytes, int64_t key) {
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto it = g_problems.find(key);
        if (it != g_problems.end()) return it->second;
    }
    at::Tensor host = json_bytes.detach().to(at::kCPU).contiguous();
    if (host.scalar_type() != at::kByte) refuse("json_bytes must be a uint8 tensor");
    auto p = std::make_shared<Problem>();
    p->desc.assign(reinterpret_cast<const char*>(host.data_ptr<uint8_t>()), (size_t)host.numel());
    const int rc = oeqb_query(p->desc.data(), p->desc.size(), key, &p->prop);
    if (rc != 0) refuse("oeqb_query failed (code " + std::to_string(rc) + "): " + oeqb_last_error());
    std::lock_guard<std::mutex> lock(g_mutex);
    g_problems[key] = p;
    return p;
}

at::ScalarType torch_dtype(int e) {
    switch (e) {
        case 1: return at::kFloat;
        case 2: return at::kDouble;
        case 3: return at::kInt;
        case 4: return at::kLong;
        default: return at::kByte;
    }
}

// Messages are put together with std::string and std::to_string only: no iostream formatting in this library.
// (A shape message formatted through std::ostringstream crashed inside the stream's integer insertion on GPU machines,
// in processes where the CUDA driver's libraries were loaded, and only there; the cause was not found.)
std::string shape_str(const std::vector<int64_t>& s) {
    std::string o = "[";
    for (size_t i = 0; i < s.size(); ++i) o += (i ? ", " : "") + std::to_string(s[i]);
    return o + "]";
}



// Messages as in check_tensor (torch_core.hpp:109-134); -1 in `shape` accepts any extent.
void check(const at::Tensor& t, const std::vector<int64_t>& shape, at::ScalarType dt, const char* name) {
    const std::vector<int64_t> got = t.sizes().vec();
    bool ok = got.size() == shape.size();
    for (size_t i = 0; ok && i < shape.size(); ++i)
        if (shape[i] >= 0 && got[i] != shape[i]) ok = false;
    if (!ok) refuse(std::string("Shape mismatch for tensor '") + name + "'. Expected: " + shape_str(shape) + ". Got: " + shape_str(got));
#ifndef OEQB_TEST_ANY_DEVICE   // (a test build runs the argument checks on CPU tensors)
    if (!t.is_cuda()) refuse(std::string("Tensor '") + name + "' is not on the GPU.");
#endif
    if (t.scalar_type() != dt)
        refuse(std::string("Dtype mismatch for tensor '") + name + "'. Expected: " + c10::toString(dt) + ". Got: " +
               c10::toString(t.scalar_type()));
}

int64_t first_dim(const at::Tensor& t, const char* name) {
    if (t.dim() < 1)
        refuse(std::string("Shape mismatch for tensor '") + name + "'. Expected a leading batch dimension. Got: " +
               shape_str(t.sizes().vec()));
    return t.size(0);
}

const void* ptr(const at::Tensor& t) { return t.numel() > 0 ? t.data_ptr() : nullptr; }
void* mptr(at::Tensor& t) { return t.numel() > 0 ? t.data_ptr() : nullptr; }

void* current_stream(const at::Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

void done(int rc, const char* what) {
    if (rc != 0) refuse(std::string(what) + " failed (code " + std::to_string(rc) + "): " + oeqb_last_error());
}

int64_t tp_checks(const Problem& p, const at::Tensor& x, const at::Tensor& y, const at::Tensor& W) {
    const at::ScalarType dt = torch_dtype(p.prop.irrep_dtype);
    const int64_t B = first_dim(x, "L1_in");
    check(x, {B, p.prop.L1_dim}, dt, "L1_in");
    check(y, {B, p.prop.L2_dim}, dt, "L2_in");
    if (p.prop.shared_weights) check(W, {p.prop.weight_numel}, torch_dtype(p.prop.weight_dtype), "W");
    else check(W, {B, p.prop.weight_numel}, torch_dtype(p.prop.weight_dtype), "W");
    return B;
}

at::Tensor jit_tp_forward(const at::Tensor& json_bytes, int64_t hash, const at::Tensor& L1_in, const at::Tensor& L2_in,
                          const at::Tensor& W, int64_t L3_dim) {
    (void)L3_dim;
    auto p = problem(json_bytes, hash);
    const int64_t B = tp_checks(*p, L1_in, L2_in, W);
    at::Tensor x = L1_in.contiguous(), y = L2_in.contiguous(), w = W.contiguous();
    at::Tensor out = at::empty({B, p->prop.L3_dim}, x.options());
    c10::cuda::CUDAGuard guard(x.device());
    done(oeqb_tp_forward(p->desc.data(), p->desc.size(), hash, B, ptr(x), ptr(y), ptr(w), mptr(out), current_stream(x)),
         "jit_tp_forward");
    return out;
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> jit_tp_backward(const at::Tensor& json_bytes, int64_t hash,
                                                               const at::Tensor& L1_in, const at::Tensor& L2_in,
                                                               const at::Tensor& W, const at::Tensor& L3_grad) {
    auto p = problem(json_bytes, hash);
    const int64_t B = tp_checks(*p, L1_in, L2_in, W);
    check(L3_grad, {B, p->prop.L3_dim}, torch_dtype(p->prop.irrep_dtype), "L3_grad");
    at::Tensor x = L1_in.contiguous(), y = L2_in.contiguous(), w = W.contiguous(), g = L3_grad.contiguous();
    at::Tensor dx = at::empty_like(x), dy = at::empty_like(y), dw = at::empty_like(w);
    c10::cuda::CUDAGuard guard(x.device());
    done(oeqb_tp_backward(p->desc.data(), p->desc.size(), hash, B, ptr(x), ptr(y), ptr(w), ptr(g), mptr(dx), mptr(dy), mptr(dw),
                          current_stream(x)),
         "jit_tp_backward");
    return {dx, dy, dw};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> jit_tp_double_backward(
    const at::Tensor& json_bytes, int64_t hash, const at::Tensor& L1_in, const at::Tensor& L2_in, const at::Tensor& W,
    const at::Tensor& L3_grad, const at::Tensor& L1_dgrad, const at::Tensor& L2_dgrad, const at::Tensor& W_dgrad) {
    auto p = problem(json_bytes, hash);
    const int64_t B = tp_checks(*p, L1_in, L2_in, W);
    const at::ScalarType dt = torch_dtype(p->prop.irrep_dtype);
    check(L3_grad, {B, p->prop.L3_dim}, dt, "L3_grad");
    check(L1_dgrad, {B, p->prop.L1_dim}, dt, "L1_dgrad");
    check(L2_dgrad, {B, p->prop.L2_dim}, dt, "L2_dgrad");
    check(W_dgrad, W.sizes().vec(), W.scalar_type(), "W_dgrad");
    at::Tensor x = L1_in.contiguous(), y = L2_in.contiguous(), w = W.contiguous(), g = L3_grad.contiguous();
    at::Tensor x2 = L1_dgrad.contiguous(), y2 = L2_dgrad.contiguous(), w2 = W_dgrad.contiguous();
    at::Tensor dx = at::empty_like(x), dy = at::empty_like(y), dw = at::empty_like(w), dg = at::empty_like(g);
    c10::cuda::CUDAGuard guard(x.device());
    done(oeqb_tp_double_backward(p->desc.data(), p->desc.size(), hash, B, ptr(x), ptr(y), ptr(w), ptr(g), ptr(x2), ptr(y2),
                                 ptr(w2), mptr(dx), mptr(dy), mptr(dw), mptr(dg), current_stream(x)),
         "jit_tp_double_backward");
    return {dx, dy, dw, dg};
}

struct ConvSizes { int64_t N, E; };

ConvSizes conv_checks(const Problem& p, const at::Tensor& x, const at::Tensor& y, const at::Tensor& W, const at::Tensor& rows,
                      const at::Tensor& cols, const at::Tensor& workspace, const at::Tensor& perm) {
    const at::ScalarType dt = torch_dtype(p.prop.irrep_dtype), it = torch_dtype(p.prop.idx_dtype);
    const int64_t N = first_dim(x, "L1_in"), E = first_dim(rows, "rows");
    check(x, {N, p.prop.L1_dim}, dt, "L1_in");
    check(y, {E, p.prop.L2_dim}, dt, "L2_in");
    if (p.prop.shared_weights) check(W, {p.prop.weight_numel}, torch_dtype(p.prop.weight_dtype), "W");
    else check(W, {E, p.prop.weight_numel}, torch_dtype(p.prop.weight_dtype), "W");
    check(rows, {E}, it, "rows");
    check(cols, {E}, it, "cols");
    if (p.prop.deterministic) check(perm, {E}, it, "transpose_perm");
    check(workspace, {-1}, at::kByte, "workspace");
    return {N, E};
}

// the caller's workspace when it is large enough, else a fresh one from torch's caching allocator
at::Tensor scratch(const Problem& p, int64_t key, int direction, ConvSizes s, const at::Tensor& workspace) {
    const int64_t need = oeqb_conv_workspace_bytes(p.desc.data(), p.desc.size(), key, direction, s.N, s.E);
    if (need < 0) refuse("oeqb_conv_workspace_bytes failed (code " + std::to_string(-need) + "): " + oeqb_last_error());
    if (workspace.numel() >= need) return workspace;
    return at::empty({need}, workspace.options());
}

at::Tensor jit_conv_forward(const at::Tensor& json_bytes, int64_t hash, const at::Tensor& L1_in, const at::Tensor& L2_in,
                            const at::Tensor& W, int64_t L3_dim, const at::Tensor& rows, const at::Tensor& cols,
                            const at::Tensor& workspace, const at::Tensor& transpose_perm) {
    (void)L3_dim;
    auto p = problem(json_bytes, hash);
    const ConvSizes s = conv_checks(*p, L1_in, L2_in, W, rows, cols, workspace, transpose_perm);
    at::Tensor x = L1_in.contiguous(), y = L2_in.contiguous(), w = W.contiguous();
    at::Tensor r = rows.contiguous(), c = cols.contiguous(), pm = transpose_perm.contiguous();
    at::Tensor out = at::empty({s.N, p->prop.L3_dim}, x.options());
    c10::cuda::CUDAGuard guard(x.device());
    at::Tensor ws = scratch(*p, hash, 0, s, workspace);
    done(oeqb_conv_forward(p->desc.data(), p->desc.size(), hash, s.N, s.E, ptr(x), ptr(y), ptr(w), mptr(out), ptr(r), ptr(c),
                           p->prop.deterministic ? ptr(pm) : nullptr, mptr(ws), ws.numel(), current_stream(x)),
         "jit_conv_forward");
    return out;
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> jit_conv_backward(const at::Tensor& json_bytes, int64_t hash,
                                                                 const at::Tensor& L1_in, const at::Tensor& L2_in,
                                                                 const at::Tensor& W, const at::Tensor& L3_grad,
                                                                 const at::Tensor& rows, const at::Tensor& cols,
                                                                 const at::Tensor& workspace, const at::Tensor& transpose_perm) {
    auto p = problem(json_bytes, hash);
    const ConvSizes s = conv_checks(*p, L1_in, L2_in, W, rows, cols, workspace, transpose_perm);
    check(L3_grad, {s.N, p->prop.L3_dim}, torch_dtype(p->prop.irrep_dtype), "L3_grad");
    at::Tensor x = L1_in.contiguous(), y = L2_in.contiguous(), w = W.contiguous(), g = L3_grad.contiguous();
    at::Tensor r = rows.contiguous(), c = cols.contiguous(), pm = transpose_perm.contiguous();
    at::Tensor dx = at::empty_like(x), dy = at::empty_like(y), dw = at::empty_like(w);
    c10::cuda::CUDAGuard guard(x.device());
    at::Tensor ws = scratch(*p, hash, 1, s, workspace);
    done(oeqb_conv_backward(p->desc.data(), p->desc.size(), hash, s.N, s.E, ptr(x), ptr(y), ptr(w), ptr(g), mptr(dx), mptr(dy),
                            mptr(dw), ptr(r), ptr(c), p->prop.deterministic ? ptr(pm) : nullptr, mptr(ws), ws.numel(),
                            current_stream(x)),
         "jit_conv_backward");
    return {dx, dy, dw};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> jit_conv_double_backward(
    const at::Tensor& json_bytes, int64_t hash, const at::Tensor& L1_in, const at::Tensor& L2_in, const at::Tensor& W,
    const at::Tensor& L3_grad, const at::Tensor& L1_dgrad, const at::Tensor& L2_dgrad, const at::Tensor& W_dgrad,
    const at::Tensor& rows, const at::Tensor& cols, const at::Tensor& workspace, const at::Tensor& transpose_perm) {
    auto p = problem(json_bytes, hash);
    const ConvSizes s = conv_checks(*p, L1_in, L2_in, W, rows, cols, workspace, transpose_perm);
    const at::ScalarType dt = torch_dtype(p->prop.irrep_dtype);
    check(L3_grad, {s.N, p->prop.L3_dim}, dt, "L3_grad");
    check(L1_dgrad, {s.N, p->prop.L1_dim}, dt, "L1_dgrad");
    check(L2_dgrad, {s.E, p->prop.L2_dim}, dt, "L2_dgrad");
    check(W_dgrad, W.sizes().vec(), W.scalar_type(), "W_dgrad");
    at::Tensor x = L1_in.contiguous(), y = L2_in.contiguous(), w = W.contiguous(), g = L3_grad.contiguous();
    at::Tensor x2 = L1_dgrad.contiguous(), y2 = L2_dgrad.contiguous(), w2 = W_dgrad.contiguous();
    at::Tensor r = rows.contiguous(), c = cols.contiguous(), pm = transpose_perm.contiguous();
    at::Tensor dx = at::empty_like(x), dy = at::empty_like(y), dw = at::empty_like(w), dg = at::empty_like(g);
    c10::cuda::CUDAGuard guard(x.device());
    at::Tensor ws = scratch(*p, hash, 2, s, workspace);
    done(oeqb_conv_double_backward(p->desc.data(), p->desc.size(), hash, s.N, s.E, ptr(x), ptr(y), ptr(w), ptr(g), ptr(x2),
                                   ptr(y2), ptr(w2), mptr(dx), mptr(dy), mptr(dw), mptr(dg), ptr(r), ptr(c),
                                   p->prop.deterministic ? ptr(pm) : nullptr, mptr(ws), ws.numel(), current_stream(x)),
         "jit_conv_double_backward");
    return {dx, dy, dw, dg};
}

// ---- autograd chain: forward -> backward -> double backward ----------------------------------------------------
// An op's autograd kernel costs host time on every call, and small calls are nothing but host time: the same chain
// registered from Python took 125 us for forward + gradients of a 1,000-item product whose two kernels run for 6 us.
// A kernel with nothing to record redispatches below autograd at once.
//
// The index tensors, the workspace and the descriptor travel in saved_data (they are not differentiable); the operands
// that the next order differentiates are saved variables.
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
typedef std::tuple<at::Tensor, at::Tensor, at::Tensor> Three;
typedef std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> Four;

typedef at::Tensor TpFwdSig(const at::Tensor&, int64_t, const at::Tensor&, const at::Tensor&, const at::Tensor&, int64_t);
typedef Three TpBwdSig(const at::Tensor&, int64_t, const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&);
typedef Four TpDblSig(const at::Tensor&, int64_t, const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&,
                      const at::Tensor&, const at::Tensor&, const at::Tensor&);
typedef at::Tensor ConvFwdSig(const at::Tensor&, int64_t, const at::Tensor&, const at::Tensor&, const at::Tensor&, int64_t,
                              const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&);
typedef Three ConvBwdSig(const at::Tensor&, int64_t, const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&,
                         const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&);
typedef Four ConvDblSig(const at::Tensor&, int64_t, const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&,
                        const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&,
                        const at::Tensor&, const at::Tensor&);
const c10::TypedOperatorHandle<TpFwdSig>& tp_fwd_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("libtorch_tp_jit::jit_tp_forward", "").typed<TpFwdSig>();
    return op;
}
const c10::TypedOperatorHandle<TpBwdSig>& tp_bwd_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("libtorch_tp_jit::jit_tp_backward", "").typed<TpBwdSig>();
    return op;
}
const c10::TypedOperatorHandle<TpDblSig>& tp_dbl_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("libtorch_tp_jit::jit_tp_double_backward", "").typed<TpDblSig>();
    return op;
}
const c10::TypedOperatorHandle<ConvFwdSig>& conv_fwd_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("libtorch_tp_jit::jit_conv_forward", "").typed<ConvFwdSig>();
    return op;
}
const c10::TypedOperatorHandle<ConvBwdSig>& conv_bwd_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("libtorch_tp_jit::jit_conv_backward", "").typed<ConvBwdSig>();
    return op;
}
const c10::TypedOperatorHandle<ConvDblSig>& conv_dbl_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("libtorch_tp_jit::jit_conv_double_backward", "").typed<ConvDblSig>();
    return op;
}

template <class... Ts>
bool records(const Ts&... ts) { return at::GradMode::is_enabled() && (ts.requires_grad() || ...); }

void keep(AutogradContext* ctx, const at::Tensor& json, int64_t hash) {
    ctx->saved_data["json"] = json;
    ctx->saved_data["hash"] = hash;
}
void keep(AutogradContext* ctx, const at::Tensor& json, int64_t hash, const at::Tensor& rows, const at::Tensor& cols,
          const at::Tensor& workspace, const at::Tensor& perm) {
    keep(ctx, json, hash);
    ctx->saved_data["rows"] = rows;
    ctx->saved_data["cols"] = cols;
    ctx->saved_data["workspace"] = workspace;
    ctx->saved_data["perm"] = perm;
}
at::Tensor kept(AutogradContext* ctx, const char* name) { return ctx->saved_data[name].toTensor(); }
int64_t kept_hash(AutogradContext* ctx) { return ctx->saved_data["hash"].toInt(); }

struct TpForward : torch::autograd::Function<TpForward> {
    static at::Tensor forward(AutogradContext* ctx, const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y,
                              const at::Tensor& W, int64_t L3_dim) {
        keep(ctx, json, hash);
        ctx->save_for_backward({x, y, W});
        at::AutoDispatchBelowADInplaceOrView below;
        return tp_fwd_op().call(json, hash, x, y, W, L3_dim);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
        const variable_list v = ctx->get_saved_variables();
        auto [dx, dy, dw] = tp_bwd_op().call(kept(ctx, "json"), kept_hash(ctx), v[0], v[1], v[2], grads[0]);
        return {at::Tensor(), at::Tensor(), dx, dy, dw, at::Tensor()};
    }
};

struct TpBackward : torch::autograd::Function<TpBackward> {
    static variable_list forward(AutogradContext* ctx, const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y,
                                 const at::Tensor& W, const at::Tensor& g) {
        keep(ctx, json, hash);
        ctx->save_for_backward({x, y, W, g});
        at::AutoDispatchBelowADInplaceOrView below;
        auto [dx, dy, dw] = tp_bwd_op().call(json, hash, x, y, W, g);
        return {dx, dy, dw};
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& grads) {   // undefined cotangents arrive as zeros
        const variable_list v = ctx->get_saved_variables();
        auto [dx, dy, dw, dg] = tp_dbl_op().call(kept(ctx, "json"), kept_hash(ctx), v[0], v[1], v[2], v[3], grads[0], grads[1], grads[2]);
        return {at::Tensor(), at::Tensor(), dx, dy, dw, dg};
    }
};

struct ConvForward : torch::autograd::Function<ConvForward> {
    static at::Tensor forward(AutogradContext* ctx, const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y,
                              const at::Tensor& W, int64_t L3_dim, const at::Tensor& rows, const at::Tensor& cols,
                              const at::Tensor& workspace, const at::Tensor& perm) {
        keep(ctx, json, hash, rows, cols, workspace, perm);
        ctx->save_for_backward({x, y, W});
        at::AutoDispatchBelowADInplaceOrView below;
        return conv_fwd_op().call(json, hash, x, y, W, L3_dim, rows, cols, workspace, perm);
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
        const variable_list v = ctx->get_saved_variables();
        auto [dx, dy, dw] = conv_bwd_op().call(kept(ctx, "json"), kept_hash(ctx), v[0], v[1], v[2], grads[0], kept(ctx, "rows"),
                                               kept(ctx, "cols"), kept(ctx, "workspace"), kept(ctx, "perm"));
        return {at::Tensor(), at::Tensor(), dx, dy, dw, at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
    }
};

struct ConvBackward : torch::autograd::Function<ConvBackward> {
    static variable_list forward(AutogradContext* ctx, const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y,
                                 const at::Tensor& W, const at::Tensor& g, const at::Tensor& rows, const at::Tensor& cols,
                                 const at::Tensor& workspace, const at::Tensor& perm) {
        keep(ctx, json, hash, rows, cols, workspace, perm);
        ctx->save_for_backward({x, y, W, g});
        at::AutoDispatchBelowADInplaceOrView below;
        auto [dx, dy, dw] = conv_bwd_op().call(json, hash, x, y, W, g, rows, cols, workspace, perm);
        return {dx, dy, dw};
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
        const variable_list v = ctx->get_saved_variables();
        auto [dx, dy, dw, dg] = conv_dbl_op().call(kept(ctx, "json"), kept_hash(ctx), v[0], v[1], v[2], v[3], grads[0], grads[1],
                                                   grads[2], kept(ctx, "rows"), kept(ctx, "cols"), kept(ctx, "workspace"),
                                                   kept(ctx, "perm"));
        return {at::Tensor(), at::Tensor(), dx, dy, dw, dg, at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
    }
};

at::Tensor autograd_tp_forward(const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y, const at::Tensor& W,
                               int64_t L3_dim) {
    if (records(x, y, W)) return TpForward::apply(json, hash, x, y, W, L3_dim);
    at::AutoDispatchBelowADInplaceOrView below;
    return tp_fwd_op().call(json, hash, x, y, W, L3_dim);
}

Three autograd_tp_backward(const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y, const at::Tensor& W,
                           const at::Tensor& g) {
    if (records(x, y, W, g)) {
        const variable_list out = TpBackward::apply(json, hash, x, y, W, g);
        return {out[0], out[1], out[2]};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    return tp_bwd_op().call(json, hash, x, y, W, g);
}

at::Tensor autograd_conv_forward(const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y, const at::Tensor& W,
                                 int64_t L3_dim, const at::Tensor& rows, const at::Tensor& cols, const at::Tensor& workspace,
                                 const at::Tensor& perm) {
    if (records(x, y, W)) return ConvForward::apply(json, hash, x, y, W, L3_dim, rows, cols, workspace, perm);
    at::AutoDispatchBelowADInplaceOrView below;
    return conv_fwd_op().call(json, hash, x, y, W, L3_dim, rows, cols, workspace, perm);
}

Three autograd_conv_backward(const at::Tensor& json, int64_t hash, const at::Tensor& x, const at::Tensor& y, const at::Tensor& W,
                             const at::Tensor& g, const at::Tensor& rows, const at::Tensor& cols, const at::Tensor& workspace,
                             const at::Tensor& perm) {
    if (records(x, y, W, g)) {
        const variable_list out = ConvBackward::apply(json, hash, x, y, W, g, rows, cols, workspace, perm);
        return {out[0], out[1], out[2]};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    return conv_bwd_op().call(json, hash, x, y, W, g, rows, cols, workspace, perm);
}

// ---- symmetric contraction ---------------------------------------------------------------------------------------
// `terms`, `meta` (CPU), `place` and `U_rows` describe the contraction's tensors U (made by _torch/symmetric_contraction.py);
// `keys` holds the element of each node; `weights` one tensor [elements, columns, channels] per (irrep, order).  The dense
// tensors `U` are used by gradients that are differentiated again, which Python composes, and to see that they still are what
// the description was made from (`U_made`).  Besides the result the forward returns what the backward takes again, the nodes by
// element and the polynomials' coefficients, and on the host whether U has changed (1: the result is then to be thrown away) or the
// call was captured (2: the description has to live as long as the graph may be replayed).
int symcon_dtype(const at::Tensor& x) {
    if (x.scalar_type() == at::kFloat) return 1;
    if (x.scalar_type() == at::kDouble) return 2;
    refuse("symmetric_contraction: x must be float32 or float64");
}
// The description's host part: 32-bit integers on the host, as many as its own counts say.
const int32_t* host_part(const at::Tensor& t, const char* name, int64_t least) {
    if (!t.is_cpu() || t.scalar_type() != at::kInt || !t.is_contiguous() || t.numel() < least)
        refuse(std::string("symmetric_contraction: '") + name + "' must be a contiguous int32 tensor on the host with " + std::to_string(least) + " entries");
    return t.data_ptr<int32_t>();
}
void same_device(const at::Tensor& x, std::initializer_list<at::TensorList> lists) {
    for (const at::TensorList& list : lists)
        for (const at::Tensor& t : list)
            if (t.device() != x.device())
                refuse("symmetric_contraction: expected all tensors to be on the same device, but found " + x.device().str() + " and " + t.device().str());
}
struct Plan {
    const int32_t *meta, *terms;
    int n_meta;
};
Plan checked_plan(const at::Tensor& terms, const at::Tensor& place, const at::Tensor& U_rows, const at::Tensor& meta, const at::Tensor& x) {
    const int32_t* m = host_part(meta, "meta", 9);
    host_part(meta, "meta", 9 + 2 * (int64_t)std::max(m[3], 0) + 2 * (int64_t)std::max(m[4], 0));
    int64_t values = 0;
    for (int s = 0; s < m[4]; ++s) values += (int64_t)m[9 + 2 * s] * m[10 + 2 * s];
    check(place, {m[6]}, at::kInt, "place");
    check(U_rows, {values}, x.scalar_type(), "U");
    if (!place.is_contiguous() || !U_rows.is_contiguous()) refuse("symmetric_contraction: the plan does not fit the operands");
    return {m, host_part(terms, "terms", 4 * (int64_t)m[6]), (int)meta.numel()};
}
// A plan's tensors were allocated on the stream of the call that made it, and the plan may be dropped by another thread while this
// call's kernels run: their memory is not given away before those have finished.
void used_here(const at::Tensor& t) {
    if (t.is_cuda()) t.record_stream(c10::cuda::getCurrentCUDAStream(t.device().index()).unwrap());
}
at::Tensor aligned(const at::Tensor& t) {   // rows are read 16 bytes at a time
    at::Tensor c = t.contiguous();
    return ((uintptr_t)c.data_ptr() & 15u) ? c.clone() : c;
}

Four symcon_forward(const at::Tensor& x_in, const at::Tensor& keys_in, at::TensorList weights, at::TensorList U, at::TensorList U_made,
                    const at::Tensor& terms_in, const at::Tensor& place, const at::Tensor& U_rows, const at::Tensor& meta_in, int64_t out_dim,
                    bool check_keys) {
    const auto [meta, terms, n_meta] = checked_plan(terms_in, place, U_rows, meta_in, x_in);
    const int dt = symcon_dtype(x_in);
    const int64_t N = first_dim(x_in, "x");
    check(x_in, {N, meta[1], meta[2]}, x_in.scalar_type(), "x");
    check(keys_in, {N}, at::kLong, "keys");
    same_device(x_in, {{keys_in, place, U_rows}, weights, U, U_made});
    if (out_dim != meta[5] || (int64_t)weights.size() != meta[4]) refuse("symmetric_contraction: the plan does not fit the operands");
    c10::cuda::CUDAGuard guard(x_in.device());
    at::Tensor x = aligned(x_in), keys = keys_in.contiguous();
    std::vector<at::Tensor> held;
    std::vector<const void*> w, now, made;
    std::vector<int64_t> size;
    for (size_t s = 0; s < weights.size(); ++s) {
        check(weights[s], {meta[0], meta[9 + 2 * s], meta[1]}, x.scalar_type(), "weights");
        held.push_back(weights[s].contiguous());
        w.push_back(held.back().data_ptr());
    }
    if (U.size() != U_made.size()) refuse("symmetric_contraction: the plan does not fit the operands");
    for (size_t s = 0; s < U.size(); ++s) {
        check(U[s], U_made[s].sizes().vec(), U_made[s].scalar_type(), "U");
        held.push_back(U[s].contiguous());
        now.push_back(ptr(held.back()));
        made.push_back(ptr(U_made[s]));
        size.push_back((int64_t)U_made[s].nbytes());
    }
    const int64_t bytes = oeqb_symcon_bytes(dt, meta, n_meta, 0, N);
    if (bytes < 0) done((int)-bytes, "symmetric_contraction");
    at::Tensor group = at::empty({oeqb_symcon_group_ints(N, meta[0])}, x.options().dtype(at::kInt));
    at::Tensor out = at::empty({N, out_dim}, x.options()), coef = at::empty({bytes}, x.options().dtype(at::kByte));
    for (const at::Tensor& t : U_made) used_here(t);
    used_here(place);
    used_here(U_rows);
    // The comparison goes first and is waited for last: the work proper is under way meanwhile.  So does the grouping, which checks
    // the elements, where these are the caller's (`check_keys`).  A captured call does not wait, and has its replays report what
    // they find.
    const bool captured = oeqb_stream_is_capturing(current_stream(x)) == 1;
    at::Tensor changed = at::empty({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(!captured));
    *changed.data_ptr<int32_t>() = captured ? 2 : 0;
    done(oeqb_symcon_compare((int)U.size(), now.data(), made.data(), size.data(), captured ? nullptr : changed.data_ptr<int32_t>(),
                             current_stream(x)),
         "symmetric_contraction");
    struct Compared {   // `changed` is the device's until then, whatever happens below
        c10::Event event{c10::DeviceType::CUDA};
        bool waits = false;
        void record(const at::Tensor& t) { event.record(c10::cuda::getCurrentCUDAStream(t.device().index())); waits = true; }
        void wait() { if (waits) event.synchronize(); waits = false; }
        ~Compared() { try { wait(); } catch (...) {} }
    } compared;
    if (!captured) compared.record(x);
    done(oeqb_symcon_group(N, meta[0], keys.data_ptr<int64_t>(), group.data_ptr<int32_t>(), current_stream(x)), "symmetric_contraction");
    if (!captured && check_keys) compared.record(x);
    done(oeqb_symcon_forward(dt, meta, n_meta, terms, place.data_ptr<int32_t>(), U_rows.data_ptr(), N,
                             nullptr, ptr(x), w.data(), group.data_ptr<int32_t>(), coef.data_ptr(), mptr(out),
                             current_stream(x)),
         "symmetric_contraction");
    compared.wait();
    if (!captured && check_keys) done(oeqb_check_status(), "symmetric_contraction");
    return {out, group, coef, changed};
}

std::tuple<at::Tensor, std::vector<at::Tensor>> symcon_backward(const at::Tensor& cot_in, const at::Tensor& x_in, const at::Tensor& keys,
                                                               const at::Tensor& group, const at::Tensor& coef, at::TensorList weights,
                                                               at::TensorList U, const at::Tensor& terms_in, const at::Tensor& place,
                                                               const at::Tensor& U_rows, const at::Tensor& meta_in) {
    (void)U; (void)keys;
    const auto [meta, terms, n_meta] = checked_plan(terms_in, place, U_rows, meta_in, x_in);
    const int dt = symcon_dtype(x_in);
    const int64_t N = first_dim(x_in, "x");
    check(x_in, {N, meta[1], meta[2]}, x_in.scalar_type(), "x");
    check(cot_in, {N, meta[5]}, x_in.scalar_type(), "grad");
    const int64_t bytes = oeqb_symcon_bytes(dt, meta, n_meta, 0, N);
    if (bytes < 0) done((int)-bytes, "symmetric_contraction_backward");
    check(group, {oeqb_symcon_group_ints(N, meta[0])}, at::kInt, "group");
    check(coef, {bytes}, at::kByte, "coef");
    same_device(x_in, {{cot_in, group, coef, place, U_rows}, weights});
    if ((int64_t)weights.size() != meta[4]) refuse("symmetric_contraction: the plan does not fit the operands");
    for (size_t s = 0; s < weights.size(); ++s) check(weights[s], {meta[0], meta[9 + 2 * s], meta[1]}, x_in.scalar_type(), "weights");
    c10::cuda::CUDAGuard guard(x_in.device());
    at::Tensor x = aligned(x_in), cot = cot_in.contiguous(), dx = at::empty_like(x);
    // one allocation for the weight gradients and the scratch
    const int64_t elt = (int64_t)x.element_size(), part = oeqb_symcon_bytes(dt, meta, n_meta, 1, N);
    if (part < 0) done((int)-part, "symmetric_contraction_backward");
    std::vector<at::Tensor> dw;
    std::vector<void*> dwp;
    for (const at::Tensor& t : weights) {
        dw.push_back(at::empty(t.sizes(), x.options()));
        dwp.push_back(dw.back().data_ptr());
    }
    at::Tensor ws = at::empty({part / elt + 1}, x.options());
    used_here(place);
    used_here(U_rows);
    done(oeqb_symcon_backward(dt, meta, n_meta, terms, place.data_ptr<int32_t>(), U_rows.data_ptr(), N,
                              group.data_ptr<int32_t>(), coef.data_ptr(), ptr(x), ptr(cot), ws.data_ptr(), mptr(dx), dwp.data(),
                              current_stream(x)),
         "symmetric_contraction_backward");
    return {dx, dw};
}

typedef Four SymFwdSig(const at::Tensor&, const at::Tensor&, at::TensorList, at::TensorList, at::TensorList, const at::Tensor&,
                       const at::Tensor&, const at::Tensor&, const at::Tensor&, int64_t, bool);
typedef std::tuple<at::Tensor, std::vector<at::Tensor>> SymBwdSig(const at::Tensor&, const at::Tensor&, const at::Tensor&, const at::Tensor&,
                                                                  const at::Tensor&, at::TensorList, at::TensorList, const at::Tensor&,
                                                                  const at::Tensor&, const at::Tensor&, const at::Tensor&);
const c10::TypedOperatorHandle<SymFwdSig>& sym_fwd_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("oeq_b200::symmetric_contraction", "").typed<SymFwdSig>();
    return op;
}
const c10::TypedOperatorHandle<SymBwdSig>& sym_bwd_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("oeq_b200::symmetric_contraction_backward", "").typed<SymBwdSig>();
    return op;
}

typedef at::Tensor SymComposedSig(const at::Tensor&, const at::Tensor&, at::TensorList, at::TensorList, c10::IntArrayRef, int64_t);
const c10::TypedOperatorHandle<SymComposedSig>& sym_composed_op() {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("oeq_b200::symmetric_contraction_composed", "").typed<SymComposedSig>();
    return op;
}

bool mapped(const at::Tensor& t) {   // a transform maps over it
    return t.key_set().has(c10::DispatchKey::FuncTorchBatched) || t.key_set().has(c10::DispatchKey::Batched);
}

// Gradients (of x, then of the weights; undefined where none is needed) that may be differentiated again, or that a transform maps
// over: those of the composed form, whose recorded graph the next order continues.  It is formed on aliases of the operands: the graph stays connected to
// them, so every order is right, and a gradient ends at the operand it is for even where one operand was made from another.
variable_list symcon_composed_gradients(const at::Tensor& cot, const variable_list& operands, const at::Tensor& keys, at::TensorList U,
                                        const at::Tensor& meta) {
    const bool again = at::GradMode::is_enabled();
    at::AutoGradMode recording(true);
    variable_list alias, wanted, found(operands.size());
    for (const at::Tensor& t : operands) {
        alias.push_back(again ? t.view_as(t) : t.detach().requires_grad_(t.requires_grad()));
        if (t.requires_grad()) wanted.push_back(alias.back());
    }
    const int32_t* end = meta.data_ptr<int32_t>() + meta.numel() - 1;   // orders of every irrep, then their number
    if (*end < 0 || *end >= meta.numel()) refuse("symmetric_contraction: the plan does not fit the operands");
    const std::vector<int64_t> orders(end - *end, end);
    const std::vector<at::Tensor> weights(alias.begin() + 1, alias.end());
    const at::Tensor out = sym_composed_op().call(alias[0], keys, weights, U, orders, meta.data_ptr<int32_t>()[0]);
    const variable_list got = torch::autograd::grad({out}, wanted, {cot}, c10::nullopt, again, true);
    for (size_t i = 0, j = 0; i < alias.size(); ++i)
        if (alias[i].requires_grad()) found[i] = got[j++];
    return found;
}

struct SymForward : torch::autograd::Function<SymForward> {
    static variable_list forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& keys, at::TensorList weights, at::TensorList U,
                                 at::TensorList U_made, const at::Tensor& terms, const at::Tensor& place, const at::Tensor& U_rows,
                                 const at::Tensor& meta, int64_t out_dim, bool check_keys) {
        at::AutoDispatchBelowADInplaceOrView below;
        auto [out, group, coef, changed] = sym_fwd_op().call(x, keys, weights, U, U_made, terms, place, U_rows, meta, out_dim, check_keys);
        ctx->mark_non_differentiable({group, coef, changed});
        ctx->set_materialize_grads(false);
        variable_list saved{x};
        saved.insert(saved.end(), weights.begin(), weights.end());
        ctx->save_for_backward(saved);
        ctx->saved_data["fixed"] = std::vector<at::Tensor>{keys, group, coef, terms, place, U_rows, meta};
        ctx->saved_data["U"] = U.vec();
        std::vector<int64_t> versions;
        for (const at::Tensor& u : U) versions.push_back(u.is_inference() ? 0 : (int64_t)u._version());
        ctx->saved_data["versions"] = versions;
        return {out, group, coef, changed};
    }
    static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
        const variable_list v = ctx->get_saved_variables();
        const std::vector<at::Tensor> U = ctx->saved_data["U"].toTensorVector(), fixed = ctx->saved_data["fixed"].toTensorVector();
        variable_list out(v.size() + 1);
        if (grads[0].defined() && (at::GradMode::is_enabled() || mapped(grads[0]))) {
            const std::vector<int64_t> versions = ctx->saved_data["versions"].toIntVector();
            for (size_t s = 0; s < U.size(); ++s)
                if (!U[s].is_inference() && (int64_t)U[s]._version() != versions[s])
                    refuse("one of the variables needed for gradient computation has been modified by an inplace operation: U");
            const variable_list d = symcon_composed_gradients(grads[0], v, fixed[0], U, fixed[6]);
            out[0] = d[0];
            std::copy(d.begin() + 1, d.end(), out.begin() + 2);
        } else if (grads[0].defined()) {
            const std::vector<at::Tensor> weights(v.begin() + 1, v.end());
            auto [dx, dw] = sym_bwd_op().call(grads[0], v[0], fixed[0], fixed[1], fixed[2], weights, U, fixed[3], fixed[4], fixed[5], fixed[6]);
            out[0] = dx;
            std::copy(dw.begin(), dw.end(), out.begin() + 2);
        }
        out.resize(out.size() + 2 * U.size() + 6);   // U, U_made, terms, place, U_rows, meta, out_dim, check_keys
        return out;
    }
};

Four autograd_symcon(const at::Tensor& x, const at::Tensor& keys, at::TensorList weights, at::TensorList U, at::TensorList U_made,
                     const at::Tensor& terms, const at::Tensor& place, const at::Tensor& U_rows, const at::Tensor& meta, int64_t out_dim,
                     bool check_keys) {
    bool any = records(x);
    for (const at::Tensor& w : weights) any = any || records(w);
    if (any) {
        const variable_list out = SymForward::apply(x, keys, weights, U, U_made, terms, place, U_rows, meta, out_dim, check_keys);
        return {out[0], out[1], out[2], out[3]};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    return sym_fwd_op().call(x, keys, weights, U, U_made, terms, place, U_rows, meta, out_dim, check_keys);
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(oeq_b200, m) {
    m.def("symmetric_contraction(Tensor x, Tensor keys, Tensor[] weights, Tensor[] U, Tensor[] U_made, Tensor terms, Tensor place, Tensor U_rows, Tensor meta, int out_dim, bool check_keys) -> (Tensor, Tensor, Tensor, Tensor)");
    m.def("symmetric_contraction_backward(Tensor grad, Tensor x, Tensor keys, Tensor group, Tensor coef, Tensor[] weights, Tensor[] U, Tensor terms, Tensor place, Tensor U_rows, Tensor meta) -> (Tensor, Tensor[])");
}
TORCH_LIBRARY_IMPL(oeq_b200, CUDA, m) {
    m.impl("symmetric_contraction", &symcon_forward);
    m.impl("symmetric_contraction_backward", &symcon_backward);
}
TORCH_LIBRARY_IMPL(oeq_b200, Autograd, m) { m.impl("symmetric_contraction", &autograd_symcon); }

TORCH_LIBRARY(libtorch_tp_jit, m) {
    m.def("jit_tp_forward(Tensor json_bytes, int hash, Tensor L1_in, Tensor L2_in, Tensor W, int L3_dim) -> Tensor");
    m.def("jit_tp_backward(Tensor json_bytes, int hash, Tensor L1_in, Tensor L2_in, Tensor W, Tensor L3_grad) -> (Tensor, Tensor, Tensor)");
    m.def("jit_tp_double_backward(Tensor json_bytes, int hash, Tensor L1_in, Tensor L2_in, Tensor W, Tensor L3_grad, Tensor L1_dgrad, Tensor L2_dgrad, Tensor W_dgrad) -> (Tensor, Tensor, Tensor, Tensor)");
    m.def("jit_conv_forward(Tensor json_bytes, int hash, Tensor L1_in, Tensor L2_in, Tensor W, int L3_dim, Tensor rows, Tensor cols, Tensor workspace, Tensor transpose_perm) -> Tensor");
    m.def("jit_conv_backward(Tensor json_bytes, int hash, Tensor L1_in, Tensor L2_in, Tensor W, Tensor L3_grad, Tensor rows, Tensor cols, Tensor workspace, Tensor transpose_perm) -> (Tensor, Tensor, Tensor)");
    m.def("jit_conv_double_backward(Tensor json_bytes, int hash, Tensor L1_in, Tensor L2_in, Tensor W, Tensor L3_grad, Tensor L1_dgrad, Tensor L2_dgrad, Tensor W_dgrad, Tensor rows, Tensor cols, Tensor workspace, Tensor transpose_perm) -> (Tensor, Tensor, Tensor, Tensor)");
}

TORCH_LIBRARY_IMPL(libtorch_tp_jit, CUDA, m) {
    m.impl("jit_tp_forward", &jit_tp_forward);
    m.impl("jit_tp_backward", &jit_tp_backward);
    m.impl("jit_tp_double_backward", &jit_tp_double_backward);
    m.impl("jit_conv_forward", &jit_conv_forward);
    m.impl("jit_conv_backward", &jit_conv_backward);
    m.impl("jit_conv_double_backward", &jit_conv_double_backward);
}

TORCH_LIBRARY_IMPL(libtorch_tp_jit, Autograd, m) {
    m.impl("jit_tp_forward", &autograd_tp_forward);
    m.impl("jit_tp_backward", &autograd_tp_backward);
    m.impl("jit_conv_forward", &autograd_conv_forward);
    m.impl("jit_conv_backward", &autograd_conv_backward);
}
