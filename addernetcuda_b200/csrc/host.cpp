// Host path of the eager layer calls: a CPython extension over libadder_b200.so that does in C++ what the Python layer
// (adder.py, adder_cuda.py, inference.py) does around a launch - checks, output allocation, the autograd node, the side stream
// of the weight gradient.  A small layer's kernels take 10-20 us; the Python around its forward and backward took 150.
//
// Every entry point takes the common case only (contiguous fp32 CUDA tensors of a geometry the fused kernels are built for) and
// returns None for anything else, errors included: the caller then goes through the Python layer, which handles or rejects it.
#include <torch/extension.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDAGuard.h>

#include <array>
#include <atomic>
#include <mutex>

#include "../../include/adder_b200.h"

namespace {

struct Api {      // entry points of the loaded libadder_b200.so
    decltype(&adder_b200_status_string) status_string = nullptr;
    decltype(&adder_b200_forward) forward = nullptr;
    decltype(&adder_b200_forward_stat_slices) forward_stat_slices = nullptr;
    decltype(&adder_b200_forward_with_stats) forward_with_stats = nullptr;
    decltype(&adder_b200_forward_affine) forward_affine = nullptr;
    decltype(&adder_b200_affine_forward) affine_forward = nullptr;
    decltype(&adder_b200_backward_input_workspace_bytes) backward_input_workspace_bytes = nullptr;
    decltype(&adder_b200_backward_input_with_workspace) backward_input_with_workspace = nullptr;
    decltype(&adder_b200_backward_weight_workspace_bytes) backward_weight_workspace_bytes = nullptr;
    decltype(&adder_b200_backward_weight) backward_weight = nullptr;
    decltype(&adder_b200_conv_forward) conv_forward = nullptr;
    decltype(&adder_b200_conv_backward_input_workspace_bytes) conv_backward_input_workspace_bytes = nullptr;
    decltype(&adder_b200_conv_backward_input_with_workspace) conv_backward_input_with_workspace = nullptr;
    decltype(&adder_b200_conv_backward_weight_workspace_bytes) conv_backward_weight_workspace_bytes = nullptr;
    decltype(&adder_b200_conv_backward_weight) conv_backward_weight = nullptr;
};
// Written once, by the first bind to the product library, which is never unloaded: autograd nodes made by this path call through it
// for as long as they live, from any thread.  `enabled` is what bind() switches, and only the Python entry points look at it.
Api api;
std::atomic<bool> enabled{false};
PyObject* g_adder_dict = nullptr;          // module dictionaries that hold FAST_CLAMP, OVERLAP_BACKWARD and ETA
PyObject* g_cuda_dict = nullptr;

// A torch.jit trace records the Python layer's autograd functions as operators; what runs here would leave a constant in it.
bool available() { return enabled.load(std::memory_order_acquire) && !torch::jit::tracer::isTracing(); }

// ValueError for what the caller can mend, RuntimeError otherwise, as _lib.check raises.
void check(int status, const char* what) {
    const bool runtime = status == ADDER_ERR_CUDA || status == ADDER_ERR_INTERNAL || status == ADDER_ERR_TIMEOUT;
    TORCH_CHECK(status == ADDER_OK || !runtime, what, ": ", api.status_string(status), " (status ", status, ")");
    TORCH_CHECK_VALUE(status == ADDER_OK, what, ": ", api.status_string(status), " (status ", status, ")");
}

cudaStream_t current_stream(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

at::Tensor empty_on(const at::Tensor& like, at::IntArrayRef sizes, at::ScalarType type = at::kFloat) {
    return at::detail::empty_cuda(sizes, type, like.device(), c10::nullopt);
}

struct Layer {      // geometry arguments of the C interface
    int n, ci, h, w, co, k, stride, pad, ho, wo;
};
#define ADDER_GEOM(L) (L).n, (L).ci, (L).h, (L).w, (L).co, (L).k, (L).stride, (L).pad

// What the kernels take.  A dual tensor of forward-mode differentiation is left to the Python layer, which refuses it: without a node,
// its tangent would be dropped without a word.
bool plain(const at::Tensor& t) {
    static const c10::DispatchKeySet wrapped({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                              c10::DispatchKey::Functionalize, c10::DispatchKey::Python,
                                              c10::DispatchKey::Conjugate, c10::DispatchKey::Negative});
    return t.is_cuda() && t.scalar_type() == at::kFloat && t.layout() == at::kStrided && t.is_contiguous() && !t.key_set().has_any(wrapped) &&
           !t._fw_grad(0).defined();
}

bool layer_of(const at::Tensor& x, const at::Tensor& w, int64_t stride, int64_t pad, Layer* L) {
    if (!plain(x) || !plain(w) || x.device() != w.device() || x.dim() != 4 || w.dim() != 4) return false;
    const int64_t k = w.size(2);
    if (w.size(3) != k || (k != 1 && k != 3) || (stride != 1 && stride != 2) || pad < 0 || pad >= k) return false;
    if (w.size(1) != x.size(1) || x.numel() == 0 || w.numel() == 0) return false;
    const int64_t h = x.size(2), wd = x.size(3), ho = (h + 2 * pad - k) / stride + 1, wo = (wd + 2 * pad - k) / stride + 1;
    if (h + 2 * pad < k || wd + 2 * pad < k) return false;
    constexpr int64_t lim = 2147483647;
    if (x.numel() > lim || w.numel() > lim || x.size(0) * w.size(0) * ho * wo > lim) return false;
    *L = Layer{(int)x.size(0), (int)x.size(1), (int)h, (int)wd, (int)w.size(0), (int)k, (int)stride, (int)pad, (int)ho, (int)wo};
    return true;
}

// ------------------------------------------------------------------------------------------ the operations

at::Tensor forward(const at::Tensor& x, const at::Tensor& w, const Layer& L) {
    const c10::cuda::CUDAGuard guard(x.device());
    at::Tensor out = empty_on(x, {L.n, L.co, L.ho, L.wo});
    check(api.forward(x.const_data_ptr<float>(), w.const_data_ptr<float>(), out.mutable_data_ptr<float>(), ADDER_GEOM(L), current_stream(x)),
          "adder_b200_forward");
    return out;
}

std::pair<at::Tensor, at::Tensor> forward_with_stats(const at::Tensor& x, const at::Tensor& w, const Layer& L) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int slices = api.forward_stat_slices(ADDER_GEOM(L));
    at::Tensor st = empty_on(x, {L.co, slices > 0 ? slices : 0, 2}, at::kDouble);
    if (slices <= 0) return {forward(x, w, L), st};
    at::Tensor out = empty_on(x, {L.n, L.co, L.ho, L.wo});
    check(api.forward_with_stats(x.const_data_ptr<float>(), w.const_data_ptr<float>(), out.mutable_data_ptr<float>(),
                                 st.mutable_data_ptr<double>(), slices, ADDER_GEOM(L), current_stream(x)), "adder_b200_forward_with_stats");
    return {out, st};
}

// The scratch comes from torch's caching allocator on the current stream: a cached block most of the time, safe with any number
// of threads and streams, and part of the graph's own pool under capture.
void backward_input(const at::Tensor& g, const at::Tensor& x, const at::Tensor& w, const at::Tensor& gx, const Layer& L, bool fast) {
    const size_t bytes = api.backward_input_workspace_bytes(ADDER_GEOM(L));
    at::Tensor ws;
    if (bytes > 0) ws = empty_on(x, {(int64_t)bytes}, at::kByte);
    check(api.backward_input_with_workspace(g.const_data_ptr<float>(), x.const_data_ptr<float>(), w.const_data_ptr<float>(), gx.mutable_data_ptr<float>(),
                                            bytes > 0 ? ws.mutable_data_ptr() : nullptr, bytes, ADDER_GEOM(L), fast ? ADDER_FLAG_FAST_CLAMP : 0,
                                            current_stream(x)), "adder_b200_backward_input");
}

void backward_weight(const at::Tensor& g, const at::Tensor& x, const at::Tensor& w, const at::Tensor& gw, const Layer& L, float eta) {
    const int64_t bytes = (int64_t)api.backward_weight_workspace_bytes(ADDER_GEOM(L));
    at::Tensor ws = empty_on(x, {bytes}, at::kByte);
    check(api.backward_weight(g.const_data_ptr<float>(), x.const_data_ptr<float>(), w.const_data_ptr<float>(), gw.mutable_data_ptr<float>(), eta,
                              nullptr, ws.mutable_data_ptr(), (size_t)bytes, ADDER_GEOM(L), 0, current_stream(x)), "adder_b200_backward_weight");
}

c10::cuda::CUDAStream side_stream(c10::DeviceIndex dev) {
    static std::mutex mu;
    static std::array<std::unique_ptr<c10::cuda::CUDAStream>, 64> streams;
    std::lock_guard<std::mutex> lock(mu);
    auto& s = streams.at(dev);
    if (!s) s = std::make_unique<c10::cuda::CUDAStream>(c10::cuda::getStreamFromPool(false, dev));
    return *s;
}

// Both gradients; with `overlap` the weight gradient runs on a side stream beside the input gradient.
// What that gives depends on what else runs.  Among other passes (250 drawn layers) it saves 4 % from 1.5e8 to 2.5e8 terms, 2 % up to
// 1e9, less above.  A pass that is waited for gains or loses: where the input gradient is one long chain on few CTAs, the weight
// gradient's CTAs, each of which fills an SM, may take the SMs first and leave it crowded on the rest (256->256 14x14 at batch 2:
// 356 us, 200 one after the other; the other order loses as much on 256->512 14x14 stride 2 at batch 4, 596 against 250).  Below 1.5e8
// terms one after the other is the faster on average there, and the events cost 6 us of host time; inside a graph capture they
// cost nothing.
constexpr double OVERLAP_TERMS = 1.5e8;

template <class Input, class Weight>
void run_both(const at::Tensor& x, bool overlap, double terms, Input input, Weight weight) {
    if (!overlap || (terms < OVERLAP_TERMS && at::cuda::currentStreamCaptureStatusMayInitCtx() == at::cuda::CaptureStatus::None)) {
        input();
        weight();
        return;
    }
    const auto cur = c10::cuda::getCurrentCUDAStream(x.device().index());
    const auto side = side_stream(x.device().index());
    at::cuda::CUDAEvent ready, done;
    ready.record(cur);
    ready.block(side);
    {
        const c10::cuda::CUDAStreamGuard on_side(side);
        weight();
        done.record(side);
    }
    input();
    done.block(cur);
}

void backward_both(const at::Tensor& g, const at::Tensor& x, const at::Tensor& w, const at::Tensor& gx, const at::Tensor& gw,
                   const Layer& L, float eta, bool fast, bool overlap) {
    run_both(x, overlap, (double)L.n * L.ho * L.wo * L.co * L.ci * L.k * L.k, [&] { backward_input(g, x, w, gx, L, fast); }, [&] { backward_weight(g, x, w, gw, L, eta); });
}

// ------------------------------------------------------------------------------------------ any other geometry

// n, ci, h, w, co, kh, kw, sh, sw, ph, pw, dh, dw; then ho, wo
using Conv = std::array<int, 15>;
#define ADDER_CONV_GEOM(c) c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9], c[10], c[11], c[12]

bool conv_of(const at::Tensor& x, const at::Tensor& w, const std::array<int64_t, 6>& p, Conv* c) {
    if (!plain(x) || !plain(w) || x.device() != w.device() || x.dim() != 4 || w.dim() != 4) return false;
    if (w.size(1) != x.size(1) || x.numel() == 0 || w.numel() == 0) return false;
    constexpr int64_t lim = 2147483647;
    for (int i = 0; i < 6; ++i)
        if (p[i] < (i == 2 || i == 3 ? 0 : 1) || p[i] > (1 << 20)) return false;      // stride, padding, dilation
    // Beyond 24x24 the input gradient is mostly zeros between the pixels that a window reaches, which columns fold faster (16->16 on
    // 256x256 at batch 8, forward and backward: 1x1 stride 64 1220 us here, 395 as columns; 2x2 stride 24 452 and 399, 1x1 stride 17
    // 177 and 401).
    if (p[0] * p[1] > 600) return false;
    const int64_t h = x.size(2), wd = x.size(3), kh = w.size(2), kw = w.size(3);
    const int64_t eh = h + 2 * p[2] - p[4] * (kh - 1) - 1, ew = wd + 2 * p[3] - p[5] * (kw - 1) - 1;
    if (eh < 0 || ew < 0) return false;
    const int64_t ho = eh / p[0] + 1, wo = ew / p[1] + 1;
    if (x.numel() > lim || w.numel() > lim || x.size(0) * w.size(0) * ho * wo > lim) return false;
    *c = Conv{(int)x.size(0), (int)x.size(1), (int)h, (int)wd, (int)w.size(0), (int)kh, (int)kw, (int)p[0], (int)p[1], (int)p[2], (int)p[3],
              (int)p[4], (int)p[5], (int)ho, (int)wo};
    return api.conv_backward_weight_workspace_bytes(ADDER_CONV_GEOM((*c))) > 0;
}

at::Tensor conv_forward(const at::Tensor& x, const at::Tensor& w, const Conv& c) {
    const c10::cuda::CUDAGuard guard(x.device());
    at::Tensor out = empty_on(x, {c[0], c[4], c[13], c[14]});
    check(api.conv_forward(x.const_data_ptr<float>(), w.const_data_ptr<float>(), out.mutable_data_ptr<float>(), ADDER_CONV_GEOM(c),
                           current_stream(x)), "adder_b200_conv_forward");
    return out;
}

void conv_backward_input(const at::Tensor& g, const at::Tensor& x, const at::Tensor& w, const at::Tensor& gx, const Conv& c, bool fast) {
    const size_t bytes = api.conv_backward_input_workspace_bytes(ADDER_CONV_GEOM(c));
    at::Tensor ws;
    if (bytes > 0) ws = empty_on(x, {(int64_t)bytes}, at::kByte);
    check(api.conv_backward_input_with_workspace(g.const_data_ptr<float>(), x.const_data_ptr<float>(), w.const_data_ptr<float>(),
                                                 gx.mutable_data_ptr<float>(), bytes > 0 ? ws.mutable_data_ptr() : nullptr, bytes, ADDER_CONV_GEOM(c),
                                                 fast ? ADDER_FLAG_FAST_CLAMP : 0, current_stream(x)), "adder_b200_conv_backward_input");
}

void conv_backward_weight(const at::Tensor& g, const at::Tensor& x, const at::Tensor& w, const at::Tensor& gw, const Conv& c, float eta) {
    const int64_t bytes = (int64_t)api.conv_backward_weight_workspace_bytes(ADDER_CONV_GEOM(c));
    at::Tensor ws = empty_on(x, {bytes}, at::kByte);
    check(api.conv_backward_weight(g.const_data_ptr<float>(), x.const_data_ptr<float>(), w.const_data_ptr<float>(),
                                   gw.mutable_data_ptr<float>(), eta, ws.mutable_data_ptr(), (size_t)bytes, ADDER_CONV_GEOM(c),
                                   current_stream(x)), "adder_b200_conv_backward_weight");
}

// ------------------------------------------------------------------------------------------ autograd nodes

using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// What a saved-tensor hook hands back need not be what it was given: every backward looks at its tensors again.
constexpr const char* SAVED = "the saved tensors came back in another form: contiguous float32 CUDA tensors of the forward's shapes are needed";

at::Tensor gradient(const Variable& grad, const at::Tensor& x, at::IntArrayRef shape) {
    const at::Tensor g = grad.contiguous();
    TORCH_CHECK(g.scalar_type() == at::kFloat && g.device() == x.device(), "grad_out must be a float32 tensor on the layer's device");
    TORCH_CHECK(g.sizes() == shape, "grad_out has shape ", g.sizes(), ", expected ", shape);
    return g;
}

struct Settings { bool fast, overlap; float eta; };

// The module-level switches are read when the backward runs, as the Python layer reads them.
Settings settings() {
    pybind11::gil_scoped_acquire gil;
    auto flag = [](PyObject* dict, const char* name) {
        PyObject* v = PyDict_GetItemString(dict, name);
        return v != nullptr && PyObject_IsTrue(v) == 1;
    };
    PyObject* eta = PyDict_GetItemString(g_cuda_dict, "ETA");
    return {flag(g_adder_dict, "FAST_CLAMP"), flag(g_adder_dict, "OVERLAP_BACKWARD"), eta != nullptr ? (float)PyFloat_AsDouble(eta) : 0.2f};
}


// adder2d on NCHW tensors (adder.py:22-80 of the reference).
struct AdderLayer : public torch::autograd::Function<AdderLayer> {
    static variable_list forward(AutogradContext* ctx, const Variable& x, const Variable& w, int64_t stride, int64_t pad, bool stats) {
        Layer L;
        TORCH_CHECK(layer_of(x, w, stride, pad, &L));
        ctx->save_for_backward({x, w});
        ctx->saved_data["stride"] = stride;
        ctx->saved_data["pad"] = pad;
        if (!stats) return {::forward(x, w, L)};
        auto r = ::forward_with_stats(x, w, L);
        ctx->mark_non_differentiable({r.second});
        ctx->set_materialize_grads(false);
        return {r.first, r.second};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        if (!grads[0].defined()) return {Variable(), Variable(), Variable(), Variable(), Variable()};
        const auto saved = ctx->get_saved_variables();
        const Variable &x = saved[0], &w = saved[1];
        Layer L;
        TORCH_CHECK(layer_of(x, w, ctx->saved_data["stride"].toInt(), ctx->saved_data["pad"].toInt(), &L), SAVED);
        const at::Tensor g = gradient(grads[0], x, {L.n, L.co, L.ho, L.wo});
        const c10::cuda::CUDAGuard guard(x.device());
        const Settings set = settings();
        at::Tensor gx, gw;
        if (ctx->needs_input_grad(0)) gx = empty_on(x, x.sizes());
        if (ctx->needs_input_grad(1)) gw = empty_on(w, w.sizes());
        if (gx.defined() && gw.defined()) backward_both(g, x, w, gx, gw, L, set.eta, set.fast, set.overlap);
        else if (gx.defined()) backward_input(g, x, w, gx, L, set.fast);
        else if (gw.defined()) backward_weight(g, x, w, gw, L, set.eta);
        return {gx, gw, Variable(), Variable(), Variable()};
    }
};

struct ConvLayer : public torch::autograd::Function<ConvLayer> {
    static Variable forward(AutogradContext* ctx, const Variable& x, const Variable& w, const std::vector<int64_t>& p) {
        Conv c;
        TORCH_CHECK(conv_of(x, w, {p[0], p[1], p[2], p[3], p[4], p[5]}, &c));
        ctx->save_for_backward({x, w});
        ctx->saved_data["p"] = p;
        return conv_forward(x, w, c);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Variable &x = saved[0], &w = saved[1];
        const auto p = ctx->saved_data["p"].toIntVector();
        Conv c;
        TORCH_CHECK(conv_of(x, w, {p[0], p[1], p[2], p[3], p[4], p[5]}, &c), SAVED);
        const at::Tensor g = gradient(grads[0], x, {c[0], c[4], c[13], c[14]});
        const c10::cuda::CUDAGuard guard(x.device());
        const Settings set = settings();
        at::Tensor gx, gw;
        if (ctx->needs_input_grad(0)) gx = empty_on(x, x.sizes());
        if (ctx->needs_input_grad(1)) gw = empty_on(w, w.sizes());
        auto input = [&] { conv_backward_input(g, x, w, gx, c, set.fast); };
        auto weight = [&] { conv_backward_weight(g, x, w, gw, c, set.eta); };
        if (gx.defined() && gw.defined()) run_both(x, set.overlap, (double)w.numel() * g.size(0) * c[13] * c[14], input, weight);
        else if (gx.defined()) input();
        else if (gw.defined()) weight();
        return {gx, gw, Variable()};
    }
};

// The column-matrix op (adder.py:43-80 of the reference): X[K,P] is the 1x1 layer [1,K,1,P], W[Co,K] its kernel.
bool column_of(const at::Tensor& w, const at::Tensor& x, Layer* L) {
    if (!plain(w) || !plain(x) || w.dim() != 2 || x.dim() != 2 || w.size(1) != x.size(0) || w.numel() == 0 || x.numel() == 0 ||
        w.device() != x.device())
        return false;
    constexpr int64_t lim = 2147483647;
    if (w.numel() > lim || x.numel() > lim || w.size(0) * x.size(1) > lim) return false;
    *L = Layer{1, (int)x.size(0), 1, (int)x.size(1), (int)w.size(0), 1, 1, 0, 1, (int)x.size(1)};
    return true;
}

struct AdderColumn : public torch::autograd::Function<AdderColumn> {
    static Variable forward(AutogradContext* ctx, const Variable& w, const Variable& x) {
        Layer L;
        TORCH_CHECK(column_of(w, x, &L));
        ctx->save_for_backward({w, x});
        return ::forward(x, w, L).view({L.co, L.w});
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Variable &w = saved[0], &x = saved[1];
        Layer L;
        TORCH_CHECK(column_of(w, x, &L), SAVED);
        const at::Tensor g = gradient(grads[0], x, {L.co, L.w});
        const c10::cuda::CUDAGuard guard(x.device());
        at::Tensor gx = empty_on(x, x.sizes()), gw = empty_on(w, w.sizes());
        backward_both(g, x, w, gx, gw, L, 0.2f, false, true);
        return {gw, gx};
    }
};

// ------------------------------------------------------------------------------------------ Python entry points

const at::Tensor* tensor_arg(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

bool int_arg(PyObject* o, int64_t* v) {
    if (!PyLong_CheckExact(o)) return false;
    int overflow = 0;
    *v = PyLong_AsLongLongAndOverflow(o, &overflow);
    return overflow == 0;
}

bool needs_node(const at::Tensor& a, const at::Tensor& b) { return at::GradMode::is_enabled() && (a.requires_grad() || b.requires_grad()); }

// layer(x, w, stride, padding) -> out, or None
PyObject* py_layer(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4 || !available()) Py_RETURN_NONE;
    const at::Tensor *x = tensor_arg(args[0]), *w = tensor_arg(args[1]);
    int64_t stride, pad;
    Layer L;
    if (x == nullptr || w == nullptr || !int_arg(args[2], &stride) || !int_arg(args[3], &pad) || !layer_of(*x, *w, stride, pad, &L)) Py_RETURN_NONE;
    at::Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        out = needs_node(*x, *w) ? AdderLayer::apply(*x, *w, stride, pad, false)[0] : forward(*x, *w, L);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// conv(x, w, sh, sw, ph, pw, dh, dw) -> out, or None
PyObject* py_conv(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8 || !available()) Py_RETURN_NONE;
    const at::Tensor *x = tensor_arg(args[0]), *w = tensor_arg(args[1]);
    std::array<int64_t, 6> p;
    for (int i = 0; i < 6; ++i)
        if (!int_arg(args[2 + i], &p[i])) Py_RETURN_NONE;
    Conv c;
    if (x == nullptr || w == nullptr || !conv_of(*x, *w, p, &c)) Py_RETURN_NONE;
    at::Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        out = needs_node(*x, *w) ? ConvLayer::apply(*x, *w, std::vector<int64_t>(p.begin(), p.end())) : conv_forward(*x, *w, c);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// layer_with_stats(x, w, stride, padding) -> (out, statistics), or None
PyObject* py_layer_with_stats(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4 || !available()) Py_RETURN_NONE;
    const at::Tensor *x = tensor_arg(args[0]), *w = tensor_arg(args[1]);
    int64_t stride, pad;
    Layer L;
    if (x == nullptr || w == nullptr || !int_arg(args[2], &stride) || !int_arg(args[3], &pad) || !layer_of(*x, *w, stride, pad, &L)) Py_RETURN_NONE;
    at::Tensor out, st;
    {
        pybind11::gil_scoped_release no_gil;
        if (needs_node(*x, *w)) {
            auto r = AdderLayer::apply(*x, *w, stride, pad, true);
            out = r[0]; st = r[1];
        } else {
            std::tie(out, st) = forward_with_stats(*x, *w, L);
        }
    }
    return Py_BuildValue("(NN)", THPVariable_Wrap(std::move(out)), THPVariable_Wrap(std::move(st)));
    END_HANDLE_TH_ERRORS
}

bool affine_args(PyObject* scale, PyObject* shift, PyObject* residual, const at::Tensor& like, int64_t channels, at::IntArrayRef shape,
                 const at::Tensor** sc, const at::Tensor** sh, const at::Tensor** res) {
    *sc = tensor_arg(scale); *sh = tensor_arg(shift);
    *res = residual == Py_None ? nullptr : tensor_arg(residual);
    if (*sc == nullptr || *sh == nullptr || (residual != Py_None && *res == nullptr)) return false;
    for (const at::Tensor* t : {*sc, *sh})
        if (!plain(*t) || t->numel() != channels || t->device() != like.device()) return false;
    return *res == nullptr || (plain(**res) && (*res)->sizes() == shape && (*res)->device() == like.device() && !(*res)->requires_grad());
}

// layer_affine(x, w, stride, padding, scale, shift, residual, relu) -> relu?(layer * scale + shift + residual) without autograd, or None
PyObject* py_layer_affine(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8 || !available()) Py_RETURN_NONE;
    const at::Tensor *x = tensor_arg(args[0]), *w = tensor_arg(args[1]), *sc, *sh, *res;
    int64_t stride, pad;
    Layer L;
    if (x == nullptr || w == nullptr || !int_arg(args[2], &stride) || !int_arg(args[3], &pad) || !layer_of(*x, *w, stride, pad, &L) || needs_node(*x, *w))
        Py_RETURN_NONE;
    const std::array<int64_t, 4> shape{L.n, L.co, L.ho, L.wo};
    if (!affine_args(args[4], args[5], args[6], *x, L.co, shape, &sc, &sh, &res)) Py_RETURN_NONE;
    const int relu = PyObject_IsTrue(args[7]);
    at::Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(x->device());
        out = empty_on(*x, shape);
        check(api.forward_affine(x->const_data_ptr<float>(), w->const_data_ptr<float>(), sc->const_data_ptr<float>(), sh->const_data_ptr<float>(),
                                 res != nullptr ? res->const_data_ptr<float>() : nullptr, relu, out.mutable_data_ptr<float>(), ADDER_GEOM(L),
                                 current_stream(*x)), "adder_b200_forward_affine");
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// affine(y, scale, shift, residual, relu) -> the same behind a tensor, or None
PyObject* py_affine(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5 || !available()) Py_RETURN_NONE;
    const at::Tensor *y = tensor_arg(args[0]), *sc, *sh, *res;
    if (y == nullptr || !plain(*y) || y->dim() != 4 || y->numel() == 0 || y->numel() > 2147483647) Py_RETURN_NONE;
    if (!affine_args(args[1], args[2], args[3], *y, y->size(1), y->sizes(), &sc, &sh, &res)) Py_RETURN_NONE;
    const int relu = PyObject_IsTrue(args[4]);
    at::Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(y->device());
        out = empty_on(*y, y->sizes());
        check(api.affine_forward(y->const_data_ptr<float>(), sc->const_data_ptr<float>(), sh->const_data_ptr<float>(),
                                 res != nullptr ? res->const_data_ptr<float>() : nullptr, out.mutable_data_ptr<float>(), relu, (int)y->size(0),
                                 (int)y->size(1), (int)(y->size(2) * y->size(3)), current_stream(*y)), "adder_b200_affine_forward");
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// column(W[Co,K], X[K,P]) -> [Co,P], or None
PyObject* py_column(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2 || !available()) Py_RETURN_NONE;
    const at::Tensor *w = tensor_arg(args[0]), *x = tensor_arg(args[1]);
    Layer L;
    if (w == nullptr || x == nullptr || !column_of(*w, *x, &L)) Py_RETURN_NONE;
    at::Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        if (needs_node(*w, *x)) out = AdderColumn::apply(*w, *x);
        else out = forward(*x, *w, L).view({L.co, L.w});
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// bind({name: address}, adder module dict, adder_cuda module dict) switches the entry points on, bind(None, ...) off
PyObject* py_bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(n == 3 && PyDict_Check(args[1]) && PyDict_Check(args[2]), "bind(addresses, dict, dict)");
    enabled.store(false, std::memory_order_release);
    const bool on = args[0] != Py_None;
    if (on && api.forward == nullptr) {
        Api a;
        auto get = [&](const char* name, auto* fn) {
            PyObject* v = PyDict_GetItemString(args[0], name);
            TORCH_CHECK(v != nullptr && PyLong_Check(v), "no address for ", name);
            *fn = reinterpret_cast<std::remove_pointer_t<decltype(fn)>>(PyLong_AsVoidPtr(v));
        };
        get("adder_b200_status_string", &a.status_string);
        get("adder_b200_forward", &a.forward);
        get("adder_b200_forward_stat_slices", &a.forward_stat_slices);
        get("adder_b200_forward_with_stats", &a.forward_with_stats);
        get("adder_b200_forward_affine", &a.forward_affine);
        get("adder_b200_affine_forward", &a.affine_forward);
        get("adder_b200_backward_input_workspace_bytes", &a.backward_input_workspace_bytes);
        get("adder_b200_backward_input_with_workspace", &a.backward_input_with_workspace);
        get("adder_b200_backward_weight_workspace_bytes", &a.backward_weight_workspace_bytes);
        get("adder_b200_backward_weight", &a.backward_weight);
        get("adder_b200_conv_forward", &a.conv_forward);
        get("adder_b200_conv_backward_input_workspace_bytes", &a.conv_backward_input_workspace_bytes);
        get("adder_b200_conv_backward_input_with_workspace", &a.conv_backward_input_with_workspace);
        get("adder_b200_conv_backward_weight_workspace_bytes", &a.conv_backward_weight_workspace_bytes);
        get("adder_b200_conv_backward_weight", &a.conv_backward_weight);
        api = a;
    }
    Py_INCREF(args[1]); Py_INCREF(args[2]);
    Py_XDECREF(g_adder_dict); Py_XDECREF(g_cuda_dict);
    g_adder_dict = args[1]; g_cuda_dict = args[2];
    enabled.store(on, std::memory_order_release);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

#define ADDER_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ADDER_METHOD("bind", py_bind), ADDER_METHOD("layer", py_layer), ADDER_METHOD("conv", py_conv), ADDER_METHOD("layer_with_stats", py_layer_with_stats),
                         ADDER_METHOD("layer_affine", py_layer_affine), ADDER_METHOD("affine", py_affine), ADDER_METHOD("column", py_column),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_adder_host", nullptr, -1, methods};

}  // namespace

#ifndef ADDER_HOST_MARK
#define ADDER_HOST_MARK ""
#endif

// The mark says which torch this file was linked with; build.py looks for it before it is loaded.
PyMODINIT_FUNC PyInit__adder_host() {
    PyObject* m = PyModule_Create(&module_def);
    if (m != nullptr) PyModule_AddStringConstant(m, "built_for", ADDER_HOST_MARK);
    return m;
}
