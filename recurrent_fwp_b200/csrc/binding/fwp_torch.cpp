// Host path of the autograd entry points: argument checks, output allocation, the launch through the C ABI of
// fwp.h and the autograd node, all in native code.
//
// Most calls of these ops are shorter on the GPU than a Python autograd.Function takes to issue them: the acting step
// of 32 environments runs 3-5 us on the device and took 44 us from the Python wrappers (descriptors through ctypes,
// one torch.empty per output, Function.apply), and the language-model training step was host-bound at 762 us for
// 310 us of device time.  Here a call costs one METH_FASTCALL entry, the allocations and the launch.
//
// Division of labour with the Python modules: a function here returns NotImplemented when an argument is not in the
// form the kernels take (wrong type, device, shape or a strided inner dimension).  The module then runs its own
// checks, which raise the documented error, or lays the streams out and calls again.  So the checks below only have
// to recognise good arguments.
#include <Python.h>
#include <array>
#include <mutex>
#include <vector>
#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/Exception.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/utils/pybind.h>
#include "../../../include/fwp.h"

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

bool g_check_fault = false;     // FWP_CHECK_DEVICE_FAULT: ask for a device fault after every launch of the delta and sum rules

struct Dims {
    int64_t N, H, L, E, M;
};

// ---------------------------------------------------------------- descriptors
fwp_tensor desc(const Tensor& t) {
    fwp_tensor d;
    if (!t.defined()) {
        d.data = nullptr;
        for (auto& s : d.stride) s = 0;
        return d;
    }
    d.data = t.data_ptr();
    const auto st = t.strides();
    for (int i = 0; i < 4; i++) d.stride[i] = st[i];
    if (t.size(3) == 1) d.stride[3] = 1;
    return d;
}
struct Desc {        // a descriptor whose address can be passed in the call expression
    fwp_tensor d;
    explicit Desc(const Tensor& t) : d(desc(t)) {}
    operator const fwp_tensor*() const { return &d; }
};
struct Desc3 {
    fwp_tensor d[3];
    explicit Desc3(const Tensor* t) : d{desc(t[0]), desc(t[1]), desc(t[2])} {}
    operator const fwp_tensor*() const { return d; }
};

void check(int rc, const char* what) {
    if (rc == FWP_OK) return;
    if (rc == FWP_ERR_CUDA)
        TORCH_CHECK(false, what, " failed: ", fwp_status_string(rc), " [cudaError ", fwp_last_cuda_error(), "]");
    TORCH_CHECK(false, what, " failed: ", fwp_status_string(rc));
}
// for the ops whose kernels have bounded waits
void check_waits(int rc, const char* what) {
    check(rc, what);
    if (g_check_fault)
        TORCH_CHECK(fwp_delta_device_fault() == 0, what, ": a bounded wait inside the kernel ran out; its results are invalid");
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kFloat ? FWP_F32 : FWP_BF16; }

// Outputs come straight from the caching allocator (no dispatcher round trip: about 0.5 us less per tensor).
Tensor empty(std::initializer_list<int64_t> size, at::ScalarType type, const Tensor& like) {
    return Tensor(at::detail::empty_cuda(at::IntArrayRef(size.begin(), size.size()), type, like.device(), std::nullopt));
}
Tensor empty(const Dims& d, int64_t width, const Tensor& like) {
    return empty({d.N, d.H, d.L, width}, at::kFloat, like);
}

// ------------------------------------------------------------------ arguments
bool shaped(const Tensor& t, at::ScalarType type, const at::Device& dev, int64_t n, int64_t h, int64_t l, int64_t w) {
    if (!t.defined() || t.dim() != 4 || t.layout() != at::kStrided || t.scalar_type() != type || t.device() != dev) return false;
    const auto s = t.sizes();
    return s[0] == n && s[1] == h && s[2] == l && s[3] == w && (w == 1 || t.strides()[3] == 1);
}
bool first_stream(const Tensor& t, bool bf16) {
    return t.defined() && t.dim() == 4 && t.is_cuda() && t.layout() == at::kStrided &&
           (t.scalar_type() == at::kFloat || (bf16 && t.scalar_type() == at::kBFloat16)) &&
           (t.size(3) == 1 || t.stride(3) == 1);
}

// Borrowed tensor arguments of a METH_FASTCALL function; false when one of them is not a plain tensor.  A tensor with a
// forward-mode tangent or a wrapper of a function transform is not, and nothing is while torch.jit traces: a call from here
// would drop the tangent, or leave its result in the trace as a constant.  The module has an autograd.Function for those.
template <size_t K>
bool tensors(PyObject* const* args, Py_ssize_t n, std::array<const Tensor*, K>& out) {
    if (n < (Py_ssize_t)K || at::tracer::impl::is_dispatch_enabled()) return false;
    constexpr c10::DispatchKeySet wrappers({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper});
    for (size_t i = 0; i < K; i++) {
        if (!THPVariable_Check(args[i])) return false;
        const Tensor& t = THPVariable_Unpack(args[i]);
        const auto* impl = t.unsafeGetTensorImpl();
        if (impl->key_set().has_any(wrappers) || (impl->autograd_meta() && torch::autograd::isFwGradDefined(t))) return false;
        out[i] = &t;
    }
    return true;
}
PyObject* not_implemented() { Py_RETURN_NOTIMPLEMENTED; }

template <size_t K>
bool needs_grad(const std::array<const Tensor*, K>& in) {
    if (!at::GradMode::is_enabled()) return false;
    for (auto* t : in)
        if (t->requires_grad()) return true;
    return false;
}

// ------------------------------------------------------------- autograd nodes
// What a backward needs is saved as torch's own nodes save it, so that saved-tensor hooks (activation checkpointing,
// offloading) see all of it: `user` holds what the caller can also reach (inputs, states, outputs; version-checked on
// unpack), `own` the buffers only this call knows.  Gradients are returned in the order of the forward's arguments,
// undefined for the states.
struct OpNode : public Node {
    Dims d;
    std::vector<SavedVariable> user, own;
    void save(const Tensor& t) { user.emplace_back(t, false); }
    void save_output(const Tensor& t) { user.emplace_back(t, true); }
    void keep(std::initializer_list<Tensor> l) {
        own.reserve(l.size());
        for (auto& t : l) own.emplace_back(t, false);
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto& s : user) s.reset_data();
        for (auto& s : own) s.reset_data();
    }
    std::vector<Tensor> unpack(std::vector<SavedVariable>& saved) {
        std::vector<Tensor> t;
        t.reserve(saved.size());
        for (auto& s : saved) t.push_back(s.unpack(shared_from_this()));
        return t;
    }
    // the incoming gradient in the streams' element type with a unit inner stride
    static Tensor incoming(const Tensor& g, const Tensor& like, at::IntArrayRef shape) {
        if (!g.defined()) return at::zeros(shape, like.options());
        TORCH_CHECK(g.device() == like.device() && g.sizes() == shape, "grad_out is ", g.sizes(), " on ", g.device(),
                    ", expected ", shape, " on ", like.device());
        Tensor r = g.scalar_type() == like.scalar_type() ? g : g.to(like.scalar_type());
        return r.size(-1) == 1 || r.stride(-1) == 1 ? r : r.contiguous();
    }
    Tensor like_stream(int64_t width, const Tensor& like) const { return empty({d.N, d.H, d.L, width}, like.scalar_type(), like); }
};

template <class NodeT, size_t K>
std::shared_ptr<NodeT> make_node(const std::array<const Tensor*, K>& in, const Dims& d) {
    auto node = std::shared_ptr<NodeT>(new NodeT(), torch::autograd::deleteNode);
    torch::autograd::edge_list edges;
    edges.reserve(K);
    for (auto* t : in) edges.push_back(t->requires_grad() ? torch::autograd::impl::gradient_edge(*t) : torch::autograd::Edge());
    node->set_next_edges(std::move(edges));
    node->d = d;
    return node;
}

// ------------------------------------------------------------------ delta rule
// the backward with the scratch memory it asks for; where the device has none left, without
void delta_backward(const Dims& d, const Tensor& Q, const Tensor& K, const Tensor& V, const Tensor& beta, const Tensor& v_old, const Desc& gy,
                    const Tensor& W, const Tensor& gQ, const Tensor& gK, const Tensor& gV, const Tensor& gb) {
    int64_t need = fwp_fast_weight_backward_scratch_floats(d.N, d.H, d.L, d.E, d.M, dtype_code(Q));
    Tensor scratch;
    if (need > 0) try {
        scratch = empty({need}, at::kFloat, Q);
    } catch (const c10::OutOfMemoryError&) {
        need = 0;
    }
    check_waits(fwp_fast_weight_backward_with_scratch(d.N, d.H, d.L, d.E, d.M, Desc(Q), Desc(K), Desc(V), Desc(beta), Desc(v_old), gy,
                                                      Desc(W), Desc(gQ), Desc(gK), Desc(gV), Desc(gb),
                                                      need > 0 ? scratch.data_ptr<float>() : nullptr, need, dtype_code(Q), stream_of(Q),
                                                      Q.device().index()), "fast_weight_backward");
}

struct DeltaNode final : public OpNode {
    std::string name() const override { return "DeltaFastWeightBackward"; }
    variable_list apply(variable_list&& g) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        const auto t = unpack(user), o = unpack(own);
        const Tensor &Q = t[0], &K = t[1], &V = t[2], &beta = t[3], &W = t[4];
        const Tensor gy = incoming(g[0], Q, {d.N, d.H, d.L, d.M});
        Tensor gQ = like_stream(d.E, Q), gK = like_stream(d.E, Q), gV = like_stream(d.M, Q), gb = like_stream(1, Q);
        delta_backward(d, Q, K, V, beta, o[0], Desc(gy), W, gQ, gK, gV, gb);
        return {gQ, gK, gV, gb, Tensor()};
    }
};

PyObject* fast_weight_delta(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    std::array<const Tensor*, 5> in;
    if (n != 5 || !tensors(args, n, in)) return not_implemented();
    const Tensor &Q = *in[0], &K = *in[1], &V = *in[2], &beta = *in[3], &W = *in[4];
    if (!first_stream(Q, true) || !V.defined() || V.dim() != 4) return not_implemented();
    const Dims d{Q.size(0), Q.size(1), Q.size(2), Q.size(3), V.size(3)};
    const auto ty = Q.scalar_type();
    const auto dev = Q.device();
    if (!shaped(K, ty, dev, d.N, d.H, d.L, d.E) || !shaped(V, ty, dev, d.N, d.H, d.L, d.M) ||
        !shaped(beta, ty, dev, d.N, d.H, d.L, 1) || !shaped(W, at::kFloat, dev, d.N, d.H, d.E, d.M))
        return not_implemented();
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        const bool grad = needs_grad(in);
        out = empty({d.N, d.H, d.L, d.M}, ty, Q);
        Tensor v_old;
        if (grad) v_old = empty(d, d.M, Q);
        check_waits(fwp_fast_weight_forward(d.N, d.H, d.L, d.E, d.M, Desc(Q), Desc(K), Desc(V), Desc(beta), Desc(v_old),
                                            Desc(Tensor()), Desc(W), Desc(out), dtype_code(Q), stream_of(Q), dev.index()),
                    "fast_weight_forward");
        if (grad) {
            auto node = make_node<DeltaNode>(in, d);
            for (auto* t : in) node->save(*t);
            node->keep({v_old});
            torch::autograd::create_gradient_edge(out, node);
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ------------------------------------- delta-rule attention layer: prologue, delta rule, epilogue in one node
// The layer's scale goes into the queries, and the delta rule writes its output (and reads the incoming gradient) as the
// (len, B, H, D) tensor it is: no transposing pass on either side (two of 8 us each at 256 sequences x 512 steps, D = 32).
Desc heads_first(const Tensor& t, const Dims& d) {
    Desc r(Tensor{});
    r.d.data = t.data_ptr();
    r.d.stride[0] = d.H * d.M;
    r.d.stride[1] = d.M;
    r.d.stride[2] = d.N * d.H * d.M;
    r.d.stride[3] = 1;
    return r;
}
struct DeltaLayerNode final : public OpNode {
    double scale = 1;
    std::string name() const override { return "DeltaAttentionBackward"; }
    variable_list apply(variable_list&& g) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        const auto t = unpack(user), o = unpack(own);
        const Tensor &x = t[0], &W = t[1], &q = o[0], &k = o[1], &v = o[2], &beta = o[3], &v_old = o[4];
        const Tensor gout = incoming(g[0], x, {d.L, d.N, d.H * d.M}).contiguous();
        void* st = stream_of(x);
        const int dev = x.device().index();
        const Desc gy = heads_first(gout, d);
        Tensor gq = empty(d, d.E, x), gk = empty(d, d.E, x), gv = empty(d, d.M, x), gb = empty(d, 1, x);
        delta_backward(d, q, k, v, beta, v_old, gy, W, gq, gk, gv, gb);
        Tensor gx = empty({d.L, d.N, d.H, 3 * d.E + 1}, at::kFloat, x);
        check(fwp_delta_layer_prologue_backward_scaled(d.L, d.N, d.H, d.E, x.data_ptr<float>(), gq.data_ptr<float>(), gk.data_ptr<float>(),
                                                       gv.data_ptr<float>(), gb.data_ptr<float>(), gx.data_ptr<float>(), (float)scale, st, dev),
              "delta_layer_prologue_backward");
        return {gx, Tensor()};
    }
};

PyObject* delta_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    std::array<const Tensor*, 2> in;
    if (n != 3 || !tensors(args, n, in)) return not_implemented();
    const double scale = PyFloat_AsDouble(args[2]);
    if (scale == -1. && PyErr_Occurred()) return nullptr;
    const Tensor &x = *in[0], &W = *in[1];
    if (!first_stream(x, false) || !x.is_contiguous() || (x.size(3) - 1) % 3) return not_implemented();
    const int64_t D = (x.size(3) - 1) / 3;
    const Dims d{x.size(1), x.size(2), x.size(0), D, D};
    if (!shaped(W, at::kFloat, x.device(), d.N, d.H, D, D)) return not_implemented();
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        void* st = stream_of(x);
        const int dev = x.device().index();
        Tensor q = empty(d, D, x), k = empty(d, D, x), v = empty(d, D, x), beta = empty(d, 1, x), v_old;
        out = empty({d.L, d.N, d.H * D}, at::kFloat, x);
        const bool grad = needs_grad(in);
        if (grad) v_old = empty(d, D, x);
        check(fwp_delta_layer_prologue_forward_scaled(d.L, d.N, d.H, D, x.data_ptr<float>(), q.data_ptr<float>(), k.data_ptr<float>(),
                                                      v.data_ptr<float>(), beta.data_ptr<float>(), (float)scale, st, dev),
              "delta_layer_prologue_forward");
        check_waits(fwp_fast_weight_forward(d.N, d.H, d.L, D, D, Desc(q), Desc(k), Desc(v), Desc(beta), Desc(v_old), Desc(Tensor()),
                                            Desc(W), heads_first(out, d), FWP_F32, st, dev), "fast_weight_forward");
        if (grad) {
            auto node = make_node<DeltaLayerNode>(in, d);
            node->save(x);
            node->save(W);
            node->keep({q, k, v, beta, v_old});
            node->scale = scale;
            torch::autograd::create_gradient_edge(out, node);
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// -------------------------------------------------------------------- sum rule
struct SumNode final : public OpNode {
    std::string name() const override { return "FastWeightSumBackward"; }
    variable_list apply(variable_list&& g) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        const auto t = unpack(user);
        const Tensor &Q = t[0], &K = t[1], &V = t[2];
        const Tensor gy = incoming(g[0], Q, {d.N, d.H, d.L, d.M});
        Tensor gQ = like_stream(d.E, Q), gK = like_stream(d.E, Q), gV = like_stream(d.M, Q);
        check_waits(fwp_causal_dot_backward(d.N, d.H, d.L, d.E, d.M, Desc(Q), Desc(K), Desc(V), Desc(gy), Desc(gQ), Desc(gK), Desc(gV),
                                            dtype_code(Q), stream_of(Q), Q.device().index()), "causal_dot_backward");
        return {gQ, gK, gV, Tensor()};
    }
};

PyObject* fast_weight_sum(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    std::array<const Tensor*, 4> in;
    if (n != 4 || !tensors(args, n, in)) return not_implemented();
    const Tensor &Q = *in[0], &K = *in[1], &V = *in[2], &W = *in[3];
    if (!first_stream(Q, true) || !V.defined() || V.dim() != 4) return not_implemented();
    const Dims d{Q.size(0), Q.size(1), Q.size(2), Q.size(3), V.size(3)};
    const auto ty = Q.scalar_type();
    const auto dev = Q.device();
    if (!shaped(K, ty, dev, d.N, d.H, d.L, d.E) || !shaped(V, ty, dev, d.N, d.H, d.L, d.M) ||
        !shaped(W, at::kFloat, dev, d.N, d.H, d.E, d.M))
        return not_implemented();
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        out = empty({d.N, d.H, d.L, d.M}, ty, Q);
        check_waits(fwp_causal_dot_product(d.N, d.H, d.L, d.E, d.M, Desc(Q), Desc(K), Desc(V), Desc(W), Desc(out), dtype_code(Q),
                                           stream_of(Q), dev.index()), "causal_dot_product");
        if (needs_grad(in)) {
            auto node = make_node<SumNode>(in, d);
            for (int i = 0; i < 3; i++) node->save(*in[i]);
            torch::autograd::create_gradient_edge(out, node);
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------ recurrent delta net
struct RecNode final : public OpNode {
    std::string name() const override { return "FastWeightRecUpdateTanhBackward"; }
    variable_list apply(variable_list&& g) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        const auto t = unpack(user), o = unpack(own);
        const Tensor *R = &t[0], &W = t[4], &out = t[5];
        const Tensor &q = o[0], &k = o[1], &v = o[2], &beta = o[3], &v_old = o[4], &h0 = o[5];
        const Tensor gy = incoming(g[0], out, {d.N, d.H, d.L, d.M});
        Tensor gq = empty(d, d.M, out), gk = empty(d, d.M, out), gv = empty(d, d.M, out), gb = empty(d, 1, out);
        Tensor gR[3];
        for (auto& x : gR) x = empty({1, d.H, d.M, d.M}, at::kFloat, out);
        Tensor grb = empty({1, d.H, 1, d.M}, at::kFloat, out);
        const int64_t nscratch = fwp_rec_update_fwm_tanh_scratch_floats(d.N, d.H, d.M);
        Tensor scratch = empty({nscratch}, at::kFloat, out);
        void* st = stream_of(out);
        const int dev = out.device().index();
        int rc = fwp_rec_update_fwm_tanh_backward_from_outputs(
            d.N, d.H, d.L, d.M, Desc(q), Desc(k), Desc(v), Desc(beta), Desc(v_old), Desc(out), Desc(h0), Desc(gy), Desc(R[0]), Desc(R[1]),
            Desc(R[2]), Desc(R[3]), Desc(W), Desc(gq), Desc(gk), Desc(gv), Desc(gb), Desc(gR[0]), Desc(gR[1]), Desc(gR[2]), Desc(grb),
            scratch.data_ptr<float>(), nscratch, FWP_F32, st, dev);
        if (rc == FWP_ERR_UNSUPPORTED) {
            Tensor delayed = empty(d, d.M, out);
            check(fwp_delayed(d.N, d.H, d.L, d.M, Desc(out), Desc(h0), Desc(Tensor()), Desc(delayed), 1, st, dev), "delayed");
            rc = fwp_rec_update_fwm_tanh_backward(
                d.N, d.H, d.L, d.M, Desc(q), Desc(k), Desc(v), Desc(beta), Desc(v_old), Desc(delayed), Desc(gy), Desc(R[0]), Desc(R[1]),
                Desc(R[2]), Desc(R[3]), Desc(W), Desc(gq), Desc(gk), Desc(gv), Desc(gb), Desc(gR[0]), Desc(gR[1]), Desc(gR[2]), Desc(grb),
                scratch.data_ptr<float>(), nscratch, FWP_F32, st, dev);
        }
        check(rc, "rec_update_fwm_tanh_backward");
        return {gq, gk, gv, gb, gR[0], gR[1], gR[2], grb, Tensor(), Tensor()};
    }
};

PyObject* rec_update_fwm_tanh(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    std::array<const Tensor*, 10> in;
    if (n != 10 || !tensors(args, n, in)) return not_implemented();
    const Tensor &qx = *in[0], &kx = *in[1], &vx = *in[2], &bx = *in[3], &W = *in[8], &h0 = *in[9];
    if (!first_stream(qx, false)) return not_implemented();
    const Dims d{qx.size(0), qx.size(1), qx.size(2), qx.size(3), qx.size(3)};
    const auto dev = qx.device();
    const auto f = at::kFloat;
    if (!shaped(kx, f, dev, d.N, d.H, d.L, d.M) || !shaped(vx, f, dev, d.N, d.H, d.L, d.M) || !shaped(bx, f, dev, d.N, d.H, d.L, 1) ||
        !shaped(W, f, dev, d.N, d.H, d.M, d.M) || !shaped(h0, f, dev, d.N, d.H, 1, d.M))
        return not_implemented();
    for (int i = 4; i < 8; i++)
        if (!shaped(*in[i], f, dev, 1, d.H, i < 7 ? d.M : 1, d.M) || !in[i]->is_contiguous()) return not_implemented();
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        const bool grad = needs_grad(in);
        out = empty(d, d.M, qx);
        Tensor q = empty(d, d.M, qx), k = empty(d, d.M, qx), v = empty(d, d.M, qx), beta = empty(d, 1, qx), v_old = empty(d, d.M, qx);
        Tensor h_init;
        if (grad) h_init = h0.detach().clone();
        check(fwp_rec_update_fwm_tanh_forward(d.N, d.H, d.L, d.M, Desc(qx), Desc(kx), Desc(vx), Desc(bx), Desc(*in[4]), Desc(*in[5]),
                                              Desc(*in[6]), Desc(*in[7]), Desc(q), Desc(k), Desc(v), Desc(beta), Desc(v_old), Desc(h0),
                                              Desc(W), Desc(out), FWP_F32, stream_of(qx), dev.index()), "rec_update_fwm_tanh_forward");
        if (grad) {
            auto node = make_node<RecNode>(in, d);
            torch::autograd::create_gradient_edge(out, node);
            for (int i = 4; i < 9; i++) node->save(*in[i]);
            node->save_output(out);
            node->keep({q, k, v, beta, v_old, h_init});
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------ delta RNN v1 and v2
template <int VERSION>
struct RnnNode final : public OpNode {
    std::string name() const override { return VERSION == 1 ? "FastRNNBackward" : "FastRNNv2Backward"; }
    variable_list apply(variable_list&& g) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        const auto t = unpack(user), o = unpack(own);
        const Tensor &K = t[0], &V = t[1], &beta = t[2], &W = t[3], &out = t[4], &v_old = o[0];
        const Tensor gy = incoming(g[0], out, {d.N, d.H, d.L, d.M});
        Tensor gZ = empty(d, d.M, out), gK = empty(d, d.M, out), gV = empty(d, d.M, out), gb = empty(d, 1, out);
        const Tensor& aux = o[1];     // v2: the normalised delayed outputs of the forward; v1: the start vector
        void* st = stream_of(out);
        const int dev = out.device().index();
        auto run = [&](auto backward, const Tensor& fed_back) {
            return backward(d.N, d.H, d.L, d.M, Desc(K), Desc(V), Desc(beta), Desc(v_old), Desc(gy), Desc(out), Desc(fed_back), Desc(W),
                            Desc(gZ), Desc(gK), Desc(gV), Desc(gb), FWP_F32, st, dev);
        };
        int rc = run(VERSION == 1 ? fwp_fast_rnn_backward_from_outputs : fwp_fast_rnn_v2_backward, aux);
        if (VERSION == 1 && rc == FWP_ERR_UNSUPPORTED) {
            Tensor delayed = empty(d, d.M, out);
            check(fwp_delayed(d.N, d.H, d.L, d.M, Desc(out), Desc(aux), Desc(Tensor()), Desc(delayed), 0, st, dev), "delayed");
            rc = run(fwp_fast_rnn_backward, delayed);
        }
        check(rc, VERSION == 1 ? "fast_rnn_backward" : "fast_rnn_v2_backward");
        return {gZ, gK, gV, Tensor(), gb, Tensor()};
    }
};

template <int VERSION>
PyObject* fast_rnn(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    std::array<const Tensor*, 6> in;
    if (n != 6 || !tensors(args, n, in)) return not_implemented();
    const Tensor &Z = *in[0], &K = *in[1], &V = *in[2], &W = *in[3], &beta = *in[4], &h0 = *in[5];
    if (!first_stream(Z, false)) return not_implemented();
    const Dims d{Z.size(0), Z.size(1), Z.size(2), Z.size(3), Z.size(3)};
    const auto dev = Z.device();
    const auto f = at::kFloat;
    if (!shaped(K, f, dev, d.N, d.H, d.L, d.M) || !shaped(V, f, dev, d.N, d.H, d.L, d.M) || !shaped(beta, f, dev, d.N, d.H, d.L, 1) ||
        !shaped(W, f, dev, d.N, d.H, d.M, d.M) || !shaped(h0, f, dev, d.N, d.H, 1, d.M))
        return not_implemented();
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        const bool grad = needs_grad(in);
        out = empty(d, d.M, Z);
        Tensor v_old = empty(d, d.M, Z), aux;
        void* st = stream_of(Z);
        if (VERSION == 1) {
            if (grad) aux = h0.detach().clone();
            check(fwp_fast_rnn_forward(d.N, d.H, d.L, d.M, Desc(Z), Desc(K), Desc(V), Desc(beta), Desc(v_old), Desc(h0), Desc(W),
                                       Desc(out), FWP_F32, st, dev.index()), "fast_rnn_forward");
        } else {
            aux = empty(d, d.M, Z);
            check(fwp_fast_rnn_v2_forward(d.N, d.H, d.L, d.M, Desc(Z), Desc(K), Desc(V), Desc(beta), Desc(v_old), Desc(h0), Desc(W),
                                          Desc(out), Desc(aux), FWP_F32, st, dev.index()), "fast_rnn_v2_forward");
        }
        if (grad) {
            auto node = make_node<RnnNode<VERSION>>(in, d);
            torch::autograd::create_gradient_edge(out, node);
            for (auto* t : {&K, &V, &beta, &W}) node->save(*t);
            node->save_output(out);
            node->keep({v_old, aux});
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------ delta LSTM v1 - v4
struct LstmNode final : public OpNode {
    int variant = 1;
    std::string name() const override {
        return variant == 1 ? "FastLSTMBackward" : "FastLSTMv" + std::to_string(variant) + "Backward";
    }
    variable_list apply(variable_list&& g) override {
        std::lock_guard<std::mutex> lock(mutex_);
        at::NoGradGuard no_grad;
        const auto t = unpack(user), o = unpack(own);       // K[3], V[3], beta[3], W[3], out, cell
        const Tensor &out = t[12], &cell = t[13];
        const Tensor *gates = &o[0], *v_old = &o[3];
        const Tensor gy = incoming(g[0], out, {d.N, d.H, d.L, d.M});        // the cell's gradient is ignored, as in the reference
        void* st = stream_of(out);
        const int dev = out.device().index();
        Tensor gZ[3], gK[3], gV[3], gb[3];
        for (int i = 0; i < 3; i++) {
            gZ[i] = empty(d, d.M, out);
            gK[i] = empty(d, d.M, out);
            gV[i] = empty(d, d.M, out);
            gb[i] = empty(d, 1, out);
        }
        auto run = [&](auto backward, const Tensor& fed_back, const Tensor& cells) {      // o[6]: h0 (v1) or the normalised delayed outputs
            return backward(variant, d.N, d.H, d.L, d.M, Desc(gy), Desc3(&t[0]), Desc3(&t[3]), Desc3(&t[6]), Desc3(v_old), Desc(out),
                            Desc(fed_back), Desc(cell), Desc(cells), Desc3(gates), Desc3(&t[9]), Desc3(gZ), Desc3(gK), Desc3(gV), Desc3(gb),
                            FWP_F32, st, dev);
        };
        int rc = run(fwp_fast_lstm_backward_from_outputs, o[6], o[7]);
        if (rc == FWP_ERR_UNSUPPORTED) {
            Tensor delayed = o[6], u_minus_c = empty(d, d.M, out);
            if (variant == 1) {
                delayed = empty(d, d.M, out);
                check(fwp_delayed(d.N, d.H, d.L, d.M, Desc(out), Desc(o[6]), Desc(Tensor()), Desc(delayed), 0, st, dev), "delayed");
            }
            check(fwp_delayed(d.N, d.H, d.L, d.M, Desc(cell), Desc(o[7]), Desc(gates[1]), Desc(u_minus_c), 0, st, dev), "delayed");
            rc = run(fwp_fast_lstm_backward, delayed, u_minus_c);
        }
        check(rc, "fast_lstm_backward");
        variable_list r;
        r.reserve(17);
        for (int i = 0; i < 3; i++)
            for (const Tensor& x : {gZ[i], gK[i], gV[i], gb[i], Tensor()}) r.push_back(x);
        r.resize(17);
        return r;
    }
};

template <int VARIANT>
PyObject* fast_lstm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    std::array<const Tensor*, 17> in;       // Z, K, V, beta, W of the input, update and output gates; h0, c0
    if (n != 17 || !tensors(args, n, in)) return not_implemented();
    const Tensor &h0 = *in[15], &c0 = *in[16], &x0 = *in[0];
    if (!first_stream(x0, false)) return not_implemented();
    const Dims d{x0.size(0), x0.size(1), x0.size(2), x0.size(3), x0.size(3)};
    const auto dev = x0.device();
    const auto f = at::kFloat;
    Tensor Z[3], K[3], V[3], B[3], W[3];
    for (int i = 0; i < 3; i++) {
        const Tensor* const* a = in.data() + 5 * i;
        if (!shaped(*a[0], f, dev, d.N, d.H, d.L, d.M) || !shaped(*a[1], f, dev, d.N, d.H, d.L, d.M) || !shaped(*a[2], f, dev, d.N, d.H, d.L, d.M) ||
            !shaped(*a[3], f, dev, d.N, d.H, d.L, 1) || !shaped(*a[4], f, dev, d.N, d.H, d.M, d.M))
            return not_implemented();
        Z[i] = *a[0]; K[i] = *a[1]; V[i] = *a[2]; B[i] = *a[3]; W[i] = *a[4];
    }
    if (!shaped(h0, f, dev, d.N, d.H, 1, d.M) || !shaped(c0, f, dev, d.N, d.H, 1, d.M)) return not_implemented();
    Tensor out, cell;
    {
        pybind11::gil_scoped_release no_gil;
        const bool grad = needs_grad(in);
        out = empty(d, d.M, x0);
        cell = empty(d, d.M, x0);
        Tensor gates[3], v_old[3], aux, c_init;
        for (auto& t : gates) t = empty(d, d.M, x0);
        for (auto& t : v_old) t = empty(d, d.M, x0);
        if (VARIANT != 1) aux = empty(d, d.M, x0);      // the normalised delayed outputs
        if (grad) c_init = c0.detach().clone();
        Tensor h_init;
        if (grad && VARIANT == 1) h_init = h0.detach().clone();
        check(fwp_fast_lstm_forward(VARIANT, d.N, d.H, d.L, d.M, Desc3(Z), Desc3(K), Desc3(V), Desc3(B), Desc(h0), Desc(c0), Desc3(W),
                                    Desc(out), Desc(aux), Desc(cell), Desc3(gates), Desc3(v_old), FWP_F32, stream_of(x0), dev.index()),
              "fast_lstm_forward");
        if (grad) {
            auto node = make_node<LstmNode>(in, d);
            node->variant = VARIANT;
            torch::autograd::create_gradient_edge(out, node);
            torch::autograd::create_gradient_edge(cell, node);
            for (int s = 1; s < 5; s++)
                for (int i = 0; i < 3; i++) node->save(*in[5 * i + s]);
            node->save_output(out);
            node->save_output(cell);
            node->keep({gates[0], gates[1], gates[2], v_old[0], v_old[1], v_old[2], VARIANT == 1 ? h_init : aux, c_init});
        }
    }
    PyObject* pair = PyTuple_New(2);
    if (!pair) return nullptr;
    PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::move(out)));
    PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::move(cell)));
    return pair;
    END_HANDLE_TH_ERRORS
}

PyObject* check_device_fault(PyObject*, PyObject* on) {
    g_check_fault = PyObject_IsTrue(on) == 1;
    Py_RETURN_NONE;
}

#define OP(name, f) {name, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    OP("fast_weight_delta", fast_weight_delta),
    OP("delta_attention", delta_attention),
    OP("fast_weight_sum", fast_weight_sum),
    OP("rec_update_fwm_tanh", rec_update_fwm_tanh),
    OP("fast_rnn", fast_rnn<1>),
    OP("fast_rnn_v2", fast_rnn<2>),
    OP("fast_lstm", fast_lstm<1>),
    OP("fast_lstm_v2", fast_lstm<2>),
    OP("fast_lstm_v3", fast_lstm<3>),
    OP("fast_lstm_v4", fast_lstm<4>),
    {"check_device_fault", check_device_fault, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_fwp_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fwp_torch(void) { return PyModule_Create(&module_def); }
