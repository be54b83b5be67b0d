// The package's per-call functions (api.py) as plain CPython functions with positional arguments.
// A decode step or a short prompt lasts a few microseconds on the GPU, so the host path is what such a call
// costs: filling the C structs through ctypes took 25 - 35 us a call, and the keyword dispatch of the pybind
// functions takes 0.2 (norm, prefill) to 1.2 (recurrent_forward: 4.2 us as it is here, 4.5 through api.py, 5.5).  Here an argument is a pointer check, and the work below is namespace gdn_cuda's.
// That work runs without the interpreter lock: a launch waits while the stream's queue is full, and other Python threads
// must not wait with it.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include "gdn_api.hpp"

namespace {

void require(bool cond, const char* msg) {
    if (!cond) throw std::runtime_error(msg);
}

at::Tensor tensor(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) throw std::runtime_error(std::string(name) + " must be a torch.Tensor");
    return THPVariable_Unpack(o);
}
std::optional<at::Tensor> optional_tensor(PyObject* o, const char* name) {
    if (o == Py_None) return std::nullopt;
    return tensor(o, name);
}
bool truth(PyObject* o) {
    const int r = PyObject_IsTrue(o);
    if (r < 0) throw python_error();
    return r != 0;
}
long integer(PyObject* o) {  // whatever int() takes
    THPObjectPtr converted;
    if (!PyLong_Check(o)) {
        converted = PyNumber_Long(o);
        if (!converted) throw python_error();
        o = converted.get();
    }
    const long r = PyLong_AsLong(o);
    if (r == -1 && PyErr_Occurred()) throw python_error();
    return r;
}
double real(PyObject* o) {
    const double r = PyFloat_AsDouble(o);
    if (r == -1.0 && PyErr_Occurred()) throw python_error();
    return r;
}
std::optional<float> optional_real(PyObject* o) {
    if (o == Py_None) return std::nullopt;
    return static_cast<float>(real(o));
}
PyObject* pair(const at::Tensor& a, const at::Tensor& b) {
    PyObject* t = PyTuple_New(2);
    if (!t) throw python_error();
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(a));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(b));
    return t;
}

// Every call runs on the device of its first tensor and on that device's current torch stream.
struct OnDevice {
    c10::cuda::OptionalCUDAGuard guard;
    OnDevice(const at::Tensor& t, const char* name) {
        if (!t.is_cuda()) throw std::runtime_error(std::string(name) + " must be a CUDA tensor");
        guard.set_device(t.device());
    }
    cudaStream_t stream() const { return at::cuda::getCurrentCUDAStream().stream(); }
};

// `work()` without the interpreter lock (an exception takes it back on its way out).
template <typename F>
auto unlocked(F&& work) {
    pybind11::gil_scoped_release release;
    return work();
}

// query, key, value, initial_state, beta, gate, cu_seqlens, num_accepted_tokens, inference_mode, is_qk_norm, scale,
// inplace_state, gating, state_indices
PyObject* recurrent_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    require(n == 14, "recurrent_forward takes 14 positional arguments");
    at::Tensor q = tensor(a[0], "query"), k = tensor(a[1], "key"), v = tensor(a[2], "value");
    auto state = optional_tensor(a[3], "initial_state");
    auto beta = optional_tensor(a[4], "beta"), gate = optional_tensor(a[5], "gate");
    auto cu = optional_tensor(a[6], "cu_seqlens"), accepted = optional_tensor(a[7], "num_accepted_tokens");
    std::optional<std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor>> gating;
    if (a[12] != Py_None) {
        THPObjectPtr seq(PySequence_Fast(a[12], "gating is (A_log, dt_bias, a, b)"));
        if (!seq) throw python_error();
        require(PySequence_Fast_GET_SIZE(seq.get()) == 4, "gating is (A_log, dt_bias, a, b)");
        PyObject** g = PySequence_Fast_ITEMS(seq.get());
        gating.emplace(tensor(g[0], "A_log"), tensor(g[1], "dt_bias"), tensor(g[2], "a"), tensor(g[3], "b"));
    }
    gdn_cuda::RecurrentExtensions ext;
    ext.inplace_state = truth(a[11]);
    ext.state_indices = optional_tensor(a[13], "state_indices");
    const auto mode = static_cast<gdn_cuda::InferenceMode>(integer(a[8]));
    const bool norm = truth(a[9]);
    const auto scale = optional_real(a[10]);
    OnDevice dev(q, "query");
    const auto r = unlocked([&] {
        return gdn_cuda::recurrent_forward_ext(q, k, v, state, beta, gate, gating, cu, accepted, mode, dev.stream(), norm, scale, ext);
    });
    return pair(r.first, r.second);
    END_HANDLE_TH_ERRORS
}

// query, key, value, beta, gate, scale, initial_state, cu_seqlens, chunk_indices, cu_chunks, total_chunks, is_qk_norm, workspace
PyObject* chunked_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    require(n == 13, "chunked_forward takes 13 positional arguments");
    at::Tensor q = tensor(a[0], "query"), k = tensor(a[1], "key"), v = tensor(a[2], "value"), beta = tensor(a[3], "beta");
    auto gate = optional_tensor(a[4], "gate"), state = optional_tensor(a[6], "initial_state");
    auto cu = optional_tensor(a[7], "cu_seqlens"), ci = optional_tensor(a[8], "chunk_indices"), cc = optional_tensor(a[9], "cu_chunks");
    std::optional<int> chunks;
    if (a[10] != Py_None) chunks = static_cast<int>(integer(a[10]));
    auto workspace = optional_tensor(a[12], "workspace");
    const auto scale = optional_real(a[5]);
    const bool norm = truth(a[11]);
    OnDevice dev(q, "query");
    const auto r = unlocked([&] {
        return gdn_cuda::chunked_forward_ext(q, k, v, beta, gate, scale, state, cu, ci, cc, chunks, dev.stream(), norm, workspace);
    });
    return pair(r.first, r.second);
    END_HANDLE_TH_ERRORS
}

// A_log, dt_bias, a, b
PyObject* fused_gdn_gating(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    require(n == 4, "fused_gdn_gating takes 4 positional arguments");
    at::Tensor A = tensor(a[0], "A_log"), dt = tensor(a[1], "dt_bias"), x = tensor(a[2], "a"), b = tensor(a[3], "b");
    OnDevice dev(x, "a");
    const auto r = unlocked([&] { return gdn_cuda::fused_gdn_gating(A, dt, x, b, false, dev.stream()); });
    return pair(r.first, r.second);
    END_HANDLE_TH_ERRORS
}

// x, weight, bias, initial_state, cu_seqlens, activation, final_state, return_final_state
PyObject* causal_conv1d(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    require(n == 8, "causal_conv1d takes 8 positional arguments");
    at::Tensor x = tensor(a[0], "x"), w = tensor(a[1], "weight");
    auto bias = optional_tensor(a[2], "bias"), s_in = optional_tensor(a[3], "initial_state"), cu = optional_tensor(a[4], "cu_seqlens");
    auto s_out = optional_tensor(a[6], "final_state");
    const bool silu = truth(a[5]), want_state = truth(a[7]);
    OnDevice dev(x, "x");
    const auto r = unlocked([&] { return gdn_cuda::causal_conv1d(x, w, bias, s_in, cu, silu, s_out, want_state, dev.stream()); });
    return r.second.has_value() ? pair(r.first, *r.second) : THPVariable_Wrap(r.first);
    END_HANDLE_TH_ERRORS
}

// x, z, weight, eps
PyObject* gated_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    require(n == 4, "gated_rmsnorm takes 4 positional arguments");
    at::Tensor x = tensor(a[0], "x"), z = tensor(a[1], "z"), w = tensor(a[2], "weight");
    const float eps = static_cast<float>(real(a[3]));
    OnDevice dev(x, "x");
    return THPVariable_Wrap(unlocked([&] { return gdn_cuda::gated_rmsnorm(x, z, w, eps, dev.stream()); }));
    END_HANDLE_TH_ERRORS
}

#define GDN_FAST(name) \
    { "_fast_" #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&name)), METH_FASTCALL, "positional form of " #name }
PyMethodDef kMethods[] = {GDN_FAST(recurrent_forward), GDN_FAST(chunked_forward), GDN_FAST(fused_gdn_gating),
                          GDN_FAST(causal_conv1d),     GDN_FAST(gated_rmsnorm),   {nullptr, nullptr, 0, nullptr}};

}  // namespace

void add_fastcall_functions(PyObject* module) {
    if (PyModule_AddFunctions(module, kMethods) != 0) throw python_error();
}
