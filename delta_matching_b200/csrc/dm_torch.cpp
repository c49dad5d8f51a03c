// The eager route of the public API as one native call: argument check, allocation, the library's composite entry points and
// the autograd node, without an interpreter in between.  At the small shapes the whole step is bound by this path: in Python
// (a rule table, ctypes, torch.empty per buffer, an autograd.Function) it took 275 us per forward + backward of any small shape,
// against about 60 us of kernels for one short sequence.
//
// The module has no link-time dependency on libdm_b200.so: `bind` receives the entry points' addresses from the Python loader
// (_lib.py), so whatever library that loader picked is the one used here.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <cmath>

#include "../../include/dm_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

decltype(&dm_attn_forward) g_forward = nullptr;
decltype(&dm_attn_backward) g_backward = nullptr;
decltype(&dm_bwd_workspace_bytes) g_ws_bytes = nullptr;
PyObject* g_split_module = nullptr;      // delta_matching_b200.split: the DM_BWD_* knobs and the per-head-group backward
std::atomic<int64_t> g_forward_calls{0}, g_backward_calls{0};

PyObject *g_str_groups, *g_str_limit, *g_str_auto, *g_str_heads, *g_str_backward;

constexpr int64_t kAlign = 256;      // of the pieces of a packed buffer: TMA bases need 16 bytes
inline int64_t up(int64_t n) { return (n + kAlign - 1) / kAlign * kAlign; }

struct Dims {
    int64_t B, H, Hk, N, D;
    bool causal, matched;
    DmShape shape() const { return DmShape{(int32_t)B, (int32_t)H, (int32_t)Hk, (int32_t)N, (int32_t)D, causal ? 1 : 0}; }
    int64_t rq() const { return D >= 256 ? 64 : 128; }
    int64_t rk() const { return D >= 256 ? 32 : 64; }
};

// What the backward needs of the forward, packed into one buffer: the codes, their scales and the LSE.
struct Saved {
    int64_t q8, k8, v8, q8s, k8s, v8s, lse, bytes;
    explicit Saved(const Dims& d) {
        const int64_t qn = d.B * d.H * d.N, kn = d.B * d.Hk * d.N;
        q8 = 0;
        k8 = q8 + up(qn * d.D);
        v8 = k8 + up(kn * d.D);
        q8s = v8 + up(kn * d.D);
        k8s = q8s + up(qn / d.rq() * 4);
        v8s = k8s + up(kn / d.rk() * 4);
        lse = v8s + up(kn / d.rk() * 4);
        bytes = lse + up(qn * 4);
    }
};

inline Tensor empty(at::IntArrayRef sizes, c10::ScalarType dt, c10::Device dev) {
    return Tensor(at::detail::empty_cuda(sizes, dt, dev, std::nullopt));
}
inline char* ptr(const Tensor& t) { return static_cast<char*>(t.data_ptr()); }
inline float* f32(char* p) { return reinterpret_cast<float*>(p); }

inline DmStrides strides_bnhd(const Tensor& t, bool head_major) {
    return DmStrides{t.stride(0), t.stride(head_major ? 2 : 1), t.stride(head_major ? 1 : 2)};
}
// The kernels read rows with a unit lane stride.
inline Tensor unit_lane(const Tensor& t) { return t.stride(3) == 1 ? t : t.contiguous(); }

inline void check(int rc, const char* name, const char* err) {
    if (rc != 0) throw std::runtime_error(std::string("delta_matching_b200.") + name + ": " + err + " (code " + std::to_string(rc) + ")");
}

// O (B, N, H, D) and the packed buffer.
Tensor run_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Dims& d, bool head_major, Tensor* packed_out) {
    const c10::Device dev = q_.device();
    const c10::cuda::CUDAGuard guard(dev);
    const Tensor q = unit_lane(q_), k = unit_lane(k_), v = unit_lane(v_);
    const Saved s(d);
    const int64_t km = up(d.B * d.Hk * d.D * 4), part = up(d.B * d.Hk * (d.N / 64) * d.D * 4);
    Tensor o = empty({d.B, d.N, d.H, d.D}, at::kBFloat16, dev);
    Tensor packed = empty({s.bytes}, at::kByte, dev);
    Tensor scratch = empty({km + part}, at::kByte, dev);
    char *p = ptr(packed), *t = ptr(scratch);
    char err[512] = "";
    g_forward_calls.fetch_add(1, std::memory_order_relaxed);
    check(g_forward(q.data_ptr(), strides_bnhd(q, head_major), k.data_ptr(), strides_bnhd(k, head_major), v.data_ptr(),
                    strides_bnhd(v, head_major), d.shape(), p + s.q8, f32(p + s.q8s), p + s.k8, f32(p + s.k8s), p + s.v8, f32(p + s.v8s),
                    f32(t), f32(t + km), o.data_ptr(), f32(p + s.lse), at::cuda::getCurrentCUDAStream(dev.index()).stream(), err, sizeof err),
          "dm_attn_forward", err);
    if (packed_out) *packed_out = std::move(packed);
    return o;
}

// dq (B, N, H, D), dk, dv (B, N, Hk, D); dO has a unit lane stride.
variable_list run_backward(const Tensor& dO, const Tensor& o, const Tensor& packed, const Dims& d) {
    const c10::Device dev = packed.device();
    const c10::cuda::CUDAGuard guard(dev);
    const Saved s(d);
    const int64_t qn = d.B * d.H * d.N;
    size_t ds_bytes = 0, psi_bytes = 0;
    check(g_ws_bytes(d.shape(), (int32_t)d.H, &ds_bytes, &psi_bytes), "dm_bwd_workspace_bytes", "failed");
    const bool gqa = d.Hk < d.H;
    // the intermediates in one buffer
    const int64_t do8 = 0, ds = do8 + up(qn * d.D), psi = ds + up((int64_t)ds_bytes), do8s = psi + up((int64_t)psi_bytes),
                  delta = do8s + up(qn / d.rq() * 4), dkh = delta + up(qn * 4), dvh = dkh + (gqa ? up(qn * d.D * 2) : 0),
                  bytes = dvh + (gqa ? up(qn * d.D * 2) : 0);
    Tensor scratch = empty({bytes}, at::kByte, dev);
    Tensor dq = empty({d.B, d.N, d.H, d.D}, at::kBFloat16, dev);
    Tensor dk = empty({d.B, d.N, d.Hk, d.D}, at::kBFloat16, dev);
    Tensor dv = empty({d.B, d.N, d.Hk, d.D}, at::kBFloat16, dev);
    char *p = ptr(packed), *t = ptr(scratch);
    char err[512] = "";
    const DmStrides os = d.matched ? DmStrides{0, 0, 0} : strides_bnhd(o, false);
    g_backward_calls.fetch_add(1, std::memory_order_relaxed);
    check(g_backward(dO.data_ptr(), strides_bnhd(dO, false), d.matched ? nullptr : o.data_ptr(), os, p + s.q8, p + s.k8, p + s.v8,
                     f32(p + s.q8s), f32(p + s.k8s), f32(p + s.v8s), f32(p + s.lse), d.shape(), d.matched ? 1 : 0, t + do8, f32(t + do8s),
                     f32(t + delta), gqa ? t + dkh : nullptr, gqa ? t + dvh : nullptr, t + ds, f32(t + psi), dq.data_ptr(), dk.data_ptr(),
                     dv.data_ptr(), at::cuda::getCurrentCUDAStream(dev.index()).stream(), err, sizeof err),
          "dm_attn_backward", err);
    return {dq, dk, dv};
}

// The backward in head groups (long context): the Python driver in split.py, whose host time is hidden by its kernels.
variable_list run_split_backward(const Tensor& dO, const Tensor& o, const Tensor& packed, const Dims& d) {
    const Saved s(d);
    const int64_t qn = d.B * d.H, kn = d.B * d.Hk;
    auto piece = [&](int64_t off, at::IntArrayRef sizes, c10::ScalarType dt) {
        int64_t n = 1;
        for (const int64_t v : sizes) n *= v;
        return packed.narrow(0, off, n * (int64_t)c10::elementSize(dt)).view(dt).view(sizes);
    };
    const Tensor in[] = {dO, o, piece(s.lse, {qn, d.N}, at::kFloat),
                         piece(s.q8, {qn, d.N, d.D}, at::kFloat8_e4m3fn), piece(s.q8s, {qn, d.N / d.rq()}, at::kFloat),
                         piece(s.k8, {kn, d.N, d.D}, at::kFloat8_e4m3fn), piece(s.k8s, {kn, d.N / d.rk()}, at::kFloat),
                         piece(s.v8, {kn, d.N, d.D}, at::kFloat8_e4m3fn), piece(s.v8s, {kn, d.N / d.rk()}, at::kFloat)};
    const PyGILState_STATE gil = PyGILState_Ensure();
    variable_list out;
    PyObject* args = PyTuple_New(14);
    for (int i = 0; i < 9; ++i) {
        PyObject* t = in[i].defined() ? THPVariable_Wrap(in[i]) : Py_NewRef(Py_None);
        PyTuple_SET_ITEM(args, i, t);
    }
    const int64_t ints[] = {d.B, d.H, d.Hk};
    for (int i = 0; i < 3; ++i) PyTuple_SET_ITEM(args, 9 + i, PyLong_FromLongLong(ints[i]));
    PyTuple_SET_ITEM(args, 12, PyBool_FromLong(d.causal));
    PyTuple_SET_ITEM(args, 13, PyBool_FromLong(d.matched));
    PyObject* fn = PyObject_GetAttr(g_split_module, g_str_backward);
    PyObject* r = fn ? PyObject_CallObject(fn, args) : nullptr;
    Py_XDECREF(fn);
    Py_DECREF(args);
    if (r && PyTuple_Check(r) && PyTuple_GET_SIZE(r) == 3)
        for (int i = 0; i < 3; ++i) out.push_back(THPVariable_Unpack(PyTuple_GET_ITEM(r, i)));
    Py_XDECREF(r);
    if (out.size() != 3) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "delta_matching_b200.split: the backward did not return dq, dk, dv");
        python_error e;
        e.persist();                    // keeps the Python exception's type across the autograd engine's threads
        PyGILState_Release(gil);
        throw e;
    }
    PyGILState_Release(gil);
    return out;
}

struct DMAttention : public torch::autograd::Function<DMAttention> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Dims& d, bool head_major, bool split) {
        Tensor packed;
        Tensor o = run_forward(q, k, v, d, head_major, &packed);
        // O takes part in the backward only through the stale delta
        ctx->save_for_backward({packed, d.matched ? Tensor() : o});
        auto& m = ctx->saved_data;
        m["d"] = c10::IValue(std::vector<int64_t>{d.B, d.H, d.Hk, d.N, d.D, d.causal, d.matched, head_major, split});
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const auto m = ctx->saved_data["d"].toIntVector();
        const Dims d{m[0], m[1], m[2], m[3], m[4], m[5] != 0, m[6] != 0};
        const bool head_major = m[7] != 0, split = m[8] != 0;
        const Tensor dO = unit_lane(grads[0]);      // e.g. the expanded gradient of o.sum()
        variable_list g;
        {
            at::AutoGradMode no_grad(false);
            g = split ? run_split_backward(dO, saved[1], saved[0], d) : run_backward(dO, saved[1], saved[0], d);
            if (head_major)
                for (auto& t : g) t = t.transpose(1, 2);
        }
        if (at::GradMode::is_enabled() && grads[0].requires_grad()) {
            // the kernels are not differentiable themselves: a second differentiation is an error, not a silent zero
            auto err = std::make_shared<torch::autograd::Error>("delta_matching: the attention backward cannot be differentiated twice",
                                                                torch::autograd::collect_next_edges(grads[0]));
            for (auto& t : g) {
                t = t.detach();
                torch::autograd::set_history(t, err);
            }
        }
        g.resize(6);
        return g;
    }
};

// attn(q, k, v, causal, softmax_scale, matched, head_major): the output, or None when the call breaks a rule of the input
// contract (core._check_inputs then raises the rule's own exception).
PyObject* attn(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 7) {
        PyErr_SetString(PyExc_TypeError, "attn takes 7 arguments");
        return nullptr;
    }
    for (int i = 0; i < 3; ++i)
        if (!THPVariable_Check(a[i])) Py_RETURN_NONE;
    const Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
    const int causal = PyObject_IsTrue(a[3]), head_major = a[6] == Py_True;
    if (causal < 0) return nullptr;
    const bool matched = a[5] == Py_True;
    for (const Tensor* t : {&q, &k, &v})
        if (t->dim() != 4 || !t->is_cuda() || t->layout() != at::kStrided || t->scalar_type() != at::kBFloat16 || t->device() != q.device())
            Py_RETURN_NONE;
    const int hd = head_major ? 1 : 2, nd = head_major ? 2 : 1;
    const Dims d{q.size(0), q.size(hd), k.size(hd), q.size(nd), q.size(3), causal != 0, matched};
    if ((matched && !causal) || k.sizes() != v.sizes() || k.size(0) != d.B || k.size(3) != d.D || k.size(nd) != d.N || d.Hk == 0 ||
        d.H == 0 || d.H % d.Hk || (d.D != 128 && d.D != 256) || d.N == 0 || d.N % (d.D == 128 ? 256 : 128) || d.B == 0 || d.B * d.H > 65535)
        Py_RETURN_NONE;
    if (a[4] != Py_None) {
        const double scale = PyFloat_AsDouble(a[4]);
        if (scale == -1.0 && PyErr_Occurred()) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        if (!(std::fabs(scale - 1.0 / std::sqrt((double)d.D)) <= 1e-12)) Py_RETURN_NONE;
    }
    const cudaDeviceProp* prop = at::cuda::getDeviceProperties(q.device().index());
    if (prop->major != 10 || prop->minor != 0) Py_RETURN_NONE;

    const bool train = at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
    bool split = false;
    if (train) {
        // the knobs are module attributes: "auto" within the limit is the common case, anything else is split.py's rule
        PyObject* groups = PyObject_GetAttr(g_split_module, g_str_groups);
        PyObject* limit = PyObject_GetAttr(g_split_module, g_str_limit);
        if (!groups || !limit) {
            Py_XDECREF(groups);
            Py_XDECREF(limit);
            return nullptr;
        }
        const bool is_auto = groups == g_str_auto || (PyUnicode_Check(groups) && PyUnicode_Compare(groups, g_str_auto) == 0);
        const double lim = PyFloat_AsDouble(limit);
        Py_DECREF(groups);
        Py_DECREF(limit);
        if (lim == -1.0 && PyErr_Occurred()) return nullptr;
        if (!is_auto || (double)d.B * d.H * d.N * d.N > lim) {
            PyObject* fn = PyObject_GetAttr(g_split_module, g_str_heads);
            PyObject* r = fn ? PyObject_CallFunction(fn, "LLLLL", (long long)d.B, (long long)d.H, (long long)d.Hk, (long long)(d.H / d.Hk), (long long)d.N)
                             : nullptr;
            Py_XDECREF(fn);
            if (!r) return nullptr;
            split = PyLong_AsLongLong(r) < d.H;
            Py_DECREF(r);
        }
    }
    Tensor o;
    {
        pybind11::gil_scoped_release no_gil;
        o = train ? DMAttention::apply(q, k, v, d, head_major != 0, split) : run_forward(q, k, v, d, head_major != 0, nullptr);
    }
    return THPVariable_Wrap(std::move(o));
    END_HANDLE_TH_ERRORS
}

// bind({name: address}, split module)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    if (nargs != 2 || !PyDict_Check(a[0])) {
        PyErr_SetString(PyExc_TypeError, "bind(addresses, split_module)");
        return nullptr;
    }
    auto addr = [&](const char* name) -> void* {
        PyObject* v = PyDict_GetItemString(a[0], name);
        return v ? PyLong_AsVoidPtr(v) : nullptr;
    };
    g_forward = reinterpret_cast<decltype(g_forward)>(addr("dm_attn_forward"));
    g_backward = reinterpret_cast<decltype(g_backward)>(addr("dm_attn_backward"));
    g_ws_bytes = reinterpret_cast<decltype(g_ws_bytes)>(addr("dm_bwd_workspace_bytes"));
    if (PyErr_Occurred()) return nullptr;
    if (!g_forward || !g_backward || !g_ws_bytes) {
        PyErr_SetString(PyExc_RuntimeError, "delta_matching_b200: bind is missing an entry point");
        return nullptr;
    }
    Py_XSETREF(g_split_module, Py_NewRef(a[1]));
    Py_RETURN_NONE;
}

// Calls of the two composite entry points since the module was loaded.
PyObject* call_counts(PyObject*, PyObject*) {
    return Py_BuildValue("LL", (long long)g_forward_calls.load(), (long long)g_backward_calls.load());
}

PyMethodDef kMethods[] = {{"attn", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(attn)), METH_FASTCALL, "the eager attention call"},
                          {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, "set the library's entry points"},
                          {"call_counts", call_counts, METH_NOARGS, "(forward, backward) calls so far"},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_dm_torch", "native eager route", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dm_torch(void) {
    g_str_groups = PyUnicode_InternFromString("_BWD_GROUPS");
    g_str_limit = PyUnicode_InternFromString("_BWD_WS_LIMIT");
    g_str_auto = PyUnicode_InternFromString("auto");
    g_str_heads = PyUnicode_InternFromString("_bwd_heads_per_call");
    g_str_backward = PyUnicode_InternFromString("split_backward");
    return PyModule_Create(&kModule);
}
