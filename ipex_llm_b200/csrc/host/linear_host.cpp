// linear_host.cpp -- the host side of one LowBitLinear.forward (reference low_bit_linear.py:638-725) in one native call:
// checks, output, scratch, stream and launch.  In Python (tensor views, a ctypes call of fourteen arguments, the scratch lookup) the
// same took 20 us around a 4 us kernel.  A CPython module (b200_host); the kernels are reached through the addresses of
// libb200lowbit.so's entry points, which the package hands over once.  Beside it, attention over the 8-bit cache (attention: the Python
// statements took 24 us around kernels of 5 to 17 us) and the look at a mixture's experts that every call of theirs begins with
// (expert_addresses).
#include <vector>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

namespace {

using MatmulFn = int (*)(const void*, int, int64_t, int64_t, const void*, int, int64_t, void*, int, const void*, int, void*, size_t, void*);
using WorkspaceFn = size_t (*)(int64_t, int64_t, int64_t, int);
using HintFn = void (*)(const void*, size_t);
using SdpFn = int (*)(const void*, int, const int64_t*, const void*, const int64_t*, const void*, const int64_t*, const void*, int, const int64_t*, int, float,
                      int, int, int, int, int, int, void*, int, void*, size_t, void*);
using SdpSupportedFn = int (*)(int, int, int, int);
using SdpWorkspaceFn = size_t (*)(int, int, int, int, int, int);
using SdpPromptFn = int (*)(const void*, int, const int64_t*, const void*, const int64_t*, const void*, const int64_t*, const void*, int, const int64_t*, int,
                            float, int, int, int, int, int, int, void*, int, const int64_t*, void*);
MatmulFn g_matmul = nullptr;
WorkspaceFn g_workspace = nullptr;
HintFn g_hint = nullptr;
SdpFn g_sdp = nullptr;
SdpSupportedFn g_sdp_supported = nullptr, g_sdp_prompt_supported = nullptr;
SdpWorkspaceFn g_sdp_workspace = nullptr;
SdpPromptFn g_sdp_prompt = nullptr;

// other threads run Python meanwhile: an allocation or a launch may have to wait for the device
struct WithoutGil {
    PyThreadState* const state = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

int dtype_code(c10::ScalarType t) {
    return t == at::kFloat ? 0 : t == at::kHalf ? 1 : t == at::kBFloat16 ? 2 : -1;
}

PyObject* attach(PyObject*, PyObject* args) {
    unsigned long long m, w, h, s, ss, sw, p, ps;
    if (!PyArg_ParseTuple(args, "KKKKKKKK", &m, &w, &h, &s, &ss, &sw, &p, &ps)) return nullptr;
    g_sdp = reinterpret_cast<SdpFn>(s);
    g_sdp_supported = reinterpret_cast<SdpSupportedFn>(ss);
    g_sdp_workspace = reinterpret_cast<SdpWorkspaceFn>(sw);
    g_sdp_prompt = reinterpret_cast<SdpPromptFn>(p);
    g_sdp_prompt_supported = reinterpret_cast<SdpSupportedFn>(ps);
    g_matmul = reinterpret_cast<MatmulFn>(m);
    g_workspace = reinterpret_cast<WorkspaceFn>(w);
    g_hint = reinterpret_cast<HintFn>(h);
    Py_RETURN_NONE;
}

// linear(x, weight, bias | None, out_features, in_features, qtype, max_rows_f32, next_weight | None)
//   -> the result; None when this call is not the plain case (the caller's general path then serves or refuses it); an int: the
//      native error code.  max_rows_f32: 32-bit activations of more rows are left to the caller (it casts them).
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 8 || !g_matmul) {
        PyErr_SetString(PyExc_TypeError, "b200_host.linear takes eight arguments, after attach()");
        return nullptr;
    }
    // exact tensors with storage only: subclasses, traced and batched tensors keep to the general path
    if (!THPVariable_CheckExact(a[0]) || !THPVariable_Check(a[1])) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(a[0]);
    const at::Tensor& w = THPVariable_Unpack(a[1]);
    if (!x.is_cuda() || !w.is_cuda() || !x.has_storage() || !w.has_storage() || x.dim() < 1 || x.device() != w.device() || !x.is_contiguous()) Py_RETURN_NONE;
    const int dt = dtype_code(x.scalar_type());
    const int64_t n = PyLong_AsLongLong(a[3]), k = PyLong_AsLongLong(a[4]);
    const int qtype = (int)PyLong_AsLong(a[5]);
    const int64_t max_f32 = PyLong_AsLongLong(a[6]);
    if (PyErr_Occurred()) return nullptr;
    if (dt < 0 || x.size(-1) != k || x.numel() == 0) Py_RETURN_NONE;
    const int64_t rows = x.numel() / k;
    if (dt == 0 && rows > max_f32) Py_RETURN_NONE;
    const void* xp = x.const_data_ptr();
    if (reinterpret_cast<uintptr_t>(xp) & 15) Py_RETURN_NONE;
    const void* bias = nullptr;
    if (a[2] != Py_None) {
        if (!THPVariable_Check(a[2])) Py_RETURN_NONE;
        const at::Tensor& b = THPVariable_Unpack(a[2]);
        if (b.scalar_type() != x.scalar_type() || b.device() != x.device() || !b.is_contiguous() || b.numel() != n) Py_RETURN_NONE;
        bias = b.const_data_ptr();
    }
    const void* next = nullptr;
    size_t next_bytes = 0;
    if (a[7] != Py_None && rows <= 32 && THPVariable_Check(a[7])) {
        const at::Tensor& nx = THPVariable_Unpack(a[7]);
        if (nx.is_cuda() && nx.has_storage()) { next = nx.const_data_ptr(); next_bytes = nx.nbytes(); }
    }
    at::Tensor y;
    int rc;
    {
        const WithoutGil released;
        const c10::cuda::CUDAGuard guard(x.device());
        auto sizes = x.sizes().vec();
        sizes.back() = n;
        const auto options = x.options().requires_grad(false);
        y = at::empty(sizes, options);
        at::Tensor scratch;
        const size_t need = g_workspace(n, k, rows, dt);
        if (need) scratch = at::empty({(int64_t)need}, options.dtype(at::kByte));
        if (next) g_hint(next, next_bytes);
        // a scratch of no bytes: any non-null pointer (NULL would ask the library for its own, under its lock)
        rc = g_matmul(w.const_data_ptr(), qtype, n, k, xp, dt, rows, y.mutable_data_ptr(), dt, bias, 0,
                      need ? scratch.mutable_data_ptr() : y.mutable_data_ptr(), need, c10::cuda::getCurrentCUDAStream(x.device().index()).stream());
    }
    if (rc) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// attention(query, key, value, causal, scale, prompts)
//   -> the result; None when this is not the plain case (dense rows, no mask, shapes that a kernel takes; with `prompts` false only
//      those of at most 32 new tokens): the caller's general path then serves or refuses it; an int: the native error code.
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 6 || !g_sdp) {
        PyErr_SetString(PyExc_TypeError, "b200_host.attention takes six arguments, after attach()");
        return nullptr;
    }
    if (!THPVariable_CheckExact(a[0]) || !THPVariable_CheckExact(a[1]) || !THPVariable_CheckExact(a[2])) Py_RETURN_NONE;
    const at::Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
    const int causal = PyObject_IsTrue(a[3]), prompts = PyObject_IsTrue(a[5]);
    const float scale = (float)PyFloat_AsDouble(a[4]);
    if (PyErr_Occurred()) return nullptr;
    for (const at::Tensor* t : {&q, &k, &v})
        if (!t->is_cuda() || !t->has_storage() || t->dim() != 4 || t->numel() == 0 || t->device() != q.device() || t->stride(3) != 1) Py_RETURN_NONE;
    const int dt = dtype_code(q.scalar_type());
    if (dt < 0 || k.scalar_type() != at::kByte || v.scalar_type() != at::kByte) Py_RETURN_NONE;
    const int64_t B = q.size(0), Hq = q.size(1), S = q.size(2), D = q.size(3), Hkv = k.size(1), L = k.size(2);
    if (k.size(0) != B || k.size(3) != D || v.sizes() != k.sizes()) Py_RETURN_NONE;
    for (const int64_t n : {B, Hq, S, L, B * Hq * S}) if (n > 0x7fffffff) Py_RETURN_NONE;
    const bool few = S <= 32 && g_sdp_supported((int)Hq, (int)Hkv, (int)S, (int)D);
    const void *const qp = q.const_data_ptr(), *const kp = k.const_data_ptr(), *const vp = v.const_data_ptr();
    const int64_t qs[3] = {q.stride(0), q.stride(1), q.stride(2)}, ks[3] = {k.stride(0), k.stride(1), k.stride(2)}, vs[3] = {v.stride(0), v.stride(1), v.stride(2)};
    if (!few) {
        const auto at16 = [](const void* p, const int64_t (&s)[3], int64_t unit) {
            return ((reinterpret_cast<uintptr_t>(p) & 15) | (uintptr_t)((s[0] | s[1] | s[2]) & (unit - 1))) == 0;
        };
        if (!prompts || dt == 0 || L < S || !g_sdp_prompt_supported((int)Hq, (int)Hkv, (int)D, dt) || !at16(kp, ks, 16) || !at16(vp, vs, 16) || !at16(qp, qs, 8))
            Py_RETURN_NONE;
    }
    at::Tensor out;
    int rc;
    {
        const WithoutGil released;
        const c10::cuda::CUDAGuard guard(q.device());
        const auto options = q.options().requires_grad(false);
        void* const stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
        if (few) {
            out = at::empty({B, Hq, S, D}, options);
            const size_t need = g_sdp_workspace((int)B, (int)Hq, (int)Hkv, (int)S, (int)L, (int)D);
            at::Tensor scratch = at::empty({(int64_t)need}, options.dtype(at::kByte));
            rc = g_sdp(qp, dt, qs, kp, ks, vp, vs, nullptr, 0, nullptr, causal, scale, (int)B, (int)Hq, (int)Hkv, (int)S, (int)L, (int)D, out.mutable_data_ptr(), dt,
                       scratch.mutable_data_ptr(), need, stream);
        } else {
            out = at::empty({B, S, Hq, D}, options).transpose(1, 2);
            const int64_t os[3] = {out.stride(0), out.stride(1), out.stride(2)};
            rc = g_sdp_prompt(qp, dt, qs, kp, ks, vp, vs, nullptr, 0, nullptr, causal, scale, (int)B, (int)Hq, (int)Hkv, (int)S, (int)L, (int)D,
                              out.mutable_data_ptr(), dt, os, stream);
        }
    }
    if (rc) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ---- the experts of a mixture: one walk over their modules for a call, however many there are
struct Name {                                       // an interned attribute name
    PyObject* const o;
    explicit Name(const char* s) : o(PyUnicode_InternFromString(s)) {}
};
// an attribute in the instance's own dictionary, borrowed; NULL when it is not there
PyObject* own(PyObject* dict, const Name& name) { return PyDict_GetItemWithError(dict, name.o); }
bool is_number(PyObject* v, long want) { return v && PyLong_Check(v) && PyLong_AsLong(v) == want; }

// whether nothing about `module` asks for its own forward: class, hooks, format, sizes; *address: its weight
bool plain_linear(PyObject* module, PyObject* cls, long qtype, long in_features, long out_features, long device, int64_t* address) {
    static const Name forward("forward"), hooks("_forward_hooks"), pre("_forward_pre_hooks"), mp("mp_group"), order("act_order"), head("optimize_lm_head"),
        training("training"), type("qtype"), in("in_len"), out("out_len"), params("_parameters"), weight("weight"), bias("bias"), quantized("quantized");
    if ((PyObject*)Py_TYPE(module) != cls) return false;
    PyObject* const d = PyObject_GenericGetDict(module, nullptr);
    if (!d) return false;
    bool ok = false;
    do {
        if (own(d, forward) || own(d, mp) != Py_None || own(d, order) != Py_False || own(d, head) != Py_False || own(d, training) != Py_False) break;
        PyObject *const fh = own(d, hooks), *const ph = own(d, pre);
        if (!fh || !ph || PyObject_Size(fh) != 0 || PyObject_Size(ph) != 0) break;
        if (!is_number(own(d, type), qtype) || !is_number(own(d, in), in_features) || !is_number(own(d, out), out_features)) break;
        PyObject* const p = own(d, params);
        if (!p || !PyDict_Check(p)) break;
        PyObject *const w = PyDict_GetItemWithError(p, weight.o), *const b = PyDict_GetItemWithError(p, bias.o);
        if (!w || b != Py_None || !THPVariable_Check(w)) break;
        const at::Tensor& t = THPVariable_Unpack(w);
        if (!t.has_storage() || !t.is_contiguous() || (device < 0 ? !t.is_cpu() : !t.is_cuda() || t.device().index() != device)) break;
        PyObject* const q = PyObject_GetAttr(w, quantized.o);
        Py_XDECREF(q);
        if (q != Py_True) break;
        *address = reinterpret_cast<int64_t>(t.const_data_ptr());
        ok = (*address & 15) == 0;
    } while (false);
    Py_DECREF(d);
    return ok;
}

// expert_addresses(class, qtype, hidden, inter, device index | -1 (CPU), gates, ups, downs: the module lists' dictionaries)
//   -> the weights' addresses, gates first, as bytes of 64-bit numbers; None when any of the modules has to run itself
PyObject* expert_addresses(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 8 || !PyDict_Check(a[5]) || !PyDict_Check(a[6]) || !PyDict_Check(a[7])) {
        PyErr_SetString(PyExc_TypeError, "b200_host.expert_addresses takes a class, four numbers and three dictionaries");
        return nullptr;
    }
    const long qtype = PyLong_AsLong(a[1]), hidden = PyLong_AsLong(a[2]), inter = PyLong_AsLong(a[3]), device = PyLong_AsLong(a[4]);
    if (PyErr_Occurred()) return nullptr;
    std::vector<int64_t> out;
    for (int i = 0; i < 3; i++) {
        PyObject *key, *module;
        Py_ssize_t pos = 0;
        while (PyDict_Next(a[5 + i], &pos, &key, &module)) {
            int64_t address = 0;
            if (!plain_linear(module, a[0], qtype, i < 2 ? hidden : inter, i < 2 ? inter : hidden, device, &address)) {
                PyErr_Clear();
                Py_RETURN_NONE;
            }
            out.push_back(address);
        }
    }
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(out.data()), (Py_ssize_t)(out.size() * sizeof(int64_t)));
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"attach", attach, METH_VARARGS, nullptr},
                         {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(attention)), METH_FASTCALL, nullptr},
                         {"expert_addresses", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(expert_addresses)), METH_FASTCALL, nullptr},
                         {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear)), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "b200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b200_host() { return PyModule_Create(&module); }
