// The host side of the small calls: a quantized linear or an expert on tensors, from the Python call to the library's
// launches.  What a call of one row costs is this path (the kernels run 5-20 us): through ctypes it was 20-33 us -- struct
// and pointer objects for some twenty arguments, seven data_ptr() calls, three tensor methods -- and here it is the
// allocation of the result and the launches (4-bit 1024 x 4096, one row: 21.7 us per call before, 6.5 now, which is the
// kernel's own time).
//
// Every function returns None where it does not cover the arguments (another device, dtype conversions, a layer that has to
// be validated first, an error from the library); the Python code around it then takes the general way and raises what
// there is to raise.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>

#include <ATen/Functions.h>
#include <ATen/core/Tensor.h>
#include <c10/core/InferenceMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/hqq_moe.h"

namespace {

struct Names {
    PyObject *dict, *W_q, *meta, *bias, *plan, *desc, *ready, *expert, *scale_q, *zero_q, *meta_scale, *meta_zero, *scale, *zero, *modules, *w1, *w2, *w3, *axis;
} N;

PyObject* g_scratch = nullptr;        // custom_layers._SCRATCH: {("cuda", index): uint8 tensor}
PyObject* g_grow = nullptr;           // custom_layers._scratch(device, bytes)
PyObject* g_keys[64];                 // ("cuda", index)

// A layer's descriptor (and with it the addresses it was made from) and the workspace of its last row count, as linear
// layer and as w1 of an expert; kept in the layer's __dict__.  It is good for as long as the layer keeps the descriptor it was
// made from (`of`, the layer's _desc, held here so that its address is not given to another) and its tensors stay where they
// are: the addresses alone do not tell a layer that was quantized again, in another format, into recycled memory.  A copied or
// pickled layer gets None and makes its own.  The descriptor is never changed once it is made.
struct Plan {
    PyObject_HEAD
    PyObject* of;
    hqm_weight w;
    int64_t linear_rows, expert_rows;
    size_t linear_bytes, f16_bytes, expert_bytes;
};
void plan_dealloc(PyObject* self) {
    Py_XDECREF(reinterpret_cast<Plan*>(self)->of);
    PyObject_Free(self);
}
PyObject* plan_copy(PyObject*, PyObject*) { Py_RETURN_NONE; }
PyObject* plan_reduce(PyObject*, PyObject*) { return Py_BuildValue("(O())", (PyObject*)Py_TYPE(Py_None)); }
PyMethodDef plan_methods[] = {{"__deepcopy__", plan_copy, METH_O, nullptr},
                              {"__copy__", plan_copy, METH_NOARGS, nullptr},
                              {"__reduce__", plan_reduce, METH_NOARGS, nullptr},
                              {nullptr, nullptr, 0, nullptr}};
PyTypeObject PlanType = {PyVarObject_HEAD_INIT(nullptr, 0) "mixtral_offloading_b200._host.Plan", sizeof(Plan)};

// borrowed reference out of a dict, null if absent (no error set)
PyObject* item(PyObject* dict, PyObject* key) {
    if (dict == nullptr || !PyDict_CheckExact(dict)) return nullptr;
    PyObject* v = PyDict_GetItemWithError(dict, key);
    if (v == nullptr) PyErr_Clear();
    return v;
}
// An owned reference.  A layer's dictionary may drop what it holds while a call is under way (another thread runs wherever
// Python code does: a workspace that grows, a descriptor that is made), so the call holds what it uses.
template <typename T>
struct Held {
    T* p;
    explicit Held(T* owned = nullptr) : p(owned) {}
    Held(const Held&) = delete;
    Held& operator=(const Held&) = delete;
    ~Held() { Py_XDECREF(reinterpret_cast<PyObject*>(p)); }
    T* operator->() const { return p; }
    explicit operator bool() const { return p != nullptr; }
    void take(T* owned) {
        Py_XDECREF(reinterpret_cast<PyObject*>(p));
        p = owned;
    }
};
PyObject* own(PyObject* borrowed) {
    Py_XINCREF(borrowed);
    return borrowed;
}
const void* address(PyObject* t) { return t != nullptr && THPVariable_Check(t) ? THPVariable_Unpack(t).const_data_ptr() : nullptr; }

// The addresses of a layer's seven tensors; false where it is not ready or has another form.
bool addresses_of(PyObject* dict, const void* (&at)[7]) {
    PyObject* meta = item(dict, N.meta);
    PyObject *ms = item(meta, N.meta_scale), *mz = item(meta, N.meta_zero);
    if (item(dict, N.ready) != Py_True || ms == nullptr || mz == nullptr) return false;
    PyObject* t[7] = {item(dict, N.W_q), item(meta, N.scale_q), item(meta, N.zero_q), item(ms, N.scale), item(ms, N.zero), item(mz, N.scale), item(mz, N.zero)};
    for (int i = 0; i < 7; ++i) at[i] = address(t[i]);
    return true;
}

// The plan of a layer whose tensors are where they were when its descriptor was made (new reference); null: not to be had here.
Plan* plan_of(PyObject* layer, PyObject* dict) {
    const void* at[7];
    if (!addresses_of(dict, at)) return nullptr;
    PyObject* kept = item(dict, N.plan);
    if (kept != nullptr && Py_TYPE(kept) == &PlanType) {
        Plan* p = reinterpret_cast<Plan*>(kept);
        if (p->of == item(dict, N.desc) && p->w.W_q == at[0] && p->w.scale_q == at[1] && p->w.zero_q == at[2] && p->w.ms_scale == at[3] && p->w.mz_scale == at[4] &&
            p->w.ms_zero == at[5] && p->w.mz_zero == at[6])
            return reinterpret_cast<Plan*>(own(kept));
    }
    PyObject* axis = item(item(dict, N.meta), N.axis);
    if (axis == nullptr || !PyLong_Check(axis) || PyLong_AsLong(axis) != 0) return nullptr;
    PyObject* d = PyObject_CallMethod(layer, "descriptor", nullptr);      // validates; a ctypes structure
    if (d == nullptr) {
        PyErr_Clear();
        return nullptr;
    }
    Plan* p = nullptr;
    Py_buffer view;
    if (PyObject_GetBuffer(d, &view, PyBUF_SIMPLE) == 0) {
        if (view.len == (Py_ssize_t)sizeof(hqm_weight) && (p = PyObject_New(Plan, &PlanType)) != nullptr) {
            memcpy(&p->w, view.buf, sizeof(hqm_weight));
            p->of = own(item(dict, N.desc));
            p->linear_rows = p->expert_rows = -1;
            p->linear_bytes = p->f16_bytes = p->expert_bytes = 0;
            if (PyDict_SetItem(dict, N.plan, reinterpret_cast<PyObject*>(p)) != 0) {
                Py_DECREF(p);
                p = nullptr;
            }
        }
        PyBuffer_Release(&view);
    }
    Py_DECREF(d);
    PyErr_Clear();
    return p;
}

PyObject* dict_of(PyObject* module) {        // new reference
    PyObject* d = PyObject_GetAttr(module, N.dict);
    if (d == nullptr) PyErr_Clear();
    return d;
}

// x if it is bf16, fp16 or fp32, contiguous, on the current device, last dimension K, at least one row; else null.
const at::Tensor* rows_of(PyObject* obj, int64_t K, int64_t* rows) {
    if (!THPVariable_CheckExact(obj)) return nullptr;
    const at::Tensor& x = THPVariable_Unpack(obj);
    const auto type = x.scalar_type();
    if (!x.is_cuda() || (type != at::kBFloat16 && type != at::kHalf && type != at::kFloat) || x.dim() < 1 || x.size(-1) != K || x.numel() == 0 || !x.is_contiguous() ||
        x.device().index() != c10::cuda::current_device())
        return nullptr;
    *rows = x.numel() / K;
    return &x;
}

// Workspace of the device (the Python module's, grown through it); its address, null on failure.
void* scratch(const at::Tensor& on, size_t bytes, size_t* have) {
    const int dev = on.device().index();
    if (dev < 0 || dev >= 64) return nullptr;
    if (g_keys[dev] == nullptr && (g_keys[dev] = Py_BuildValue("(si)", "cuda", dev)) == nullptr) return nullptr;
    PyObject* t = item(g_scratch, g_keys[dev]);
    if (t != nullptr && THPVariable_Check(t) && (size_t)THPVariable_Unpack(t).numel() >= bytes) {
        *have = (size_t)THPVariable_Unpack(t).numel();
        return THPVariable_Unpack(t).data_ptr();
    }
    PyObject* device = THPDevice_New(on.device());
    t = device == nullptr ? nullptr : PyObject_CallFunction(g_grow, "On", device, (Py_ssize_t)bytes);
    Py_XDECREF(device);
    if (t == nullptr) {
        PyErr_Clear();
        return nullptr;
    }
    void* p = THPVariable_Unpack(t).data_ptr();           // (the module keeps it)
    *have = (size_t)THPVariable_Unpack(t).numel();
    Py_DECREF(t);
    return p;
}

at::Tensor result(const at::Tensor& x, int64_t n) {
    c10::SmallVector<int64_t, 8> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = n;
    return at::empty(shape, x.options());
}

// linear(layer, x)
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) return PyErr_Format(PyExc_TypeError, "linear(layer, x)");
    try {
        Held<PyObject> dict(dict_of(args[0]));
        Held<Plan> p(dict ? plan_of(args[0], dict.p) : nullptr);
        Held<PyObject> bias(own(item(dict.p, N.bias)));
        int64_t rows = 0;
        const at::Tensor* x = p ? rows_of(args[1], p->w.K, &rows) : nullptr;
        if (x == nullptr) Py_RETURN_NONE;
        c10::InferenceMode guard;
        const auto type = x->scalar_type();
        if (p->linear_rows != rows) {
            p->linear_bytes = hqm_linear_scratch_preferred(rows, &p->w);
            p->f16_bytes = hqm_linear_f16_scratch_bytes(rows, &p->w);
            p->linear_rows = rows;
        }
        const bool f16 = type == at::kHalf && p->f16_bytes != 0;
        at::Tensor converted;
        if (type != at::kBFloat16 && !f16) {
            converted = x->to(at::kBFloat16);
            x = &converted;
        }
        const size_t bytes = f16 ? p->f16_bytes : p->linear_bytes;
        size_t have = 0;
        void* ws = nullptr;
        if (bytes && (ws = scratch(*x, bytes, &have)) == nullptr) Py_RETURN_NONE;
        at::Tensor y = result(*x, p->w.N);
        const uint16_t* b = static_cast<const uint16_t*>(address(bias.p));
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = (f16 ? hqm_linear_f16 : hqm_linear)(static_cast<uint16_t*>(y.data_ptr()), static_cast<const uint16_t*>(x->const_data_ptr()), rows,
                                                 &p->w, b, ws, bytes, c10::cuda::getCurrentCUDAStream(x->device().index()).stream());
        Py_END_ALLOW_THREADS
        if (rc < 0) Py_RETURN_NONE;
        if (y.scalar_type() != type) y = y.to(type);
        return THPVariable_Wrap(std::move(y));
    } catch (const std::exception& e) {
        return PyErr_Format(PyExc_RuntimeError, "%s", e.what());
    }
}

// dequantize(layer, code): the weight in bf16 (0), fp16 (1) or fp32 (2)
PyObject* dequantize(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) return PyErr_Format(PyExc_TypeError, "dequantize(layer, code)");
    try {
        const long code = PyLong_AsLong(args[1]);
        Held<PyObject> dict(dict_of(args[0]));
        Held<Plan> p(dict ? plan_of(args[0], dict.p) : nullptr);
        Held<PyObject> wq(own(item(dict.p, N.W_q)));
        if (!p || address(wq.p) != p->w.W_q || code < 0 || code > 2) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        const at::Tensor& like = THPVariable_Unpack(wq.p);
        if (like.device().index() != c10::cuda::current_device()) Py_RETURN_NONE;
        c10::InferenceMode guard;
        at::Tensor out = at::empty({p->w.N, p->w.K}, like.options().dtype(code == 0 ? at::kBFloat16 : code == 1 ? at::kHalf : at::kFloat));
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = hqm_dequantize(out.data_ptr(), (int)code, &p->w, c10::cuda::getCurrentCUDAStream(like.device().index()).stream());
        Py_END_ALLOW_THREADS
        if (rc < 0) Py_RETURN_NONE;
        return THPVariable_Wrap(std::move(out));
    } catch (const std::exception& e) {
        return PyErr_Format(PyExc_RuntimeError, "%s", e.what());
    }
}

// The three plans of an expert module.
bool expert_plans(PyObject* module, Held<Plan> (&p)[3]) {
    Held<PyObject> dict(dict_of(module));
    Held<PyObject> modules(own(item(dict.p, N.modules)));
    PyObject* names[3] = {N.w1, N.w2, N.w3};
    for (int i = 0; i < 3; ++i) {
        Held<PyObject> layer(own(item(modules.p, names[i])));
        Held<PyObject> d(layer ? dict_of(layer.p) : nullptr);
        p[i].take(d ? plan_of(layer.p, d.p) : nullptr);
        if (!p[i]) return false;
    }
    return true;
}

int run_expert(const Held<Plan> (&p)[3], const at::Tensor& x, int64_t rows, const int32_t* idx, const float* w, uint16_t* out, int accumulate) {
    if (p[0]->expert_rows != rows) {
        p[0]->expert_bytes = hqm_expert_ffn_scratch_bytes(rows, &p[0]->w, &p[1]->w, &p[2]->w);
        p[0]->expert_rows = rows;
    }
    size_t have = 0;
    void* ws = scratch(x, p[0]->expert_bytes, &have);
    if (ws == nullptr) return -1;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = hqm_expert_ffn(out, static_cast<const uint16_t*>(x.const_data_ptr()), rows, idx, w, accumulate, &p[0]->w, &p[1]->w, &p[2]->w, ws, have,
                        c10::cuda::getCurrentCUDAStream(x.device().index()).stream());
    Py_END_ALLOW_THREADS
    return rc;
}

// expert(module, x): all rows of x
PyObject* expert(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) return PyErr_Format(PyExc_TypeError, "expert(module, x)");
    try {
        Held<Plan> p[3];
        if (!expert_plans(args[0], p)) Py_RETURN_NONE;
        int64_t rows = 0;
        const at::Tensor* x = rows_of(args[1], p[0]->w.K, &rows);
        if (x == nullptr) Py_RETURN_NONE;
        c10::InferenceMode guard;
        const auto type = x->scalar_type();
        at::Tensor converted;
        if (type != at::kBFloat16) {
            converted = x->to(at::kBFloat16);
            x = &converted;
        }
        at::Tensor out = result(*x, p[1]->w.N);
        if (run_expert(p, *x, rows, nullptr, nullptr, static_cast<uint16_t*>(out.data_ptr()), 0) < 0) Py_RETURN_NONE;
        if (type != at::kBFloat16) out = out.to(type);
        return THPVariable_Wrap(std::move(out));
    } catch (const std::exception& e) {
        return PyErr_Format(PyExc_RuntimeError, "%s", e.what());
    }
}

// expert_addresses(experts): the addresses of all layers' descriptors and tensors as bytes; None where a layer has no descriptor
// (its tensors were replaced) or another form.  For as long as the caller holds the descriptors, what it made from them is good
// while this does not change.
PyObject* expert_addresses(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 1 || !PyList_CheckExact(args[0])) return PyErr_Format(PyExc_TypeError, "expert_addresses(list)");
    const Py_ssize_t experts = PyList_GET_SIZE(args[0]);
    Held<PyObject> out(PyBytes_FromStringAndSize(nullptr, experts * 3 * 8 * (Py_ssize_t)sizeof(void*)));
    if (!out) return nullptr;
    char* to = PyBytes_AS_STRING(out.p);
    PyObject* names[3] = {N.w1, N.w2, N.w3};
    for (Py_ssize_t e = 0; e < experts; ++e) {
        if (e >= PyList_GET_SIZE(args[0])) Py_RETURN_NONE;
        Held<PyObject> module(own(PyList_GET_ITEM(args[0], e)));
        Held<PyObject> outer(dict_of(module.p));
        if (PyObject* inner = item(outer.p, N.expert)) module.take(own(inner));       // a wrapper around the expert
        Held<PyObject> dict(dict_of(module.p));
        Held<PyObject> modules(own(item(dict.p, N.modules)));
        for (PyObject* name : names) {
            Held<PyObject> layer(own(item(modules.p, name)));
            Held<PyObject> d(layer ? dict_of(layer.p) : nullptr);
            PyObject* desc = item(d.p, N.desc);
            const void* at[7];
            if (desc == nullptr || desc == Py_None || !addresses_of(d.p, at)) Py_RETURN_NONE;
            memcpy(to, &desc, sizeof(desc));
            memcpy(to + sizeof(desc), at, sizeof(at));
            to += sizeof(desc) + sizeof(at);
        }
    }
    return own(out.p);
}

PyObject* setup(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) return PyErr_Format(PyExc_TypeError, "setup(scratch, grow)");
    Py_INCREF(args[0]);
    Py_INCREF(args[1]);
    Py_XSETREF(g_scratch, args[0]);
    Py_XSETREF(g_grow, args[1]);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"setup", (PyCFunction)(void (*)(void))setup, METH_FASTCALL, "setup(scratch_dict, grow)"},
    {"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, "linear(layer, x) -> tensor or None"},
    {"dequantize", (PyCFunction)(void (*)(void))dequantize, METH_FASTCALL, "dequantize(layer, dtype code) -> tensor or None"},
    {"expert", (PyCFunction)(void (*)(void))expert, METH_FASTCALL, "expert(module, x) -> tensor or None"},
    {"expert_addresses", (PyCFunction)(void (*)(void))expert_addresses, METH_FASTCALL, "expert_addresses(experts) -> bytes or None"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Host path of the quantized layers.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    struct {
        PyObject** to;
        const char* name;
    } all[] = {{&N.dict, "__dict__"}, {&N.W_q, "W_q"},     {&N.meta, "meta"},           {&N.bias, "bias"},           {&N.plan, "_plan"}, {&N.desc, "_desc"}, {&N.ready, "ready"}, {&N.expert, "_expert"},
               {&N.scale_q, "scale_q"}, {&N.zero_q, "zero_q"}, {&N.meta_scale, "meta_scale"}, {&N.meta_zero, "meta_zero"}, {&N.scale, "scale"}, {&N.zero, "zero"},
               {&N.modules, "_modules"}, {&N.w1, "w1"},    {&N.w2, "w2"},               {&N.w3, "w3"}, {&N.axis, "axis"}};
    for (auto& a : all)
        if ((*a.to = PyUnicode_InternFromString(a.name)) == nullptr) return nullptr;
    PlanType.tp_flags = Py_TPFLAGS_DEFAULT;
    PlanType.tp_methods = plan_methods;
    PlanType.tp_dealloc = plan_dealloc;
    if (PyType_Ready(&PlanType) != 0) return nullptr;
    return PyModule_Create(&module);
}
