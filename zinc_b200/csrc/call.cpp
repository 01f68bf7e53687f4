// Python -> C ABI calls without ctypes: one vectorcall object per exported function. A call names its buffers as CUDA
// tensors or Buffer objects; pointers and byte sizes are taken here, and the function is entered with the interpreter
// lock released, as ctypes does. A matvec's Python side costs 1.3 us this way instead of 5 us (three tensors, thirteen
// arguments), less than its kernel.
#include <Python.h>
#include <structmember.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>
#include <type_traits>
#include <utility>

#include "../../include/zinc_cuda.h"

namespace {

constexpr int kMaxWords = 32;

// Arguments as 64-bit words in order (floats apart: a function has one at most) -> the function's own parameters.
template <typename P>
P argument(const uint64_t* w, size_t at, float f) {
    if constexpr (std::is_same_v<P, float>) return f;
    else if constexpr (std::is_pointer_v<P>) return reinterpret_cast<P>(static_cast<uintptr_t>(w[at]));
    else return static_cast<P>(w[at]);
}
template <typename Fn>
struct Invoke;
template <typename... P>
struct Invoke<int32_t (*)(P...)> {
    static constexpr int kWords = ((std::is_same_v<P, float> ? 0 : 1) + ... + 0);
    static constexpr size_t word_of(size_t param) {  // word of parameter `param`: floats take none
        constexpr bool is_float[] = {std::is_same_v<P, float>...};
        size_t at = 0;
        for (size_t i = 0; i < param; ++i) at += is_float[i] ? 0 : 1;
        return at;
    }
    template <size_t... I>
    static int32_t run(uint64_t fn, const uint64_t* w, float f, std::index_sequence<I...>) {
        return reinterpret_cast<int32_t (*)(P...)>(static_cast<uintptr_t>(fn))(argument<P>(w, word_of(I), f)...);
    }
    static int32_t go(uint64_t fn, const uint64_t* w, float f) { return run(fn, w, f, std::index_sequence_for<P...>()); }
};

struct Entry {
    const char* name;
    int words;
    int32_t (*go)(uint64_t fn, const uint64_t* w, float f);
};
#define ENTRY(name) {#name, Invoke<decltype(&name)>::kWords, Invoke<decltype(&name)>::go}
constexpr Entry kEntries[] = {
    ENTRY(zc_dmmv), ENTRY(zc_dmmv_push), ENTRY(zc_dmmv_batch), ENTRY(zc_moe_dmmv), ENTRY(zc_moe_dmmv_batched),
    ENTRY(zc_moe_dmmv_batched_pair), ENTRY(zc_mul_mm_block_scaled), ENTRY(zc_count_experts), ENTRY(zc_mul_mm),
    ENTRY(zc_dmmv_fused_gate_up_swiglu), ENTRY(zc_dmmv_sigmoid_acc), ENTRY(zc_moe_fused_gate_up), ENTRY(zc_moe_fused_gate_up_act),
    ENTRY(zc_moe_gate_up_act_ex), ENTRY(zc_moe_down_acc_ex), ENTRY(zc_moe_router_topk), ENTRY(zc_rms_norm_dmmv_f32),
    ENTRY(zc_dmmv_o_proj_merge), ENTRY(zc_rms_norm_dmmv_alpha_beta), ENTRY(zc_moe_weighted_acc), ENTRY(zc_bias_add),
    ENTRY(zc_moe_bias_act), ENTRY(zc_moe_weighted_bias_acc), ENTRY(zc_moe_ep_filter), ENTRY(zc_moe_route_pack),
    ENTRY(zc_moe_route_scatter), ENTRY(zc_dequant_rows),
};
#undef ENTRY

struct Call {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    uint64_t fn;
    int32_t (*go)(uint64_t fn, const uint64_t* w, float f);
    char spec[kMaxWords + 1];  // i integer, f float, b buffer, o buffer or None
    int n;
    PyObject* to_buffer;       // Python: anything else -> Buffer (raises)
};

PyObject *s_ptr, *s_size;

bool take_int(PyObject* o, uint64_t& v) {
    if (PyLong_CheckExact(o)) {
        v = PyLong_AsUnsignedLongLongMask(o);
        return !(v == (uint64_t)-1 && PyErr_Occurred());
    }
    PyObject* i = PyNumber_Index(o);
    if (!i) return false;
    v = PyLong_AsUnsignedLongLongMask(i);
    Py_DECREF(i);
    return !(v == (uint64_t)-1 && PyErr_Occurred());
}

bool take_attr(PyObject* o, PyObject* name, uint64_t& v) {
    PyObject* a = PyObject_GetAttr(o, name);
    if (!a) return false;
    bool ok = true;
    if (a == Py_None) v = 0;
    else ok = take_int(a, v);
    Py_DECREF(a);
    return ok;
}

// *keep: an object made here that owns the memory (to be released after the call)
bool take_buffer(Call* c, PyObject* o, uint64_t& ptr, uint64_t& size, PyObject** keep) {
    // Plain tensors only: a subclass answers for itself in Python. Tensors without memory of their own (under a
    // transform or a tracer) answer with a C++ exception, which must not leave through the interpreter's C frames:
    // they go the Python way too, where the same question raises.
    if (THPVariable_CheckExact(o)) {
        try {
            const at::Tensor& t = THPVariable_Unpack(o);
            if (t.is_cuda() && t.is_contiguous()) {
                ptr = reinterpret_cast<uint64_t>(t.data_ptr());
                size = t.nbytes();
                return true;
            }
        } catch (...) {
        }
    }
    PyObject* b = PyObject_CallOneArg(c->to_buffer, o);  // a Buffer comes back as itself
    if (!b) return false;
    *keep = b;
    return take_attr(b, s_ptr, ptr) && take_attr(b, s_size, size);
}

PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    Call* c = reinterpret_cast<Call*>(self);
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    if ((kwnames && PyTuple_GET_SIZE(kwnames)) || n != c->n) {
        PyErr_Format(PyExc_TypeError, "expected %d positional arguments, got %zd", c->n, n);
        return nullptr;
    }
    uint64_t w[kMaxWords] = {0};
    PyObject* keep[kMaxWords] = {nullptr};
    float f = 0.f;
    int k = 0, kept = 0;
    bool ok = true;
    for (Py_ssize_t i = 0; i < n && ok; ++i) {
        switch (c->spec[i]) {
            case 'i': ok = take_int(args[i], w[k++]); break;
            case 'f': {
                const double d = PyFloat_AsDouble(args[i]);
                ok = !(d == -1.0 && PyErr_Occurred());
                f = (float)d;
                break;
            }
            case 'o':
                if (args[i] == Py_None) {
                    k += 2;
                    break;
                }
                [[fallthrough]];
            default:
                ok = take_buffer(c, args[i], w[k], w[k + 1], &keep[kept]);
                if (keep[kept]) ++kept;
                k += 2;
        }
    }
    int32_t rc = 0;
    if (ok) {
        Py_BEGIN_ALLOW_THREADS
        rc = c->go(c->fn, w, f);
        Py_END_ALLOW_THREADS
    }
    for (int i = 0; i < kept; ++i) Py_DECREF(keep[i]);
    return ok ? PyLong_FromLong(rc) : nullptr;
}

PyObject* call_new(PyTypeObject* type, PyObject* args, PyObject*) {
    unsigned long long fn;
    const char *name, *spec;
    PyObject* to_buffer;
    if (!PyArg_ParseTuple(args, "KssO", &fn, &name, &spec, &to_buffer)) return nullptr;
    const Entry* entry = nullptr;
    for (const Entry& e : kEntries)
        if (!std::strcmp(e.name, name)) entry = &e;
    int words = 0, n = 0;
    for (const char* p = spec; *p; ++p, ++n) words += *p == 'i' ? 1 : *p == 'f' ? 0 : 2;
    if (!entry || words != entry->words || words > kMaxWords || n > kMaxWords) {
        PyErr_Format(PyExc_ValueError, "%s does not take the arguments '%s'", name, spec);
        return nullptr;
    }
    Call* c = reinterpret_cast<Call*>(type->tp_alloc(type, 0));
    if (!c) return nullptr;
    c->vectorcall = call;
    c->fn = fn;
    c->go = entry->go;
    std::strcpy(c->spec, spec);
    c->n = n;
    Py_INCREF(to_buffer);
    c->to_buffer = to_buffer;
    return reinterpret_cast<PyObject*>(c);
}

void call_dealloc(PyObject* self) {
    Py_XDECREF(reinterpret_cast<Call*>(self)->to_buffer);
    Py_TYPE(self)->tp_free(self);
}

PyTypeObject CallType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", nullptr, -1, nullptr, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__call(void) {
    CallType.tp_name = "zinc_b200._call.Call";
    CallType.tp_basicsize = sizeof(Call);
    CallType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
    CallType.tp_vectorcall_offset = offsetof(Call, vectorcall);
    CallType.tp_call = PyVectorcall_Call;
    CallType.tp_new = call_new;
    CallType.tp_dealloc = call_dealloc;
    if (PyType_Ready(&CallType) < 0) return nullptr;
    s_ptr = PyUnicode_InternFromString("ptr");
    s_size = PyUnicode_InternFromString("size");
    PyObject* m = PyModule_Create(&module);
    if (!m || PyModule_AddObjectRef(m, "Call", reinterpret_cast<PyObject*>(&CallType)) < 0) return nullptr;
    return m;
}
