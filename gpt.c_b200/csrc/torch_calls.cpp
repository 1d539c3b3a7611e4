// The tensor-level calls of the Python package (forward, backward, linear_*, layernorm_*) as a CPython extension
// over the C ABI of libattn_sm100.so.
//
// What bounds small calls is the host: with these functions written in Python, a forward and backward of
// B=1 T=40 H=2 spent 39 us per pass on the host (three allocations of 2.6 us each, 3.2 us to find the current
// stream, 11 to 13 converted arguments per ctypes call) around 16 us of GPU work.  Here the arguments are taken
// from the tensor objects directly, outputs come from the caching allocator without going through the operator
// dispatcher, and the stream is a thread-local read.  The GIL is released around the C ABI call, as ctypes does.
// The element-wise entry points and size queries that programs call through lib() get the same treatment (shorten_calls):
// converting their arguments took ctypes 0.5 to 1 us of the 2.8 us of a call, 2.3 of which the launch itself needs.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/attn_sm100.h"
#include "../../include/layernorm_sm100.h"
#include "../../include/linear_sm100.h"
#include "../../include/tensor_sm100.h"
#include "../../include/xent_sm100.h"

#include <tuple>
#include <utility>

namespace {

PyObject *g_error = nullptr;  // the package's AttnError(code, where)

// Raises AttnError for a non-zero status.
bool failed(int code, const char *where) {
    if (code == ATTN_OK) return false;
    PyObject *args = Py_BuildValue("(is)", code, where);
    PyObject *e = args && g_error ? PyObject_CallObject(g_error, args) : nullptr;
    Py_XDECREF(args);
    if (e) {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
    } else if (!PyErr_Occurred()) {
        PyErr_Format(PyExc_RuntimeError, "%s failed with status %d", where, code);
    }
    return true;
}

// One positional argument list, read with checks that set a Python error; `ok` turns false on the first bad one.
struct Args {
    PyObject *const *v;
    bool ok = true;

    Args(PyObject *const *args, Py_ssize_t n, Py_ssize_t want) : v(args) {
        if (n != want) {
            PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
            ok = false;
        }
    }
    const at::Tensor *tensor(int i) {
        if (!ok) return nullptr;
        if (!THPVariable_Check(v[i])) {
            PyErr_Format(PyExc_TypeError, "argument %d must be a tensor", i);
            ok = false;
            return nullptr;
        }
        return &THPVariable_Unpack(v[i]);
    }
    // A tensor an output is allocated next to: on a CUDA device, with at least one dimension.
    const at::Tensor *cuda(int i) {
        const at::Tensor *t = tensor(i);
        if (ok && (!t->is_cuda() || t->dim() < 1 || t->size(-1) < 1)) {
            PyErr_SetString(PyExc_ValueError, "expected a CUDA tensor with a non-empty last dimension");
            ok = false;
        }
        return ok ? t : nullptr;
    }
    template <class T>
    T *ptr(int i) {  // None gives NULL
        if (!ok || v[i] == Py_None) return nullptr;
        const at::Tensor *t = tensor(i);
        return ok ? static_cast<T *>(t->data_ptr()) : nullptr;
    }
    float *f32(int i) { return ptr<float>(i); }
    long integer(int i) {
        if (!ok) return 0;
        const long r = PyLong_AsLong(v[i]);
        if (r == -1 && PyErr_Occurred()) ok = false;
        return r;
    }
    double real(int i) {
        if (!ok) return 0;
        const double r = PyFloat_AsDouble(v[i]);
        if (r == -1.0 && PyErr_Occurred()) ok = false;
        return r;
    }
    // None: the current stream of the current device; else a cudaStream_t as an integer.
    void *stream(int i) {
        if (!ok) return nullptr;
        if (v[i] == Py_None) return c10::cuda::getCurrentCUDAStream().stream();
        void *s = PyLong_AsVoidPtr(v[i]);
        if (PyErr_Occurred()) ok = false;
        return s;
    }
};

at::Tensor alloc(at::IntArrayRef shape, at::ScalarType type, const at::Tensor &beside) {
    return at::detail::empty_cuda(shape, type, beside.device(), std::nullopt);
}

PyObject *value_error(const char *text) {
    PyErr_SetString(PyExc_ValueError, text);
    return nullptr;
}

// forward(qkv, n_heads, flags, keep_copy) -> (out, out_copy or None, lse, saved, (B, T, H, D))
PyObject *forward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 4);
    const at::Tensor *qkv = a.tensor(0);
    const long H = a.integer(1), flags = a.integer(2);
    const int keep = a.ok ? PyObject_IsTrue(args[3]) : 0;
    if (!a.ok || keep < 0) return nullptr;
    if (!(qkv->is_cuda() && qkv->scalar_type() == at::kFloat && qkv->is_contiguous() && qkv->dim() == 3))
        return value_error("qkv must be a contiguous fp32 CUDA tensor of shape [B, T, 3C]");
    const int64_t B = qkv->size(0), T = qkv->size(1), C3 = qkv->size(2);
    if (H <= 0 || C3 % (3 * H) != 0) return value_error("last dimension must be 3 * n_heads * head_size");
    const int64_t C = C3 / 3, D = C / H;
    const size_t saved_bytes = attn_sm100_saved_bytes((int)B, (int)T, (int)H, (int)D);
    at::Tensor out = alloc({B, T, C}, at::kFloat, *qkv);
    at::Tensor copy;
    if (keep) copy = alloc({B, T, C}, at::kFloat, *qkv);
    at::Tensor lse = alloc({B, H, T}, at::kFloat, *qkv);
    at::Tensor saved = alloc({(int64_t)saved_bytes}, at::kByte, *qkv);
    void *stream = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = attn_sm100_forward(static_cast<const float *>(qkv->data_ptr()), static_cast<float *>(out.data_ptr()),
                            keep ? static_cast<float *>(copy.data_ptr()) : nullptr, static_cast<float *>(lse.data_ptr()),
                            saved.data_ptr(), (int)B, (int)T, (int)H, (int)D, (int)flags, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "attn_sm100_forward")) return nullptr;
    PyObject *second = keep ? THPVariable_Wrap(copy) : Py_NewRef(Py_None);
    return Py_BuildValue("(NNNN(iiii))", THPVariable_Wrap(out), second, THPVariable_Wrap(lse), THPVariable_Wrap(saved), (int)B,
                         (int)T, (int)H, (int)D);
    END_HANDLE_TH_ERRORS
}

// backward(saved, out, lse, dout, (B, T, H, D), flags) -> dqkv
PyObject *backward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 6);
    const void *saved = a.ptr<void>(0);
    const float *out = a.f32(1), *lse = a.f32(2);
    const at::Tensor *dout = a.tensor(3);
    const long flags = a.integer(5);
    int B, T, H, D;
    if (!a.ok || !PyArg_ParseTuple(args[4], "iiii", &B, &T, &H, &D)) return nullptr;
    if (!(dout->is_cuda() && dout->scalar_type() == at::kFloat && dout->is_contiguous() && dout->dim() == 3 &&
          dout->size(0) == B && dout->size(1) == T && dout->size(2) == (int64_t)H * D))
        return value_error("dout must be a contiguous fp32 CUDA tensor of shape [B, T, C]");
    at::Tensor dqkv = alloc({B, T, 3 * (int64_t)H * D}, at::kFloat, *dout);
    at::Tensor scratch = alloc({(int64_t)attn_sm100_backward_scratch_bytes(B, T, H, D)}, at::kByte, *dout);
    void *stream = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = attn_sm100_backward(saved, out, lse, static_cast<const float *>(dout->data_ptr()),
                             static_cast<float *>(dqkv.data_ptr()), scratch.data_ptr(), B, T, H, D, (int)flags, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "attn_sm100_backward")) return nullptr;
    return THPVariable_Wrap(dqkv);
    END_HANDLE_TH_ERRORS
}

// forward_into(qkv, out, out_copy, lse, saved, n_heads, flags, stream)
PyObject *forward_into(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 8);
    const at::Tensor *qkv = a.tensor(0);
    float *out = a.f32(1), *copy = a.f32(2), *lse = a.f32(3);
    void *saved = a.ptr<void>(4);
    const long H = a.integer(5), flags = a.integer(6);
    void *stream = a.stream(7);
    if (!a.ok) return nullptr;
    if (qkv->dim() != 3 || H == 0) return value_error("qkv must have the shape [B, T, 3C]");
    const int B = (int)qkv->size(0), T = (int)qkv->size(1), D = (int)(qkv->size(2) / 3 / H);
    const float *x = static_cast<const float *>(qkv->data_ptr());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = attn_sm100_forward(x, out, copy, lse, saved, B, T, (int)H, D, (int)flags, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "attn_sm100_forward")) return nullptr;
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// backward_into(saved, out, lse, dout, dqkv, scratch, n_heads, flags, stream)
PyObject *backward_into(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 9);
    const void *saved = a.ptr<void>(0);
    const float *out = a.f32(1), *lse = a.f32(2);
    const at::Tensor *dout = a.tensor(3);
    float *dqkv = a.f32(4);
    void *scratch = a.ptr<void>(5);
    const long H = a.integer(6), flags = a.integer(7);
    void *stream = a.stream(8);
    if (!a.ok) return nullptr;
    if (dout->dim() != 3 || H == 0) return value_error("dout must have the shape [B, T, C]");
    const int B = (int)dout->size(0), T = (int)dout->size(1), D = (int)(dout->size(2) / H);
    const float *g = static_cast<const float *>(dout->data_ptr());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = attn_sm100_backward(saved, out, lse, g, dqkv, scratch, B, T, (int)H, D, (int)flags, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "attn_sm100_backward")) return nullptr;
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// linear_forward(x, w, bias, planes, stream) -> y
PyObject *linear_forward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 5);
    const at::Tensor *x = a.cuda(0), *w = a.cuda(1);
    const float *bias = a.f32(2);
    void *planes = a.ptr<void>(3);
    void *stream = a.stream(4);
    if (!a.ok) return nullptr;
    const int64_t K = x->size(-1), N = w->size(0), M = x->numel() / K;
    c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
    shape.back() = N;
    at::Tensor y = alloc(shape, at::kFloat, *x);
    const float *xp = static_cast<const float *>(x->data_ptr()), *wp = static_cast<const float *>(w->data_ptr());
    float *yp = static_cast<float *>(y.data_ptr());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = linear_sm100_forward(xp, wp, bias, yp, planes, (int)M, (int)N, (int)K, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "linear_sm100_forward")) return nullptr;
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// linear_backward(dy, x, w, dw, db, stream, want_dx) -> dx or None
PyObject *linear_backward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 7);
    const float *dy = a.f32(0);
    const at::Tensor *x = a.cuda(1), *w = a.cuda(2);
    float *dw = a.f32(3), *db = a.f32(4);
    void *stream = a.stream(5);
    const int want_dx = a.ok ? PyObject_IsTrue(args[6]) : 0;
    if (!a.ok || want_dx < 0) return nullptr;
    const int64_t K = x->size(-1), N = w->size(0), M = x->numel() / K;
    at::Tensor dx, scratch;
    if (want_dx) dx = alloc(x->sizes(), at::kFloat, *x);
    const size_t bytes = linear_sm100_backward_scratch_bytes((int)M, (int)N, (int)K);
    if (bytes) scratch = alloc({(int64_t)bytes}, at::kByte, *x);
    const float *xp = static_cast<const float *>(x->data_ptr()), *wp = static_cast<const float *>(w->data_ptr());
    float *dxp = want_dx ? static_cast<float *>(dx.data_ptr()) : nullptr;
    void *sp = bytes ? scratch.data_ptr() : nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = linear_sm100_backward(dy, xp, wp, dxp, dw, db, sp, (int)M, (int)N, (int)K, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "linear_sm100_backward")) return nullptr;
    if (!want_dx) Py_RETURN_NONE;
    return THPVariable_Wrap(dx);
    END_HANDLE_TH_ERRORS
}

// layernorm_forward(x, w, b, eps, stream) -> (y, mean, rstd)
PyObject *layernorm_forward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 5);
    const at::Tensor *x = a.cuda(0);
    const float *w = a.f32(1), *b = a.f32(2);
    const double eps = a.real(3);
    void *stream = a.stream(4);
    if (!a.ok) return nullptr;
    const int64_t C = x->size(-1), rows = x->numel() / C;
    at::Tensor y = alloc(x->sizes(), at::kFloat, *x);
    at::Tensor mean = alloc({rows}, at::kFloat, *x), rstd = alloc({rows}, at::kFloat, *x);
    const float *xp = static_cast<const float *>(x->data_ptr());
    float *yp = static_cast<float *>(y.data_ptr()), *mp = static_cast<float *>(mean.data_ptr()),
          *rp = static_cast<float *>(rstd.data_ptr());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = layernorm_sm100_forward(xp, w, b, (float)eps, mp, rp, yp, (int)rows, (int)C, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "layernorm_sm100_forward")) return nullptr;
    return Py_BuildValue("(NNN)", THPVariable_Wrap(y), THPVariable_Wrap(mean), THPVariable_Wrap(rstd));
    END_HANDLE_TH_ERRORS
}

// layernorm_backward(dy, x, mean, rstd, w, dw, db, dx, stream)
PyObject *layernorm_backward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Args a(args, n, 9);
    const at::Tensor *x = a.cuda(1);
    const float *dy = a.f32(0), *mean = a.f32(2), *rstd = a.f32(3), *w = a.f32(4);
    float *dw = a.f32(5), *db = a.f32(6), *dx = a.f32(7);
    void *stream = a.stream(8);
    if (!a.ok) return nullptr;
    const int64_t C = x->size(-1), rows = x->numel() / C;
    const float *xp = static_cast<const float *>(x->data_ptr());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = layernorm_sm100_backward(dy, xp, mean, rstd, w, dw, db, dx, (int)rows, (int)C, stream);
    Py_END_ALLOW_THREADS
    if (failed(rc, "layernorm_sm100_backward")) return nullptr;
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------
// What calling a ctypes function of the library does instead, as the tp_call of its function object's class: a call with
// exactly as many plain numbers (or None for a pointer) as the function has arguments goes to the C ABI from here, every
// other one to ctypes.
// ------------------------------------------------------------------------------------------
template <class T>
bool take(PyObject *o, T *&out) {
    if (o == Py_None) out = nullptr;
    else if (PyLong_Check(o)) out = reinterpret_cast<T *>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(o)));
    else return false;
    return true;
}
bool take(PyObject *o, int &out) { return PyLong_Check(o) && (out = static_cast<int>(PyLong_AsUnsignedLongLongMask(o)), true); }
bool take(PyObject *o, size_t &out) { return PyLong_Check(o) && (out = static_cast<size_t>(PyLong_AsUnsignedLongLongMask(o)), true); }
bool take(PyObject *o, float &out) { return PyFloat_Check(o) && (out = static_cast<float>(PyFloat_AS_DOUBLE(o)), true); }

template <class R, class... A, size_t... I>
PyObject *invoke(R (*fn)(A...), ternaryfunc own, PyObject *self, PyObject *args, PyObject *keywords, std::index_sequence<I...>) {
    std::tuple<A...> v;
    if (keywords != nullptr || PyTuple_GET_SIZE(args) != (Py_ssize_t)sizeof...(A) || !(take(PyTuple_GET_ITEM(args, I), std::get<I>(v)) && ...)) {
        PyTypeObject *base = Py_TYPE(self)->tp_base;  // of the function's class, or of one derived from it
        while (base->tp_call == own) base = base->tp_base;
        return base->tp_call(self, args, keywords);
    }
    R rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fn(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return std::is_signed_v<R> ? PyLong_FromLong(static_cast<long>(rc)) : PyLong_FromSize_t(static_cast<size_t>(rc));
}
template <class R, class... A>
constexpr size_t arity(R (*)(A...)) { return sizeof...(A); }
template <auto kFn>
PyObject *call(PyObject *self, PyObject *args, PyObject *keywords) {
    return invoke(kFn, call<kFn>, self, args, keywords, std::make_index_sequence<arity(kFn)>());
}

#define ENTRY(name) {#name, call<name>}
const struct {
    const char *name;
    ternaryfunc call;
} kEntries[] = {ENTRY(tensor_sm100_fill),        ENTRY(tensor_sm100_arange),        ENTRY(tensor_sm100_copy),
                ENTRY(tensor_sm100_axpy),        ENTRY(tensor_sm100_gelu_forward),  ENTRY(tensor_sm100_gelu_backward),
                ENTRY(xent_sm100_forward),       ENTRY(xent_sm100_backward),        ENTRY(attn_sm100_saved_bytes),
                ENTRY(attn_sm100_backward_scratch_bytes)};

// shorten_calls({name of an entry point: class of its function alone, a Python class derived from ctypes' own})
PyObject *shorten_calls(PyObject *, PyObject *classes) {
    for (const auto &e : kEntries) {
        PyObject *cls = PyDict_Check(classes) ? PyDict_GetItemString(classes, e.name) : nullptr;
        if (cls == nullptr || !PyType_Check(cls) || !PyType_HasFeature(reinterpret_cast<PyTypeObject *>(cls), Py_TPFLAGS_HEAPTYPE) ||
            reinterpret_cast<PyTypeObject *>(cls)->tp_base->tp_call == nullptr) {
            PyErr_Format(PyExc_TypeError, "%s: expected a class derived from that of ctypes functions", e.name);
            return nullptr;
        }
        reinterpret_cast<PyTypeObject *>(cls)->tp_call = e.call;
        PyType_Modified(reinterpret_cast<PyTypeObject *>(cls));
    }
    Py_RETURN_NONE;
}

// set_error(cls): the exception class raised for a non-zero status
PyObject *set_error(PyObject *, PyObject *cls) {
    Py_INCREF(cls);
    Py_XDECREF(g_error);
    g_error = cls;
    Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FAST(forward), FAST(backward), FAST(forward_into), FAST(backward_into), FAST(linear_forward),
                          FAST(linear_backward), FAST(layernorm_forward), FAST(layernorm_backward),
                          {"set_error", set_error, METH_O, nullptr}, {"shorten_calls", shorten_calls, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "gptc_b200_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_gptc_b200_calls(void) { return PyModule_Create(&kModule); }
