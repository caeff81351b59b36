// Host side of the operator interface in native code: the tensor object (storage + shape + element strides) and one
// function per operator that checks its arguments, allocates the outputs and calls the C ABI of libmni_b200.so.
//
// Why it is native: through ctypes and Python objects an operator spent 10-12 us on the host before its first launch
// (naming the current stream 3.2 us, each output 3.2, each operand's view struct 1.1), more than the device needs for a
// small product.  Here those are tens of nanoseconds; what is left is the launch itself.
//
// The library is bound at the first call (see _lib.py, which checks that it was built from the tree's sources).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/SmallVector.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <new>
#include <vector>

#include "mni_b200.h"

namespace {

using Dims = c10::SmallVector<int64_t, MNI_B200_MAX_DIMS>;

struct TensorObj {
    PyObject_HEAD
    at::Tensor flat;               // flat f32 CUDA storage; its data pointer is the tensor's first element
    Dims shape, stride;
    bool contiguous;               // stride == row-major strides of shape
    PyObject *shape_tuple, *stride_tuple;   // built when Python asks for them
};

PyTypeObject *g_class = nullptr;       // the Python class results are instances of
PyObject *g_loader = nullptr;          // binds the library: called once, before the first native call
PyObject *g_raise_status = nullptr;    // raises for a status code
PyObject *g_check_shapes = nullptr;    // raises for operands that do not multiply

// ------------------------------------------------------------------ the bound library
struct Api {
    decltype(&mni_b200_matmul_fwd) matmul_fwd;
    decltype(&mni_b200_matmul_bwd) matmul_bwd;
    decltype(&mni_b200_matmul_bias_gelu_fwd) matmul_bias_gelu_fwd;
    decltype(&mni_b200_add_bias) add_bias;
    decltype(&mni_b200_add_bias_bwd) add_bias_bwd;
    decltype(&mni_b200_bias_gelu) bias_gelu;
    decltype(&mni_b200_bias_gelu_bwd) bias_gelu_bwd;
    decltype(&mni_b200_softmax_fwd) softmax_fwd;
    decltype(&mni_b200_softmax_bwd) softmax_bwd;
    decltype(&mni_b200_contiguous) contiguous;
    decltype(&mni_b200_grad_norm_sq) grad_norm_sq;
    decltype(&mni_b200_clip_and_step) clip_and_step;
};
Api g_api;
bool g_bound = false;

bool ensure_bound() {
    if (g_bound) return true;
    if (!g_loader) { PyErr_SetString(PyExc_RuntimeError, "host module is not set up"); return false; }
    PyObject *r = PyObject_CallNoArgs(g_loader);
    if (!r) return false;
    Py_DECREF(r);
    if (!g_bound) { PyErr_SetString(PyExc_RuntimeError, "the library was not bound"); return false; }
    return true;
}

bool check(int status) {
    if (status == MNI_B200_OK) return true;
    PyObject *r = PyObject_CallFunction(g_raise_status, "i", status);
    Py_XDECREF(r);
    if (r) PyErr_Format(PyExc_RuntimeError, "mni_b200 call failed with status %d", status);
    return false;
}

void *current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// A C++ exception (torch's: no driver, no device, out of memory) becomes a Python one instead of ending the process.
template <PyObject *(*FN)(PyObject *, PyObject *)>
PyObject *guarded(PyObject *self, PyObject *arg) {
    try {
        return FN(self, arg);
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}
template <PyObject *(*FN)(PyObject *, PyObject *const *, Py_ssize_t)>
PyObject *guarded_fast(PyObject *self, PyObject *const *args, Py_ssize_t nargs) {
    try {
        return FN(self, args, nargs);
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

// ------------------------------------------------------------------ tensor object
bool row_major(const Dims &shape, const Dims &stride) {
    if (shape.size() != stride.size()) return false;
    int64_t acc = 1;
    for (size_t i = shape.size(); i-- > 0;) {
        if (stride[i] != acc) return false;
        acc *= shape[i];
    }
    return true;
}
int64_t numel(const Dims &shape) {
    int64_t n = 1;
    for (int64_t s : shape) n *= s;
    return n;
}
void set_row_major(TensorObj *t) {
    t->stride.resize(t->shape.size());
    int64_t acc = 1;
    for (size_t i = t->shape.size(); i-- > 0;) {
        t->stride[i] = acc;
        acc *= t->shape[i];
    }
    t->contiguous = true;
}
float *data(const TensorObj *t) { return static_cast<float *>(t->flat.data_ptr()); }
// Whether the tensor has been given its storage (an object that was created without being initialised has none).
bool has_storage(const TensorObj *t) {
    if (t->flat.defined()) return true;
    PyErr_SetString(PyExc_AttributeError, "storage");
    return false;
}

// How an item that is no int becomes one: as int() does (extents and strides of a new tensor), as an index (dimensions), or only
// if it equals one (a shape that is compared with a tensor's; -1, which no extent is, if it does not).
enum class Ints { kConvert, kIndex, kEqual };
bool parse_ints(PyObject *seq, Dims &out, Ints how = Ints::kConvert) {
    PyObject *fast = PySequence_Fast(seq, "expected a sequence of integers");
    if (!fast) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
    out.resize(static_cast<size_t>(n));
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject *item = PySequence_Fast_GET_ITEM(fast, i);
        long long v;
        if (PyLong_CheckExact(item)) {
            v = PyLong_AsLongLong(item);
        } else {
            PyObject *as_int = how == Ints::kIndex ? PyNumber_Index(item) : PyNumber_Long(item);
            if (!as_int) { Py_DECREF(fast); return false; }
            v = PyLong_AsLongLong(as_int);
            const int equal = how == Ints::kEqual ? PyObject_RichCompareBool(as_int, item, Py_EQ) : 1;
            Py_DECREF(as_int);
            if (equal < 0) { Py_DECREF(fast); return false; }
            if (equal == 0) v = -1;
        }
        if (v == -1 && PyErr_Occurred()) { Py_DECREF(fast); return false; }
        out[static_cast<size_t>(i)] = v;
    }
    Py_DECREF(fast);
    return true;
}
PyObject *tuple_of(const Dims &d) {
    PyObject *t = PyTuple_New(static_cast<Py_ssize_t>(d.size()));
    if (!t) return nullptr;
    for (size_t i = 0; i < d.size(); ++i) {
        PyObject *v = PyLong_FromLongLong(d[i]);
        if (!v) { Py_DECREF(t); return nullptr; }
        PyTuple_SET_ITEM(t, static_cast<Py_ssize_t>(i), v);
    }
    return t;
}

TensorObj *alloc_tensor(PyTypeObject *type) {
    TensorObj *t = reinterpret_cast<TensorObj *>(type->tp_alloc(type, 0));
    if (!t) return nullptr;
    new (&t->flat) at::Tensor();
    new (&t->shape) Dims();
    new (&t->stride) Dims();
    t->contiguous = true;
    t->shape_tuple = t->stride_tuple = nullptr;
    return t;
}
PyObject *tensor_new(PyTypeObject *type, PyObject *, PyObject *) { return reinterpret_cast<PyObject *>(alloc_tensor(type)); }
void tensor_dealloc(PyObject *self) {
    TensorObj *t = reinterpret_cast<TensorObj *>(self);
    t->flat.~Tensor();
    t->shape.~Dims();
    t->stride.~Dims();
    Py_XDECREF(t->shape_tuple);
    Py_XDECREF(t->stride_tuple);
    Py_TYPE(self)->tp_free(self);
}

bool set_storage(TensorObj *t, PyObject *storage) {
    if (THPVariable_Check(storage)) {
        const at::Tensor &flat = THPVariable_Unpack(storage);
        if (flat.scalar_type() == at::kFloat && flat.is_cuda() && flat.dim() == 1) {
            t->flat = flat;
            return true;
        }
    }
    PyErr_SetString(PyExc_TypeError, "storage must be a flat float32 CUDA tensor");
    return false;
}

int tensor_init(PyObject *self, PyObject *args, PyObject *kwargs) {
    static const char *names[] = {"storage", "shape", "strides", nullptr};
    PyObject *storage, *shape, *strides = Py_None;
    if (!PyArg_ParseTupleAndKeywords(args, kwargs, "OO|O", const_cast<char **>(names), &storage, &shape, &strides)) return -1;
    TensorObj *t = reinterpret_cast<TensorObj *>(self);
    if (!set_storage(t, storage) || !parse_ints(shape, t->shape)) return -1;
    Py_CLEAR(t->shape_tuple);
    Py_CLEAR(t->stride_tuple);
    if (strides == Py_None) {
        set_row_major(t);
    } else {
        if (!parse_ints(strides, t->stride)) return -1;
        t->contiguous = row_major(t->shape, t->stride);
    }
    return 0;
}

// Uninitialised row-major tensor on `device`; the storage holds one element at least, so that it has an address.
TensorObj *new_tensor(const Dims &shape, const at::Device &device) {
    TensorObj *t = alloc_tensor(g_class);
    if (!t) return nullptr;
    try {
        t->shape = shape;
        set_row_major(t);
        const int64_t n = std::max<int64_t>(numel(shape), 1);
        t->flat = at::Tensor(at::detail::empty_cuda({n}, at::kFloat, device, std::nullopt));
    } catch (...) {
        Py_DECREF(t);
        torch::translate_exception_to_python(std::current_exception());   // torch.OutOfMemoryError and the like
        return nullptr;
    }
    return t;
}

TensorObj *as_tensor(PyObject *o, const char *what) {
    if (!PyObject_TypeCheck(o, g_class)) {
        PyErr_Format(PyExc_TypeError, "%s must be a DeviceTensor, not %s", what, Py_TYPE(o)->tp_name);
        return nullptr;
    }
    TensorObj *t = reinterpret_cast<TensorObj *>(o);
    return has_storage(t) ? t : nullptr;
}

bool make_view(const TensorObj *t, mni_b200_view &v) {
    if (t->shape.size() > MNI_B200_MAX_DIMS) {
        char msg[64];
        snprintf(msg, sizeof(msg), "%zu dims exceed the ABI's %d", t->shape.size(), MNI_B200_MAX_DIMS);
        PyObject *r = PyObject_CallFunction(g_raise_status, "is", static_cast<int>(MNI_B200_ERR_ARG), msg);
        Py_XDECREF(r);
        return false;
    }
    v.ptr = data(t);
    v.ndim = static_cast<int32_t>(t->shape.size());
    for (int i = 0; i < v.ndim; ++i) {
        v.shape[i] = t->shape[static_cast<size_t>(i)];
        v.stride[i] = static_cast<size_t>(i) < t->stride.size() ? t->stride[static_cast<size_t>(i)] : 0;   // none given: 0
    }
    return true;
}

// ------------------------------------------------------------------ tensor methods
PyObject *get_storage(PyObject *self, void *) {
    TensorObj *t = reinterpret_cast<TensorObj *>(self);
    return has_storage(t) ? THPVariable_Wrap(t->flat) : nullptr;
}
int put_storage(PyObject *self, PyObject *value, void *) {
    if (!value) { PyErr_SetString(PyExc_AttributeError, "storage cannot be deleted"); return -1; }
    return set_storage(reinterpret_cast<TensorObj *>(self), value) ? 0 : -1;
}
PyObject *get_dims(PyObject *self, void *which) {
    TensorObj *t = reinterpret_cast<TensorObj *>(self);
    PyObject *&cache = which ? t->stride_tuple : t->shape_tuple;
    if (!cache) cache = tuple_of(which ? t->stride : t->shape);
    Py_XINCREF(cache);
    return cache;
}
int put_dims(PyObject *self, PyObject *value, void *which) {
    TensorObj *t = reinterpret_cast<TensorObj *>(self);
    if (!value) { PyErr_SetString(PyExc_AttributeError, "shape and strides cannot be deleted"); return -1; }
    if (!parse_ints(value, which ? t->stride : t->shape)) return -1;
    Py_CLEAR(which ? t->stride_tuple : t->shape_tuple);
    t->contiguous = row_major(t->shape, t->stride);
    return 0;
}
PyObject *get_size(PyObject *self, void *) { return PyLong_FromLongLong(numel(reinterpret_cast<TensorObj *>(self)->shape)); }
PyObject *get_ndim(PyObject *self, void *) {
    return PyLong_FromSize_t(reinterpret_cast<TensorObj *>(self)->shape.size());
}
PyObject *get_ptr(PyObject *self, void *) {
    TensorObj *t = reinterpret_cast<TensorObj *>(self);
    return has_storage(t) ? PyLong_FromVoidPtr(data(t)) : nullptr;
}
PyObject *is_contiguous(PyObject *self, PyObject *) {
    return PyBool_FromLong(reinterpret_cast<TensorObj *>(self)->contiguous);
}

PyObject *permuted(TensorObj *t, const Dims &dims) {
    const size_t nd = t->shape.size();
    bool ok = dims.size() == nd;
    std::vector<char> seen(nd, 0);
    for (size_t i = 0; ok && i < nd; ++i) {
        ok = dims[i] >= 0 && dims[i] < static_cast<int64_t>(nd) && !seen[static_cast<size_t>(dims[i])];
        if (ok) seen[static_cast<size_t>(dims[i])] = 1;
    }
    if (!ok) {
        PyObject *given = tuple_of(dims), *list = given ? PySequence_List(given) : nullptr;
        if (list) PyErr_Format(PyExc_ValueError, "invalid permutation %R", list);
        Py_XDECREF(list);
        Py_XDECREF(given);
        return nullptr;
    }
    if (t->stride.size() < nd) {
        PyErr_SetString(PyExc_IndexError, "the tensor has fewer strides than dimensions");
        return nullptr;
    }
    TensorObj *r = alloc_tensor(g_class);
    if (!r) return nullptr;
    r->flat = t->flat;
    r->shape.resize(nd);
    r->stride.resize(nd);
    for (size_t i = 0; i < nd; ++i) {
        r->shape[i] = t->shape[static_cast<size_t>(dims[i])];
        r->stride[i] = t->stride[static_cast<size_t>(dims[i])];
    }
    r->contiguous = row_major(r->shape, r->stride);
    return reinterpret_cast<PyObject *>(r);
}
PyObject *permute(PyObject *self, PyObject *arg) {
    Dims dims;
    if (!has_storage(reinterpret_cast<TensorObj *>(self)) || !parse_ints(arg, dims, Ints::kIndex)) return nullptr;
    return permuted(reinterpret_cast<TensorObj *>(self), dims);
}

// New reference to `t` itself when it is contiguous, else to a gathered copy.
TensorObj *contiguous_of(TensorObj *t) {
    if (t->contiguous) { Py_INCREF(t); return t; }
    if (!has_storage(t) || !ensure_bound()) return nullptr;
    TensorObj *out = new_tensor(t->shape, t->flat.device());
    mni_b200_view v;
    if (!out || !make_view(t, v)) { Py_XDECREF(out); return nullptr; }
    int rc;
    void *stream = current_stream();
    float *dst = data(out);
    Py_BEGIN_ALLOW_THREADS
    rc = g_api.contiguous(&v, dst, stream);
    Py_END_ALLOW_THREADS
    if (!check(rc)) { Py_DECREF(out); return nullptr; }
    return out;
}
PyObject *contiguous(PyObject *self, PyObject *) {
    return reinterpret_cast<PyObject *>(contiguous_of(reinterpret_cast<TensorObj *>(self)));
}

// empty(shape, device): the device is a torch.device, a string torch.device takes, an index or None (the current one).
bool parse_device(PyObject *o, at::Device &out) {
    if (o == nullptr || o == Py_None) {
        out = at::Device(at::kCUDA, c10::cuda::current_device());
        return true;
    }
    if (THPDevice_Check(o)) {
        out = reinterpret_cast<THPDevice *>(o)->device;
    } else if (PyLong_Check(o)) {
        out = at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(PyLong_AsLong(o)));
    } else if (PyUnicode_Check(o)) {
        try {
            out = at::Device(std::string(PyUnicode_AsUTF8(o)));
        } catch (const std::exception &e) {
            PyErr_SetString(PyExc_RuntimeError, e.what());
            return false;
        }
    } else {
        PyErr_SetString(PyExc_TypeError, "device must be a torch.device, a string, an index or None");
        return false;
    }
    if (!out.is_cuda()) { PyErr_SetString(PyExc_TypeError, "storage must be a flat float32 CUDA tensor"); return false; }
    if (!out.has_index()) out = at::Device(at::kCUDA, c10::cuda::current_device());
    return true;
}
PyObject *empty(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs < 1 || nargs > 2) { PyErr_SetString(PyExc_TypeError, "empty(shape, device=None)"); return nullptr; }
    Dims shape;
    at::Device device(at::kCPU);
    if (!parse_ints(args[0], shape)) return nullptr;
    try {
        if (!parse_device(nargs == 2 ? args[1] : nullptr, device)) return nullptr;
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
    return reinterpret_cast<PyObject *>(new_tensor(shape, device));
}

PyGetSetDef tensor_getset[] = {
    {"storage", get_storage, put_storage, "flat float32 CUDA tensor that holds the elements", nullptr},
    {"shape", get_dims, put_dims, "extents", nullptr},
    {"strides", get_dims, put_dims, "element strides", reinterpret_cast<void *>(1)},
    {"size", get_size, nullptr, "number of elements", nullptr},
    {"ndim", get_ndim, nullptr, "number of dimensions", nullptr},
    {"ptr", get_ptr, nullptr, "device address of the first element", nullptr},
    {nullptr, nullptr, nullptr, nullptr, nullptr}};
PyMethodDef tensor_methods[] = {
    {"is_contiguous", is_contiguous, METH_NOARGS, "whether the strides are row-major (tensor.rs:77-89)"},
    {"permute", guarded<permute>, METH_O, "stride-only permutation sharing the storage (no kernel, no copy)"},
    {"contiguous", guarded<contiguous>, METH_NOARGS, "the tensor itself, or a device gather of it (ops/layout.rs:218-231)"},
    {nullptr, nullptr, 0, nullptr}};
PyTypeObject tensor_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ------------------------------------------------------------------ operators
// Owning reference that is dropped on every way out.
struct Ref {
    TensorObj *t = nullptr;
    Ref() = default;
    explicit Ref(TensorObj *o) : t(o) {}
    ~Ref() { Py_XDECREF(t); }
    Ref(const Ref &) = delete;
    Ref &operator=(const Ref &) = delete;
    void reset(TensorObj *o) { Py_XDECREF(t); t = o; }
    void share(TensorObj *o) { Py_INCREF(o); reset(o); }
    PyObject *release() { PyObject *o = reinterpret_cast<PyObject *>(t); t = nullptr; return o; }
    explicit operator bool() const { return t != nullptr; }
};

// Output shape of a . b; raises as the reference panics (ops/matmul.rs:89, :94, utils.rs:16).
bool product_shape(TensorObj *a, TensorObj *b, Dims &out) {
    const size_t an = a->shape.size(), bn = b->shape.size();
    bool ok = an >= 2 && bn >= 2 && a->shape[an - 1] == b->shape[bn - 2];
    if (ok) {
        const size_t nd = std::max(an, bn);
        out.resize(nd);
        for (size_t i = 0; ok && i + 2 < nd; ++i) {
            const int64_t da = i < nd - an ? 1 : a->shape[i - (nd - an)], db = i < nd - bn ? 1 : b->shape[i - (nd - bn)];
            ok = da == db || da == 1 || db == 1;
            out[i] = da == 1 ? db : da;
        }
        out[nd - 2] = a->shape[an - 2];
        out[nd - 1] = b->shape[bn - 1];
    }
    if (ok) return true;
    PyObject *r = PyObject_CallFunctionObjArgs(g_check_shapes, reinterpret_cast<PyObject *>(a), reinterpret_cast<PyObject *>(b), nullptr);
    Py_XDECREF(r);
    if (r) PyErr_SetString(PyExc_ValueError, "operands do not multiply");
    return false;
}
bool vector_of(const TensorObj *t, int64_t n) { return t->shape.size() == 1 && t->shape[0] == n; }
int64_t leading_rows(const Dims &shape) {
    int64_t n = 1;
    for (size_t i = 0; i + 1 < shape.size(); ++i) n *= shape[i];
    return n;
}
// An output the caller passed, or a new one.
bool output(PyObject *given, const Dims &shape, const at::Device &device, const char *what, Ref &out) {
    if (given == Py_None) {
        out.reset(new_tensor(shape, device));
    } else {
        TensorObj *t = as_tensor(given, what);
        if (t) out.share(t);
    }
    return static_cast<bool>(out);
}

#define ARGS(n, text)                                                                     \
    if (nargs != (n)) { PyErr_SetString(PyExc_TypeError, text); return nullptr; }         \
    if (!ensure_bound()) return nullptr
#define TENSOR(var, index, what)                        \
    TensorObj *var = as_tensor(args[index], what);      \
    if (!var) return nullptr
#define CALL(expr)                          \
    int rc;                                 \
    Py_BEGIN_ALLOW_THREADS                  \
    rc = (expr);                            \
    Py_END_ALLOW_THREADS                    \
    if (!check(rc)) return nullptr

// Flags and truth values.  Anything else than a number (or a value without a truth) is an error before anything is launched.
bool parse_flags(PyObject *o, uint32_t &out) {
    const unsigned long v = PyLong_AsUnsignedLongMask(o);
    if (v == static_cast<unsigned long>(-1) && PyErr_Occurred()) return false;
    out = static_cast<uint32_t>(v);
    return true;
}
bool parse_truth(PyObject *o, bool &out) {
    const int v = PyObject_IsTrue(o);
    out = v == 1;
    return v >= 0;
}

// matmul(a, b, bias, flags, out)
PyObject *op_matmul(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(5, "matmul(a, b, bias, flags, out)");
    uint32_t flags;
    if (!parse_flags(args[3], flags)) return nullptr;
    TENSOR(a, 0, "a");
    TENSOR(b, 1, "b");
    Dims shape;
    if (!product_shape(a, b, shape)) return nullptr;
    TensorObj *bias = nullptr;
    if (args[2] != Py_None) {
        bias = as_tensor(args[2], "bias");
        if (!bias) return nullptr;
        if (!vector_of(bias, shape.back()) || !bias->contiguous) {
            PyErr_SetString(PyExc_ValueError, "bias must be a contiguous [N] vector");
            return nullptr;
        }
    }
    Ref out;
    if (!output(args[4], shape, a->flat.device(), "out", out)) return nullptr;
    if (args[4] != Py_None && (out.t->shape != shape || !out.t->contiguous)) {
        PyErr_SetString(PyExc_ValueError, "out must be contiguous with the broadcast output shape");
        return nullptr;
    }
    mni_b200_view va, vb;
    if (!make_view(a, va) || !make_view(b, vb)) return nullptr;
    float *c = data(out.t);
    const float *bias_ptr = bias ? data(bias) : nullptr;
    void *stream = current_stream();
    CALL(g_api.matmul_fwd(&va, &vb, c, bias_ptr, flags, stream));
    return out.release();
}

// matmul_backward(grad, a, b, flags, need_da, need_db, want_dbias, da, db, dbias)
PyObject *op_matmul_backward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(10, "matmul_backward(grad, a, b, flags, need_da, need_db, want_dbias, da, db, dbias)");
    uint32_t flags;
    bool need_da, need_db, want_dbias;
    if (!parse_flags(args[3], flags) || !parse_truth(args[4], need_da) || !parse_truth(args[5], need_db) ||
        !parse_truth(args[6], want_dbias))
        return nullptr;
    TENSOR(grad, 0, "grad");
    TENSOR(a, 1, "a");
    TENSOR(b, 2, "b");
    Dims shape;
    if (!product_shape(a, b, shape)) return nullptr;
    if (grad->shape != shape) {
        PyObject *have = tuple_of(grad->shape), *want = tuple_of(shape);
        if (have && want) PyErr_Format(PyExc_ValueError, "grad has shape %R, forward output is %R", have, want);
        Py_XDECREF(have);
        Py_XDECREF(want);
        return nullptr;
    }
    const at::Device device = a->flat.device();
    Ref da, db, dbias;
    if (need_da && !output(args[7], a->shape, device, "da", da)) return nullptr;
    if (need_db && !output(args[8], b->shape, device, "db", db)) return nullptr;
    if (want_dbias && !output(args[9], Dims{shape.back()}, device, "dbias", dbias)) return nullptr;
    mni_b200_view va, vb, vg;
    if (!make_view(a, va) || !make_view(b, vb) || !make_view(grad, vg)) return nullptr;
    float *pa = da ? data(da.t) : nullptr, *pb = db ? data(db.t) : nullptr, *pbias = dbias ? data(dbias.t) : nullptr;
    void *stream = current_stream();
    CALL(g_api.matmul_bwd(&va, &vb, &vg, pa, pb, pbias, flags, stream));
    // a gradient that is not needed comes back as it was passed in
    PyObject *results[3];
    Ref *mine[3] = {&da, &db, &dbias};
    const int count = want_dbias ? 3 : 2;
    for (int i = 0; i < count; ++i) {
        results[i] = *mine[i] ? mine[i]->release() : (Py_INCREF(args[7 + i]), args[7 + i]);
    }
    PyObject *tuple = PyTuple_New(count);
    for (int i = 0; i < count; ++i) {
        if (tuple) PyTuple_SET_ITEM(tuple, i, results[i]);
        else Py_DECREF(results[i]);
    }
    return tuple;
}

PyObject *pair_of(Ref &x, Ref &y) {
    PyObject *tuple = PyTuple_New(2);
    if (!tuple) return nullptr;
    PyTuple_SET_ITEM(tuple, 0, x.release());
    PyTuple_SET_ITEM(tuple, 1, y.release());
    return tuple;
}

// add(a, b): [.., N] + [N]; the caller has checked the shapes
PyObject *op_add(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(2, "add(a, b)");
    TENSOR(a0, 0, "a");
    TENSOR(b0, 1, "b");
    if (a0->shape.empty() || !vector_of(b0, a0->shape.back())) {
        PyErr_SetString(PyExc_NotImplementedError, "only the Linear bias add ([..., N] + [N]) is on this path");
        return nullptr;
    }
    Ref a(contiguous_of(a0)), b(a ? contiguous_of(b0) : nullptr);
    if (!a || !b) return nullptr;
    Ref out(new_tensor(a.t->shape, a.t->flat.device()));
    if (!out) return nullptr;
    const float *pa = data(a.t), *pb = data(b.t);
    float *po = data(out.t);
    const int64_t rows = leading_rows(a.t->shape), n = a.t->shape.back();
    void *stream = current_stream();
    CALL(g_api.add_bias(pa, pb, po, rows, n, stream));
    return out.release();
}

// add_backward(grad, a_shape, b_shape, flags)
PyObject *op_add_backward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(4, "add_backward(grad, a_shape, b_shape, flags)");
    uint32_t flags;
    if (!parse_flags(args[3], flags)) return nullptr;
    TENSOR(grad, 0, "grad");
    Dims a_shape, b_shape;
    if (!parse_ints(args[1], a_shape, Ints::kEqual) || !parse_ints(args[2], b_shape, Ints::kEqual)) return nullptr;
    if (grad->shape != a_shape || b_shape.size() != 1 || grad->shape.empty() || b_shape[0] != grad->shape.back()) {
        PyErr_SetString(PyExc_NotImplementedError, "only the Linear bias add ([..., N] + [N]) is on this path");
        return nullptr;
    }
    Ref g(contiguous_of(grad));
    if (!g) return nullptr;
    Ref ga(new_tensor(a_shape, g.t->flat.device())), gb(ga ? new_tensor(b_shape, g.t->flat.device()) : nullptr);
    if (!ga || !gb) return nullptr;
    const float *pg = data(g.t);
    float *pa = data(ga.t), *pb = data(gb.t);
    const int64_t rows = leading_rows(a_shape), n = b_shape[0];
    void *stream = current_stream();
    CALL(g_api.add_bias_bwd(pg, pa, pb, rows, n, flags, stream));
    return pair_of(ga, gb);
}

// bias_gelu(x, bias)
PyObject *op_bias_gelu(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(2, "bias_gelu(x, bias)");
    TENSOR(x0, 0, "x");
    TENSOR(b0, 1, "bias");
    if (x0->shape.empty() || !vector_of(b0, x0->shape.back())) {
        PyErr_SetString(PyExc_ValueError, "bias must be a [C] vector matching x's last dim");
        return nullptr;
    }
    Ref x(contiguous_of(x0)), b(x ? contiguous_of(b0) : nullptr);
    if (!x || !b) return nullptr;
    Ref out(new_tensor(x.t->shape, x.t->flat.device()));
    if (!out) return nullptr;
    const float *px = data(x.t), *pb = data(b.t);
    float *po = data(out.t);
    const int64_t rows = leading_rows(x.t->shape), n = x.t->shape.back();
    void *stream = current_stream();
    CALL(g_api.bias_gelu(px, pb, po, rows, n, stream));
    return out.release();
}

// bias_gelu_backward(grad, x, bias, flags)
PyObject *op_bias_gelu_backward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(4, "bias_gelu_backward(grad, x, bias, flags)");
    uint32_t flags;
    if (!parse_flags(args[3], flags)) return nullptr;
    TENSOR(g0, 0, "grad");
    TENSOR(x0, 1, "x");
    TENSOR(b0, 2, "bias");
    if (g0->shape != x0->shape || x0->shape.empty() || !vector_of(b0, x0->shape.back())) {
        PyErr_SetString(PyExc_ValueError, "grad must have x's shape and bias must be [C]");
        return nullptr;
    }
    Ref g(contiguous_of(g0)), x(g ? contiguous_of(x0) : nullptr), b(x ? contiguous_of(b0) : nullptr);
    if (!g || !x || !b) return nullptr;
    const at::Device device = x.t->flat.device();
    Ref dx(new_tensor(x.t->shape, device)), dbias(dx ? new_tensor(b.t->shape, device) : nullptr);
    if (!dx || !dbias) return nullptr;
    const float *pg = data(g.t), *px = data(x.t), *pb = data(b.t);
    float *pdx = data(dx.t), *pdb = data(dbias.t);
    const int64_t rows = leading_rows(x.t->shape), n = x.t->shape.back();
    void *stream = current_stream();
    CALL(g_api.bias_gelu_bwd(pg, px, pb, pdx, pdb, rows, n, flags, stream));
    return pair_of(dx, dbias);
}

// matmul_bias_gelu(a, b, bias, flags, want_pre)
PyObject *op_matmul_bias_gelu(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(5, "matmul_bias_gelu(a, b, bias, flags, want_pre)");
    uint32_t flags;
    bool want_pre;
    if (!parse_flags(args[3], flags) || !parse_truth(args[4], want_pre)) return nullptr;
    TENSOR(a, 0, "a");
    TENSOR(b, 1, "b");
    TENSOR(bias, 2, "bias");
    Dims shape;
    if (!product_shape(a, b, shape)) return nullptr;
    if (!vector_of(bias, shape.back()) || !bias->contiguous) {
        PyErr_SetString(PyExc_ValueError, "bias must be a contiguous [N] vector");
        return nullptr;
    }
    Ref pre, out;
    if (want_pre) {
        pre.reset(new_tensor(shape, a->flat.device()));
        if (!pre) return nullptr;
    }
    out.reset(new_tensor(shape, a->flat.device()));
    if (!out) return nullptr;
    mni_b200_view va, vb;
    if (!make_view(a, va) || !make_view(b, vb)) return nullptr;
    const float *pb = data(bias);
    float *pp = pre ? data(pre.t) : nullptr, *po = data(out.t);
    void *stream = current_stream();
    CALL(g_api.matmul_bias_gelu_fwd(&va, &vb, pb, pp, po, flags, stream));
    PyObject *tuple = PyTuple_New(2);
    if (!tuple) return nullptr;
    PyTuple_SET_ITEM(tuple, 0, pre ? pre.release() : (Py_INCREF(Py_None), Py_None));
    PyTuple_SET_ITEM(tuple, 1, out.release());
    return tuple;
}

// [outer, size, inner] of a softmax over dimension `dim`
bool softmax_split(const TensorObj *t, PyObject *dim, int64_t &outer, int64_t &size, int64_t &inner) {
    const long long nd = static_cast<long long>(t->shape.size());
    const long long given = PyLong_AsLongLong(dim);
    if (given == -1 && PyErr_Occurred()) return false;
    const long long d = given < 0 ? given + nd : given;
    if (d < 0 || d >= nd) {
        PyObject *shape = tuple_of(t->shape);
        if (shape) PyErr_Format(PyExc_IndexError, "softmax dim %lld out of range for shape %R", given, shape);
        Py_XDECREF(shape);
        return false;
    }
    outer = inner = 1;
    for (long long i = 0; i < d; ++i) outer *= t->shape[static_cast<size_t>(i)];
    for (long long i = d + 1; i < nd; ++i) inner *= t->shape[static_cast<size_t>(i)];
    outer = std::max<int64_t>(outer, 1);
    inner = std::max<int64_t>(inner, 1);
    size = t->shape[static_cast<size_t>(d)];
    return true;
}

// softmax(a, dim)
PyObject *op_softmax(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(2, "softmax(a, dim)");
    TENSOR(a0, 0, "a");
    Ref a(contiguous_of(a0));
    int64_t outer, size, inner;
    if (!a || !softmax_split(a.t, args[1], outer, size, inner)) return nullptr;
    Ref out(new_tensor(a.t->shape, a.t->flat.device()));
    if (!out) return nullptr;
    const float *pa = data(a.t);
    float *po = data(out.t);
    void *stream = current_stream();
    CALL(g_api.softmax_fwd(pa, po, outer, size, inner, stream));
    return out.release();
}

// softmax_backward(grad, out, dim)
PyObject *op_softmax_backward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(3, "softmax_backward(grad, out, dim)");
    TENSOR(g0, 0, "grad");
    TENSOR(s0, 1, "out");
    if (g0->shape != s0->shape) {
        PyErr_SetString(PyExc_ValueError, "grad and out must have the same shape");
        return nullptr;
    }
    Ref g(contiguous_of(g0)), s(g ? contiguous_of(s0) : nullptr);
    int64_t outer, size, inner;
    if (!g || !s || !softmax_split(s.t, args[2], outer, size, inner)) return nullptr;
    Ref dx(new_tensor(s.t->shape, s.t->flat.device()));
    if (!dx) return nullptr;
    const float *pg = data(g.t), *ps = data(s.t);
    float *pd = data(dx.t);
    void *stream = current_stream();
    CALL(g_api.softmax_bwd(pg, ps, pd, outer, size, inner, stream));
    return dx.release();
}

// permute_backward(grad, dims, orig_shape): the gather of the inverse-permuted view
PyObject *op_permute_backward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(3, "permute_backward(grad, dims, orig_shape)");
    TENSOR(grad, 0, "grad");
    Dims dims, orig;
    if (!parse_ints(args[1], dims, Ints::kIndex) || !parse_ints(args[2], orig, Ints::kEqual)) return nullptr;
    const size_t nd = dims.size();
    bool ok = grad->shape.size() == nd;
    Dims inverse, want;
    inverse.resize(nd);
    want.resize(nd);
    for (size_t i = 0; i < nd; ++i) {
        if (dims[i] < 0 || static_cast<size_t>(dims[i]) >= std::min(nd, orig.size())) {
            PyErr_SetString(PyExc_IndexError, "permutation index out of range");
            return nullptr;
        }
        inverse[static_cast<size_t>(dims[i])] = static_cast<int64_t>(i);
        want[i] = orig[static_cast<size_t>(dims[i])];
    }
    if (!ok || grad->shape != want) {
        PyObject *have = tuple_of(grad->shape), *expected = tuple_of(want);
        if (have && expected) PyErr_Format(PyExc_ValueError, "grad has shape %R, expected %R", have, expected);
        Py_XDECREF(have);
        Py_XDECREF(expected);
        return nullptr;
    }
    PyObject *view = permuted(grad, inverse);
    if (!view) return nullptr;
    TensorObj *out = contiguous_of(reinterpret_cast<TensorObj *>(view));
    Py_DECREF(view);
    return reinterpret_cast<PyObject *>(out);
}

// ------------------------------------------------------------------ optimizer
// Addresses and sizes of a list of contiguous tensors.
struct TensorList {
    std::vector<float *> ptr;
    std::vector<int64_t> n;
    bool parse(PyObject *seq, const char *not_contiguous) {
        PyObject *fast = PySequence_Fast(seq, "expected a sequence of tensors");
        if (!fast) return false;
        const Py_ssize_t count = PySequence_Fast_GET_SIZE(fast);
        ptr.reserve(static_cast<size_t>(count));
        n.reserve(static_cast<size_t>(count));
        for (Py_ssize_t i = 0; i < count; ++i) {
            TensorObj *t = as_tensor(PySequence_Fast_GET_ITEM(fast, i), "every element");
            if (t && !t->contiguous) { PyErr_SetString(PyExc_ValueError, not_contiguous); t = nullptr; }
            if (!t) { Py_DECREF(fast); return false; }
            ptr.push_back(data(t));
            n.push_back(numel(t->shape));
        }
        Py_DECREF(fast);
        return true;
    }
};

// grad_norm_sq(grads, address of a device double)
PyObject *op_grad_norm_sq(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(2, "grad_norm_sq(grads, out)");
    TensorList grads;
    if (!grads.parse(args[0], "gradients must be contiguous")) return nullptr;
    double *out = static_cast<double *>(PyLong_AsVoidPtr(args[1]));
    if (!out && PyErr_Occurred()) return nullptr;
    void *stream = current_stream();
    CALL(g_api.grad_norm_sq(static_cast<int64_t>(grads.ptr.size()), grads.ptr.data(), grads.n.data(), out, stream));
    Py_RETURN_NONE;
}

// clip_and_step(params, ms, vs, grads, lr, beta1, beta2, eps, weight_decay, step, max_grad_norm) -> norm
PyObject *op_clip_and_step(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    ARGS(11, "clip_and_step(params, ms, vs, grads, lr, beta1, beta2, eps, weight_decay, step, max_grad_norm)");
    TensorList p, m, v, g;
    const char *text = "adamw_step needs contiguous tensors";
    if (!g.parse(args[3], "gradients must be contiguous") || !p.parse(args[0], text) || !m.parse(args[1], text) ||
        !v.parse(args[2], text))
        return nullptr;
    const size_t count = p.ptr.size();
    if (m.ptr.size() != count || v.ptr.size() != count || g.ptr.size() != count) {
        PyErr_SetString(PyExc_ValueError, "params, ms, vs and grads must have the same length");
        return nullptr;
    }
    if (p.n != m.n || p.n != v.n || p.n != g.n) {
        PyErr_SetString(PyExc_ValueError, "param, m, v and grad must have the same size");
        return nullptr;
    }
    float hyper[5];
    for (int i = 0; i < 5; ++i) hyper[i] = static_cast<float>(PyFloat_AsDouble(args[4 + i]));
    const uint32_t step = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(args[9]));
    const float max_norm = static_cast<float>(PyFloat_AsDouble(args[10]));
    if (PyErr_Occurred()) return nullptr;
    float norm = 0.f;
    void *stream = current_stream();
    CALL(g_api.clip_and_step(static_cast<int64_t>(count), p.ptr.data(), m.ptr.data(), v.ptr.data(), g.ptr.data(), p.n.data(),
                             hyper[0], hyper[1], hyper[2], hyper[3], hyper[4], step, max_norm, &norm, stream));
    return PyFloat_FromDouble(static_cast<double>(norm));
}

// ------------------------------------------------------------------ module
// setup(cls, loader, raise_status, check_shapes): the Python side of the bindings
PyObject *setup(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 4 || !PyType_Check(args[0]) || !PyType_IsSubtype(reinterpret_cast<PyTypeObject *>(args[0]), &tensor_type)) {
        PyErr_SetString(PyExc_TypeError, "setup(cls, loader, raise_status, check_shapes)");
        return nullptr;
    }
    for (int i = 0; i < 4; ++i) Py_INCREF(args[i]);
    g_class = reinterpret_cast<PyTypeObject *>(args[0]);
    g_loader = args[1];
    g_raise_status = args[2];
    g_check_shapes = args[3];
    Py_RETURN_NONE;
}

// bind({name: address}): the library's entry points
PyObject *bind(PyObject *, PyObject *table) {
    struct { const char *name; void **slot; } entries[] = {
#define ENTRY(field) {"mni_b200_" #field, reinterpret_cast<void **>(&g_api.field)}
        ENTRY(matmul_fwd), ENTRY(matmul_bwd), ENTRY(matmul_bias_gelu_fwd), ENTRY(add_bias), ENTRY(add_bias_bwd),
        ENTRY(bias_gelu), ENTRY(bias_gelu_bwd), ENTRY(softmax_fwd), ENTRY(softmax_bwd), ENTRY(contiguous),
        ENTRY(grad_norm_sq), ENTRY(clip_and_step),
#undef ENTRY
    };
    for (auto &e : entries) {
        PyObject *address = PyDict_GetItemString(table, e.name);
        void *p = address ? PyLong_AsVoidPtr(address) : nullptr;
        if (!p) {
            if (!PyErr_Occurred()) PyErr_Format(PyExc_ImportError, "%s has no address", e.name);
            return nullptr;
        }
        *e.slot = p;
    }
    g_bound = true;
    Py_RETURN_NONE;
}

PyObject *raw_stream(PyObject *, PyObject *) { return PyLong_FromVoidPtr(current_stream()); }

#define FAST(name, fn, doc) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded_fast<fn>)), METH_FASTCALL, doc}
PyMethodDef module_methods[] = {
    FAST("setup", setup, "registers the Python side"),
    {"bind", bind, METH_O, "binds the library's entry points"},
    {"current_stream", guarded<raw_stream>, METH_NOARGS, "address of the current CUDA stream of the current device"},
    FAST("empty", empty, "uninitialised row-major tensor"),
    FAST("matmul", op_matmul, "ops.matmul"),
    FAST("matmul_backward", op_matmul_backward, "ops.matmul_backward"),
    FAST("add", op_add, "ops.add"),
    FAST("add_backward", op_add_backward, "ops.add_backward"),
    FAST("bias_gelu", op_bias_gelu, "ops.bias_gelu"),
    FAST("bias_gelu_backward", op_bias_gelu_backward, "ops.bias_gelu_backward"),
    FAST("matmul_bias_gelu", op_matmul_bias_gelu, "ops.matmul_bias_gelu"),
    FAST("softmax", op_softmax, "ops.softmax"),
    FAST("softmax_backward", op_softmax_backward, "ops.softmax_backward"),
    FAST("permute_backward", op_permute_backward, "ops.permute_backward"),
    FAST("grad_norm_sq", op_grad_norm_sq, "squared global gradient norm into a device double"),
    FAST("clip_and_step", op_clip_and_step, "ops.clip_and_step"),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "native host side of the operator interface", -1, module_methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

#ifndef MNI_HOST_SOURCE_HASH
#define MNI_HOST_SOURCE_HASH ""
#endif

PyMODINIT_FUNC PyInit__host(void) {
    tensor_type.tp_name = "framework_b200._host.Tensor";
    tensor_type.tp_basicsize = sizeof(TensorObj);
    tensor_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE;
    tensor_type.tp_new = tensor_new;
    tensor_type.tp_init = tensor_init;
    tensor_type.tp_dealloc = tensor_dealloc;
    tensor_type.tp_getset = tensor_getset;
    tensor_type.tp_methods = tensor_methods;
    if (PyType_Ready(&tensor_type) < 0) return nullptr;
    PyObject *m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&tensor_type);
    if (PyModule_AddObject(m, "Tensor", reinterpret_cast<PyObject *>(&tensor_type)) < 0 ||
        PyModule_AddStringConstant(m, "source_hash", MNI_HOST_SOURCE_HASH) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
