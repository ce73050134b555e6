// The per-call half of the Python binding: torch tensors to kvc_tensor descriptors and back without going
// through Python objects for every shape and stride. A layer call of a decode step describes four tensors,
// allocates one and asks for the current stream; in Python (ctypes structures filled field by field) that was
// 25 us of a 31 us call, more than the kernels of a small step take.
//
// The entry points of libkvcache_b200.so are handed over as addresses by the package (init), so this module
// links against torch only.
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include "../../../../include/kvcache_b200.h"

namespace {

typedef kvc_status (*AttentionFn)(kvc_cache *, const kvc_tensor *, const kvc_tensor *, const kvc_tensor *, float, int32_t,
                                  const kvc_tensor *, const kvc_tensor *, void *);
typedef kvc_status (*AttentionRopeFn)(kvc_cache *, const kvc_tensor *, const kvc_tensor *, const kvc_tensor *,
                                      const kvc_rope_config *, float, int32_t, const kvc_tensor *, const kvc_tensor *, void *);
typedef kvc_status (*SdpaFn)(const kvc_tensor *, const kvc_tensor *, const kvc_tensor *, float, int32_t, const kvc_tensor *,
                             const kvc_tensor *, void *);
AttentionFn g_attention = nullptr;
AttentionRopeFn g_attention_rope = nullptr;
SdpaFn g_sdpa = nullptr;

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return KVC_F32;
        case at::kHalf: return KVC_F16;
        case at::kBFloat16: return KVC_BF16;
        case at::kInt:
        case at::kUInt32: return KVC_U32;
        case at::kBool:
        case at::kByte: return KVC_BOOL;
        default: return -1;
    }
}

// False with a Python error set when `o` is no tensor this library can describe.
bool describe(PyObject *o, kvc_tensor *out) {
    if (!THPVariable_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "expected a torch tensor");
        return false;
    }
    const at::Tensor &t = THPVariable_Unpack(o);
    const int code = dtype_code(t.scalar_type());
    if (code < 0) {
        PyErr_Format(PyExc_KeyError, "no library dtype for a tensor of %s", c10::toString(t.scalar_type()));
        return false;
    }
    if (t.dim() > KVC_MAX_DIMS) {
        PyErr_Format(PyExc_IndexError, "a tensor of %d dims: at most %d", (int)t.dim(), KVC_MAX_DIMS);
        return false;
    }
    *out = kvc_tensor{};
    out->data = t.data_ptr();
    out->dtype = code;
    out->ndim = (int32_t)t.dim();
    for (int i = 0; i < out->ndim; ++i) {
        out->shape[i] = t.size(i);
        out->stride[i] = t.stride(i);
    }
    return true;
}

// On a machine without a device there is no stream to ask for: the library's call says so by its status.
void *current_stream() { return c10::cuda::device_count() > 0 ? (void *)c10::cuda::getCurrentCUDAStream().stream() : nullptr; }

void *stream_arg(PyObject *o) {     // None: the current stream, else an address
    return o == Py_None ? current_stream() : PyLong_AsVoidPtr(o);
}

// What the three attention calls share: (..., q, k, v, scale, mode, mask, out, stream) from args[at] on.
struct Call {
    kvc_tensor q, k, v, mask, out;
    const kvc_tensor *pmask = nullptr;
    float scale = 0.f;
    int mode = 0;
    void *stream = nullptr;
    PyObject *result = nullptr;     // new reference

    bool parse(PyObject *const *a) {
        if (!describe(a[0], &q) || !describe(a[1], &k) || !describe(a[2], &v)) return false;
        scale = (float)PyFloat_AsDouble(a[3]);
        mode = (int)PyLong_AsLong(a[4]);
        if (PyErr_Occurred()) return false;
        if (a[5] != Py_None) {
            if (!describe(a[5], &mask)) return false;
            pmask = &mask;
        }
        stream = stream_arg(a[7]);
        if (PyErr_Occurred()) return false;
        if (a[6] == Py_None) {
            const at::Tensor &tq = THPVariable_Unpack(a[0]);
            result = THPVariable_Wrap(at::empty(tq.sizes(), tq.options()));
        } else {
            Py_INCREF(a[6]);
            result = a[6];
        }
        if (!result || !describe(result, &out)) {
            Py_XDECREF(result);
            return false;
        }
        return true;
    }
    PyObject *finish(kvc_status st) {
        if (st == KVC_OK) return result;
        Py_DECREF(result);
        return PyLong_FromLong(st);
    }
};

template <typename F> PyObject *guarded(F &&f) {
    try {
        return f();
    } catch (const std::exception &e) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

bool want(Py_ssize_t n, Py_ssize_t expected) {
    if (n == expected) return true;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", expected, n);
    return false;
}

PyObject *py_init(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!want(n, 3)) return nullptr;
    g_attention = (AttentionFn)PyLong_AsVoidPtr(a[0]);
    g_attention_rope = (AttentionRopeFn)PyLong_AsVoidPtr(a[1]);
    g_sdpa = (SdpaFn)PyLong_AsVoidPtr(a[2]);
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

// attention(handle, q, k, v, scale, mode, mask, out, stream) -> out, or the status of a failed call
PyObject *py_attention(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!want(n, 9)) return nullptr;
    return guarded([&]() -> PyObject * {
        Call c;
        kvc_cache *h = (kvc_cache *)PyLong_AsVoidPtr(a[0]);
        if (PyErr_Occurred() || !c.parse(a + 1)) return nullptr;
        kvc_status st;
        Py_BEGIN_ALLOW_THREADS
        st = g_attention(h, &c.q, &c.k, &c.v, c.scale, c.mode, c.pmask, &c.out, c.stream);
        Py_END_ALLOW_THREADS
        return c.finish(st);
    });
}

// attention_rope(handle, dims, traditional, base, rope scale, q, k, v, scale, mode, mask, out, stream)
PyObject *py_attention_rope(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!want(n, 13)) return nullptr;
    return guarded([&]() -> PyObject * {
        Call c;
        kvc_cache *h = a[0] == Py_None ? nullptr : (kvc_cache *)PyLong_AsVoidPtr(a[0]);
        kvc_rope_config r = {};
        r.dims = (int32_t)PyLong_AsLong(a[1]);
        r.traditional = (int32_t)PyLong_AsLong(a[2]);
        r.base = (float)PyFloat_AsDouble(a[3]);
        r.scale = (float)PyFloat_AsDouble(a[4]);
        if (PyErr_Occurred() || !c.parse(a + 5)) return nullptr;
        kvc_status st;
        Py_BEGIN_ALLOW_THREADS
        st = g_attention_rope(h, &c.q, &c.k, &c.v, &r, c.scale, c.mode, c.pmask, &c.out, c.stream);
        Py_END_ALLOW_THREADS
        return c.finish(st);
    });
}

// sdpa(q, k, v, scale, mode, mask, out, stream)
PyObject *py_sdpa(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!want(n, 8)) return nullptr;
    return guarded([&]() -> PyObject * {
        Call c;
        if (!c.parse(a)) return nullptr;
        kvc_status st;
        Py_BEGIN_ALLOW_THREADS
        st = g_sdpa(&c.q, &c.k, &c.v, c.scale, c.mode, c.pmask, &c.out, c.stream);
        Py_END_ALLOW_THREADS
        return c.finish(st);
    });
}

// describe(tensor, address): fills the kvc_tensor at `address`
PyObject *py_describe(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!want(n, 2)) return nullptr;
    return guarded([&]() -> PyObject * {
        kvc_tensor *out = (kvc_tensor *)PyLong_AsVoidPtr(a[1]);
        if (PyErr_Occurred() || !describe(a[0], out)) return nullptr;
        Py_RETURN_NONE;
    });
}

// wrap(address of a kvc_tensor, device index): a tensor over the library memory it describes
PyObject *py_wrap(PyObject *, PyObject *const *a, Py_ssize_t n) {
    if (!want(n, 2)) return nullptr;
    return guarded([&]() -> PyObject * {
        const kvc_tensor *t = (const kvc_tensor *)PyLong_AsVoidPtr(a[0]);
        const long device = PyLong_AsLong(a[1]);
        if (PyErr_Occurred()) return nullptr;
        at::ScalarType st = at::kFloat;
        switch (t->dtype) {
            case KVC_F32: st = at::kFloat; break;
            case KVC_F16: st = at::kHalf; break;
            case KVC_BF16: st = at::kBFloat16; break;
            case KVC_U32: st = at::kInt; break;
            default: st = at::kByte; break;
        }
        const at::Device dev(at::kCUDA, (c10::DeviceIndex)device);
        return THPVariable_Wrap(at::from_blob(t->data, at::IntArrayRef(t->shape, t->ndim), at::IntArrayRef(t->stride, t->ndim),
                                              [](void *) {}, at::TensorOptions().dtype(st).device(dev), dev));
    });
}

PyObject *py_current_stream(PyObject *, PyObject *) {
    return guarded([&]() -> PyObject * { return PyLong_FromVoidPtr(current_stream()); });
}

PyMethodDef methods[] = {
    {"init", (PyCFunction)(void (*)(void))py_init, METH_FASTCALL, nullptr},
    {"attention", (PyCFunction)(void (*)(void))py_attention, METH_FASTCALL, nullptr},
    {"attention_rope", (PyCFunction)(void (*)(void))py_attention_rope, METH_FASTCALL, nullptr},
    {"sdpa", (PyCFunction)(void (*)(void))py_sdpa, METH_FASTCALL, nullptr},
    {"describe", (PyCFunction)(void (*)(void))py_describe, METH_FASTCALL, nullptr},
    {"wrap", (PyCFunction)(void (*)(void))py_wrap, METH_FASTCALL, nullptr},
    {"current_stream", py_current_stream, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" PyObject *PyInit__binding(void) { return PyModule_Create(&module); }
