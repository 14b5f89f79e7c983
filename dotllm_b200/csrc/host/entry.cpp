// The Python side's way to the kernel library's entry points: a CPython module that calls them without ctypes.
//
// A step of few rows is a chain of short kernels, and outside a captured graph the host launches them one by one: there, what a
// call costs on the host is what the step costs.  Through ctypes an entry point of 20 arguments takes about 2.5 us beside the launch itself, the
// tensors' addresses (`data_ptr()`, 0.1 us each) and sizes as much again, and an output from `torch.empty` 2 us.  Here a tensor is
// passed as it is, sizes and strides are read in one call, and outputs come from ATen directly.  Host time of a pass outside a graph, before and
// after: one row through a gated MLP (2 launches) 27 -> 20 us, attention of two sequences' one token each (3) 58 -> 36, in float32 (7) 83 -> 60,
// a delta rule layer's (9) 125 -> 77.
//
// Every entry point of the library has a packed form beside it (DL_PACKED in common.cuh): its arguments as 64-bit words,
// with their kinds as a text.  bind() looks both up and returns the callable.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <string.h>

namespace {

constexpr int MOST = 64;                     // arguments of an entry point, at most

struct Entry {
    int (*call)(const unsigned long long*, int);
    int n;
    char kinds[MOST + 1];                    // 'p' pointer, 'i' int, 'l' 64-bit integer, 'f' float
};

bool pack(const char kind, PyObject* o, unsigned long long* out) {
    switch (kind) {
        case 'p':
            if (o == Py_None) { *out = 0; return true; }
            if (THPVariable_Check(o)) { *out = (unsigned long long)(uintptr_t)THPVariable_Unpack(o).data_ptr(); return true; }
            [[fallthrough]];
        case 'i':
        case 'l': {
            if (PyFloat_Check(o)) {
                PyErr_SetString(PyExc_TypeError, "an integer is required, got a float");
                return false;
            }
            *out = PyLong_AsUnsignedLongLongMask(o);
            return !(*out == ~0ull && PyErr_Occurred());
        }
        default: {
            const double d = PyFloat_AsDouble(o);
            if (d == -1.0 && PyErr_Occurred()) return false;
            const float f = (float)d;
            unsigned bits;
            memcpy(&bits, &f, 4);
            *out = bits;
            return true;
        }
    }
}

// C++ exceptions stay on this side: they become Python's.
template <typename F> PyObject* guarded(F f) {
    try {
        return f();
    } catch (const std::exception& e) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyObject* call_entry(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Entry* e = static_cast<const Entry*>(PyCapsule_GetPointer(self, "dotllm.entry"));
        if (e == nullptr) return nullptr;
        if (n != e->n) {
            PyErr_Format(PyExc_TypeError, "the entry point takes %d arguments, got %zd", e->n, n);
            return nullptr;
        }
        unsigned long long packed[MOST];
        for (Py_ssize_t i = 0; i < n; ++i)
            if (!pack(e->kinds[i], args[i], packed + i)) return nullptr;
        int status;
        Py_BEGIN_ALLOW_THREADS
        status = e->call(packed, (int)n);
        Py_END_ALLOW_THREADS
        return PyLong_FromLong(status);
    });
}
PyMethodDef call_entry_def = {"entry", (PyCFunction)(void (*)(void))call_entry, METH_FASTCALL, nullptr};

// bind(library handle, name): the callable of an entry point, or None where the library has no packed form of it.
PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long handle;
    const char* name;
    if (!PyArg_ParseTuple(args, "Ks", &handle, &name)) return nullptr;
    char symbol[128];
    if (snprintf(symbol, sizeof(symbol), "%s_packed", name) >= (int)sizeof(symbol)) Py_RETURN_NONE;
    void* fn = dlsym((void*)(uintptr_t)handle, symbol);
    if (fn == nullptr || snprintf(symbol, sizeof(symbol), "%s_kinds", name) >= (int)sizeof(symbol)) Py_RETURN_NONE;
    void* kinds_fn = dlsym((void*)(uintptr_t)handle, symbol);
    if (kinds_fn == nullptr) Py_RETURN_NONE;
    Entry* e = new Entry;
    e->call = reinterpret_cast<int (*)(const unsigned long long*, int)>(fn);
    e->n = reinterpret_cast<int (*)(char*, int)>(kinds_fn)(e->kinds, MOST + 1);
    if (e->n < 0) {
        delete e;
        Py_RETURN_NONE;
    }
    PyObject* capsule = PyCapsule_New(e, "dotllm.entry", [](PyObject* c) { delete static_cast<Entry*>(PyCapsule_GetPointer(c, "dotllm.entry")); });
    if (capsule == nullptr) {
        delete e;
        return nullptr;
    }
    PyObject* callable = PyCFunction_New(&call_entry_def, capsule);
    Py_DECREF(capsule);
    return callable;
}

// kinds(library handle, name) -> text, for the check against the Python side's declarations.
PyObject* kinds(PyObject*, PyObject* args) {
    unsigned long long handle;
    const char* name;
    if (!PyArg_ParseTuple(args, "Ks", &handle, &name)) return nullptr;
    char symbol[128];
    if (snprintf(symbol, sizeof(symbol), "%s_kinds", name) >= (int)sizeof(symbol)) Py_RETURN_NONE;
    void* fn = dlsym((void*)(uintptr_t)handle, symbol);
    char text[MOST + 1];
    const int n = fn == nullptr ? -1 : reinterpret_cast<int (*)(char*, int)>(fn)(text, MOST + 1);
    if (n < 0) Py_RETURN_NONE;
    return PyUnicode_FromStringAndSize(text, n);
}

const at::Tensor* tensor_of(PyObject* o) {
    return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
}

// all_cuda(*tensors): is every one that is not None a tensor on a CUDA device?
PyObject* all_cuda(PyObject*, PyObject* const* args, Py_ssize_t n) {
    for (Py_ssize_t i = 0; i < n; ++i) {
        if (args[i] == Py_None) continue;
        const at::Tensor* t = tensor_of(args[i]);
        if (t == nullptr || !t->is_cuda()) Py_RETURN_FALSE;
    }
    Py_RETURN_TRUE;
}

// row_stride(t): the distance of a 2-D tensor's contiguous rows (of a single row at least its width), -1 where it is no such tensor.
int64_t rows_of(const at::Tensor& t) {
    if (t.dim() != 2 || (t.size(1) > 1 && t.stride(1) != 1)) return -1;
    const int64_t s = t.stride(0);
    return t.size(0) > 1 ? s : (s > t.size(1) ? s : t.size(1));
}
PyObject* row_stride(PyObject*, PyObject* o) {
    return guarded([&]() -> PyObject* {
        const at::Tensor* t = tensor_of(o);
        return PyLong_FromLongLong(t == nullptr ? -1 : rows_of(*t));
    });
}

// product(x, w): (rows, k, n, x's row stride, kind) of y = x W^T for 2-D x and contiguous W on CUDA devices; None where they do not fit or
// differ in type.  kind: 0 float32, 1 bfloat16, 2 bfloat16 as the weight-streaming kernels take it (16-byte aligned rows of x and W).
PyObject* product(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 2) {
            PyErr_SetString(PyExc_TypeError, "product(x, w)");
            return nullptr;
        }
        const at::Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]);
        if (x == nullptr || w == nullptr || !x->is_cuda() || !w->is_cuda() || x->dim() != 2 || w->dim() != 2 || x->scalar_type() != w->scalar_type() ||
            x->size(1) != w->size(1) || !w->is_contiguous())
            Py_RETURN_NONE;
        int kind;
        if (x->scalar_type() == at::kFloat) kind = 0;
        else if (x->scalar_type() == at::kBFloat16) kind = 1;
        else Py_RETURN_NONE;
        const int64_t K = x->size(1), s = rows_of(*x);
        if (s < 0) Py_RETURN_NONE;
        if (kind == 1 && K % 8 == 0 && x->stride(1) == 1 && x->stride(0) % 8 == 0 && (uintptr_t)x->data_ptr() % 16 == 0 && (uintptr_t)w->data_ptr() % 16 == 0) kind = 2;
        PyObject* out = PyTuple_New(5);
        if (out == nullptr) return nullptr;
        const int64_t v[5] = {x->size(0), K, w->size(0), s, kind};
        for (int i = 0; i < 5; ++i) {
            PyObject* o = PyLong_FromLongLong(v[i]);
            if (o == nullptr) {
                Py_DECREF(out);
                return nullptr;
            }
            PyTuple_SET_ITEM(out, i, o);
        }
        return out;
    });
}

// The lock is given up while the allocator works, as torch.empty does: it may wait for the device, or for another thread's allocation.
struct WithoutLock {
    PyThreadState* state = PyEval_SaveThread();
    ~WithoutLock() { PyEval_RestoreThread(state); }
};

// empty(rows, width, bfloat16, like): a contiguous tensor on like's device, float32 or bfloat16.
PyObject* empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor* like = n == 4 ? tensor_of(args[3]) : nullptr;
        if (like == nullptr) {
            PyErr_SetString(PyExc_TypeError, "empty(rows, width, bfloat16, like)");
            return nullptr;
        }
        const int64_t rows = PyLong_AsLongLong(args[0]), width = PyLong_AsLongLong(args[1]);
        const int half = PyObject_IsTrue(args[2]);
        if (half < 0 || ((rows == -1 || width == -1) && PyErr_Occurred())) return nullptr;
        at::Tensor t;
        {
            WithoutLock unlocked;
            t = at::empty({rows, width}, at::TensorOptions().dtype(half ? at::kBFloat16 : at::kFloat).device(like->device()));
        }
        return THPVariable_Wrap(std::move(t));
    });
}

// stream(): the current CUDA stream's handle.
PyObject* stream(PyObject*, PyObject*) {
    return guarded([&]() -> PyObject* { return PyLong_FromUnsignedLongLong((unsigned long long)(uintptr_t)c10::cuda::getCurrentCUDAStream().stream()); });
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr},
                         {"kinds", kinds, METH_VARARGS, nullptr},
                         {"all_cuda", (PyCFunction)(void (*)(void))all_cuda, METH_FASTCALL, nullptr},
                         {"row_stride", row_stride, METH_O, nullptr},
                         {"product", (PyCFunction)(void (*)(void))product, METH_FASTCALL, nullptr},
                         {"empty", (PyCFunction)(void (*)(void))empty, METH_FASTCALL, nullptr},
                         {"stream", stream, METH_NOARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "dotllm_entry", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_dotllm_entry(void) { return PyModule_Create(&module); }
