// Native half of the Python binding for the calls that take CUDA tensors: checks the tensors, reads their
// addresses and the current stream, and calls the C ABI.
//
// Done in Python, one call costs 8 us on the host (five attribute reads per tensor, the stream object, eleven
// ctypes conversions), more than the kernels of small problems take on the GPU: a 512 x 512 SpMM with N = 128
// was issued every 11 us for a kernel of 5.5 us.  Here the same work is below a microsecond.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/dlspm.h"

namespace {

// One positional argument after the other; the first failure sets a Python error and sticks.
struct Args {
    PyObject *const *v;
    Py_ssize_t n, at = 0;
    bool ok = true;

    PyObject *next()
    {
        if (!ok) return nullptr;
        if (at >= n) {
            PyErr_SetString(PyExc_TypeError, "too few arguments");
            ok = false;
            return nullptr;
        }
        return v[at++];
    }
    // integers, and numpy integers through __index__, in the range of an int
    int i32()
    {
        PyObject *o = next();
        if (!o) return 0;
        PyObject *x = PyNumber_Index(o);
        const long r = x ? PyLong_AsLong(x) : -1;
        Py_XDECREF(x);
        if (r == -1 && PyErr_Occurred()) ok = false;
        else if (r != (int)r) {
            PyErr_SetString(PyExc_OverflowError, "argument does not fit an int");
            ok = false;
        }
        return (int)r;
    }
    float f32()
    {
        PyObject *o = next();
        const double r = o ? PyFloat_AsDouble(o) : 0.0;
        if (o && r == -1.0 && PyErr_Occurred()) ok = false;
        return (float)r;
    }
    void *address()
    {
        PyObject *o = next();
        if (!o || o == Py_None) return nullptr;
        void *r = PyLong_AsVoidPtr(o);
        if (!r && PyErr_Occurred()) ok = false;
        return r;
    }
    // device pointer of a contiguous CUDA tensor of the given type; None and empty tensors give NULL
    void *tensor(at::ScalarType type, const char *what)
    {
        PyObject *o = next();
        if (!o || o == Py_None) return nullptr;
        if (!THPVariable_Check(o) || !THPVariable_Unpack(o).is_cuda()) {
            PyErr_Format(PyExc_TypeError, "%s: expected a CUDA torch tensor", what);
            ok = false;
            return nullptr;
        }
        const at::Tensor &t = THPVariable_Unpack(o);
        if (t.scalar_type() != type || !t.is_contiguous()) {
            PyErr_Format(PyExc_TypeError, "%s: expected contiguous %s, got %s contiguous=%s", what, at::toString(type),
                         at::toString(t.scalar_type()), t.is_contiguous() ? "True" : "False");
            ok = false;
            return nullptr;
        }
        return t.numel() ? t.data_ptr() : nullptr;
    }
    float *floats(const char *what) { return (float *)tensor(at::kFloat, what); }
    int *ints(const char *what) { return (int *)tensor(at::kInt, what); }
    // None: the current stream; an address; or an object with `cuda_stream`
    void *stream()
    {
        PyObject *o = next();
        if (!o) return nullptr;
        if (o == Py_None) return (void *)c10::cuda::getCurrentCUDAStream().stream();
        PyObject *x = PyLong_Check(o) ? Py_NewRef(o) : PyObject_GetAttrString(o, "cuda_stream");
        void *r = x ? PyLong_AsVoidPtr(x) : nullptr;
        Py_XDECREF(x);
        if (!r && PyErr_Occurred()) ok = false;
        return r;
    }
    bool end()
    {
        if (ok && at != n) {
            PyErr_SetString(PyExc_TypeError, "too many arguments");
            ok = false;
        }
        return ok;
    }
};

// The interpreter lock is released around the call, as ctypes does.
template <typename F>
PyObject *finish(F call)
{
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = call();
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

struct Sizes {
    int M, K, N, nnz;
    explicit Sizes(Args &a) : M(a.i32()), K(a.i32()), N(a.i32()), nnz(a.i32()) {}
};

#define DLSPM_GUARD_BEGIN try {
#define DLSPM_GUARD_END                                   \
    }                                                     \
    catch (const std::exception &e)                       \
    {                                                     \
        PyErr_SetString(PyExc_RuntimeError, e.what());    \
        return nullptr;                                   \
    }

PyObject *py_spmm(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    DLSPM_GUARD_BEGIN
    Args a{v, n};
    dlspm_ctx *ctx = (dlspm_ctx *)a.address();
    const Sizes s(a);
    float *values = a.floats("values");
    int *ro = a.ints("row_offsets"), *ci = a.ints("column_indices");
    float *B = a.floats("B"), *C = a.floats("C");
    void *st = a.stream();
    if (!a.end()) return nullptr;
    return finish([&] { return dlspm_spmm_csr_f32(ctx, s.M, s.K, s.N, s.nnz, values, ro, ci, B, C, st); });
    DLSPM_GUARD_END
}

PyObject *py_spmm_planned(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    DLSPM_GUARD_BEGIN
    Args a{v, n};
    dlspm_ctx *ctx = (dlspm_ctx *)a.address();
    const dlspm_plan *plan = (const dlspm_plan *)a.address();
    const int N = a.i32();
    float *values = a.floats("values");
    int *ro = a.ints("row_offsets"), *ci = a.ints("column_indices");
    float *B = a.floats("B"), *C = a.floats("C");
    void *st = a.stream();
    if (!a.end()) return nullptr;
    return finish([&] { return dlspm_spmm_csr_f32_planned(ctx, plan, N, values, ro, ci, B, C, st); });
    DLSPM_GUARD_END
}

PyObject *py_sddmm(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    DLSPM_GUARD_BEGIN
    Args a{v, n};
    dlspm_ctx *ctx = (dlspm_ctx *)a.address();
    const Sizes s(a);
    int *ro = a.ints("row_offsets"), *ci = a.ints("column_indices");
    float *mask = a.floats("mask_values"), *lhs = a.floats("lhs"), *rhs = a.floats("rhs"), *out = a.floats("out");
    void *st = a.stream();
    if (!a.end()) return nullptr;
    return finish([&] { return dlspm_sddmm_csr_masked_f32(ctx, s.M, s.K, s.N, s.nnz, ro, ci, mask, lhs, rhs, out, st); });
    DLSPM_GUARD_END
}

PyObject *py_fused(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    DLSPM_GUARD_BEGIN
    Args a{v, n};
    dlspm_ctx *ctx = (dlspm_ctx *)a.address();
    const Sizes s(a);
    int *ro = a.ints("row_offsets"), *ci = a.ints("column_indices");
    float *C = a.floats("C"), *B = a.floats("B"), *D = a.floats("D"), *E = a.floats("E");
    void *st = a.stream();
    if (!a.end()) return nullptr;
    return finish([&] { return dlspm_fused_sddmm_spmm_f32(ctx, s.M, s.K, s.N, s.nnz, ro, ci, C, B, D, E, st); });
    DLSPM_GUARD_END
}

PyObject *py_attention(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    DLSPM_GUARD_BEGIN
    Args a{v, n};
    dlspm_ctx *ctx = (dlspm_ctx *)a.address();
    const Sizes s(a);
    int *ro = a.ints("row_offsets"), *ci = a.ints("column_indices");
    float *Q = a.floats("Q"), *Kmat = a.floats("Kmat"), *V = a.floats("V"), *O = a.floats("O");
    const float scale = a.f32();
    const int flags = a.i32();
    void *st = a.stream();
    if (!a.end()) return nullptr;
    return finish([&] {
        return dlspm_fused_attention_f32(ctx, s.M, s.K, s.N, s.nnz, ro, ci, Q, Kmat, V, O, scale, (unsigned)flags, st);
    });
    DLSPM_GUARD_END
}

PyMethodDef kMethods[] = {
    {"spmm", (PyCFunction)(void (*)(void))py_spmm, METH_FASTCALL, "ctx, M, K, N, nnz, values, row_offsets, column_indices, B, C, stream"},
    {"spmm_planned", (PyCFunction)(void (*)(void))py_spmm_planned, METH_FASTCALL, "ctx, plan, N, values, row_offsets, column_indices, B, C, stream"},
    {"sddmm", (PyCFunction)(void (*)(void))py_sddmm, METH_FASTCALL, "ctx, M, K, N, nnz, row_offsets, column_indices, mask, lhs, rhs, out, stream"},
    {"fused", (PyCFunction)(void (*)(void))py_fused, METH_FASTCALL, "ctx, M, K, N, nnz, row_offsets, column_indices, C, B, D, E, stream"},
    {"attention", (PyCFunction)(void (*)(void))py_attention, METH_FASTCALL,
     "ctx, M, K, N, nnz, row_offsets, column_indices, Q, Kmat, V, O, scale, flags, stream"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_dlspm_call", "Tensor-taking calls of libdlspm.so.", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dlspm_call(void) { return PyModule_Create(&kModule); }
