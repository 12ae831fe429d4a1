// The operator calls on torch CUDA tensors, as a CPython extension (module catccos_b200._torch_calls).
//
// catccos_b200/capi.py declares the calls; what they do per call is here: unpack the tensors, fill the tiling record,
// take the current stream, allocate the outputs, call the C ABI (include/catccos_b200.h).  Host time of a call, launch
// included: 8.8 us (mx_gemm) to 14 (mx_quant) with these steps in Python and ctypes, more than the kernels of the small
// problems take; 2.9 to 4.2 us here.
//
// The C ABI's functions are not linked but bound by address (bind()), so that they are those of the library that capi.py
// has loaded.  Every function returns the C ABI's code (alone, or first in a tuple with the outputs).
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>

#include <cstring>

#include "../../include/catccos_b200.h"

namespace {

#define BOUND(name) decltype(&catccos_b200_##name) name##_fn = nullptr
BOUND(mx_quant);
BOUND(mx_quant_fp4);
BOUND(mx_gemm);
BOUND(mx_gemm_quant_out);
BOUND(mx_quant_scatter_packed);
BOUND(mxfp8_matmul_reduce_scatter);
BOUND(mx_quant_matmul_static);
BOUND(mx_quant_allgather);
BOUND(mx_quant_allgather_matmul);
BOUND(fp8_mx_allgather_matmul);
BOUND(fp4_mx_allgather_matmul);
#undef BOUND

struct Error {};  // a Python exception is set

const at::Tensor& tensor(PyObject* o)
{
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "expected a torch tensor, got %s", Py_TYPE(o)->tp_name);
        throw Error{};
    }
    return THPVariable_Unpack(o);
}

struct Rows {
    const at::Tensor& t;
    uint32_t rows, cols;
};

Rows matrix(PyObject* o)
{
    const at::Tensor& t = tensor(o);
    if (t.dim() != 2) {
        PyErr_Format(PyExc_ValueError, "expected a matrix, got %d dimensions", (int)t.dim());
        throw Error{};
    }
    return {t, (uint32_t)t.size(0), (uint32_t)t.size(1)};
}

// columns of the product: b_scales is [k / 64, n, 2]
uint32_t product_columns(PyObject* b_scales)
{
    const at::Tensor& t = tensor(b_scales);
    if (t.dim() < 2) {
        PyErr_SetString(PyExc_IndexError, "b_scales is [k / 64, n, 2]");
        throw Error{};
    }
    return (uint32_t)t.size(1);
}

void* pointer(PyObject* tensor_object) { return tensor(tensor_object).data_ptr(); }

// An address as ctypes takes one: a number, None, or a pointer object with a `value` (ctypes.c_void_p).
void* address(PyObject* o)
{
    if (o == Py_None) {
        return nullptr;
    }
    if (PyLong_Check(o)) {
        void* p = PyLong_AsVoidPtr(o);
        if (p == nullptr && PyErr_Occurred()) {
            throw Error{};
        }
        return p;
    }
    PyObject* value = PyObject_GetAttrString(o, "value");
    if (value == nullptr || !(value == Py_None || PyLong_Check(value))) {
        Py_XDECREF(value);
        PyErr_Format(PyExc_TypeError, "expected an address, got %s", Py_TYPE(o)->tp_name);
        throw Error{};
    }
    void* p = value == Py_None ? nullptr : PyLong_AsVoidPtr(value);
    Py_DECREF(value);
    if (p == nullptr && PyErr_Occurred()) {
        throw Error{};
    }
    return p;
}

uint32_t count(PyObject* number)
{
    const long v = PyLong_AsLong(number);
    if (v == -1 && PyErr_Occurred()) {
        throw Error{};
    }
    return (uint32_t)v;
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

at::Tensor bytes_like(const at::Tensor& x, int64_t rows, int64_t cols)
{
    return at::detail::empty_cuda({rows, cols}, at::kByte, x.device(), std::nullopt);
}

// The reference drivers' default tile fields (main.cpp:105-118), with the problem shape filled in.
catccos_b200_tiling_t tiling(uint32_t m, uint32_t k, uint32_t n, uint32_t world)
{
    catccos_b200_tiling_t t;
    memset(&t, 0, sizeof(t));
    t.m = m;
    t.k = k;
    t.n = n;
    t.m0 = 128;
    t.k0 = 256;
    t.n0 = 256;
    t.commTileM = 64;
    t.commInterval = 3;
    t.commNpuSplit = 2;
    t.commDataSplit = 16;
    t.commBlockM = 64;
    t.rankSize = world;
    t.topK = 1;
    return t;
}

// Launches may wait for room in the stream's queue: other Python threads run meanwhile.  The lock is back before an
// exception leaves.
struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
};

template <typename F>
PyObject* released(F&& call)
{
    int rc;
    {
        Unlocked unlocked;
        rc = call();
    }
    return PyLong_FromLong(rc);
}

PyObject* with_outputs(PyObject* code, const at::Tensor& a, const at::Tensor& b)
{
    PyObject* out = PyTuple_New(3);
    PyTuple_SET_ITEM(out, 0, code);
    PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(a));
    PyTuple_SET_ITEM(out, 2, THPVariable_Wrap(b));
    return out;
}

template <typename F>
PyObject* guarded(const char* name, Py_ssize_t want, Py_ssize_t n, bool bound, F&& body)
{
    if (n != want) {
        PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, n);
        return nullptr;
    }
    if (!bound) {
        PyErr_Format(PyExc_RuntimeError, "%s is not bound to the library", name);
        return nullptr;
    }
    try {
        return body();
    } catch (const Error&) {
        return nullptr;
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());  // torch.OutOfMemoryError and the like
        return nullptr;
    }
}

void assert_activations(const at::Tensor& x)
{
    if (!x.is_cuda() || !x.is_contiguous() || x.element_size() != 2) {
        PyErr_SetString(PyExc_AssertionError, "expected a contiguous CUDA tensor of 16-bit values");
        throw Error{};
    }
}

#define CALL(name, nargs) \
    PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n) { return guarded(#name, nargs, n, name##_fn != nullptr, [&]() -> PyObject* {
#define END_CALL }); }

CALL(mx_quant, 1)
    const Rows x = matrix(a[0]);
    assert_activations(x.t);
    const at::Tensor codes = bytes_like(x.t, x.rows, x.cols), scales = bytes_like(x.t, x.rows, x.cols / 32);
    void *st = stream(), *in = x.t.data_ptr(), *c = codes.data_ptr(), *s = scales.data_ptr();
    return with_outputs(released([&] { return mx_quant_fn(st, in, x.rows, x.cols, c, s); }), codes, scales);
END_CALL

CALL(mx_quant_fp4, 1)
    const Rows x = matrix(a[0]);
    assert_activations(x.t);
    const at::Tensor packed = bytes_like(x.t, x.rows, x.cols / 2), scales = bytes_like(x.t, x.rows, x.cols / 32);
    void *st = stream(), *in = x.t.data_ptr(), *c = packed.data_ptr(), *s = scales.data_ptr();
    return with_outputs(released([&] { return mx_quant_fp4_fn(st, in, x.rows, x.cols, c, s); }), packed, scales);
END_CALL

// a, a_scales, b, b_scales, out
CALL(mx_gemm, 5)
    const Rows x = matrix(a[0]);
    const uint32_t cols = product_columns(a[3]);
    void *st = stream(), *ac = x.t.data_ptr(), *as = pointer(a[1]), *b = pointer(a[2]), *bs = pointer(a[3]), *c = pointer(a[4]);
    return released([&] { return mx_gemm_fn(st, ac, as, b, bs, c, x.rows, cols, x.cols); });
END_CALL

// a, a_scales, b, b_scales
CALL(mx_gemm_quant_out, 4)
    const Rows x = matrix(a[0]);
    const uint32_t cols = product_columns(a[3]);
    const at::Tensor codes = bytes_like(x.t, x.rows, cols), scales = bytes_like(x.t, x.rows, cols / 32);
    void *st = stream(), *ac = x.t.data_ptr(), *as = pointer(a[1]), *b = pointer(a[2]), *bs = pointer(a[3]);
    void *c = codes.data_ptr(), *s = scales.data_ptr();
    return with_outputs(released([&] { return mx_gemm_quant_out_fn(st, ac, as, b, bs, c, s, x.rows, cols, x.cols); }), codes, scales);
END_CALL

// x, expanded_row_idx, packed_out, top_k
CALL(mx_quant_scatter_packed, 4)
    const Rows x = matrix(a[0]);
    const uint32_t top_k = count(a[3]);
    void *st = stream(), *in = x.t.data_ptr(), *idx = pointer(a[1]), *out = pointer(a[2]);
    return released([&] { return mx_quant_scatter_packed_fn(st, in, (const int32_t*)idx, out, x.rows, x.cols, top_k); });
END_CALL

// a, a_scales, b, b_scales, d, symm, world
CALL(mxfp8_matmul_reduce_scatter, 7)
    const Rows x = matrix(a[0]);
    const catccos_b200_tiling_t t = tiling(x.rows, x.cols, product_columns(a[3]), count(a[6]));
    void *st = stream(), *ac = x.t.data_ptr(), *as = pointer(a[1]), *b = pointer(a[2]), *bs = pointer(a[3]), *d = pointer(a[4]);
    void* symm = address(a[5]);
    return released([&] { return mxfp8_matmul_reduce_scatter_fn(st, ac, b, as, bs, d, symm, &t, 0); });
END_CALL

// a_bf16, b, b_scales, c
CALL(mx_quant_matmul_static, 4)
    const Rows x = matrix(a[0]);
    const uint32_t cols = product_columns(a[2]);
    void *st = stream(), *in = x.t.data_ptr(), *b = pointer(a[1]), *bs = pointer(a[2]), *c = pointer(a[3]);
    return released([&] { return mx_quant_matmul_static_fn(st, in, b, bs, c, x.rows, cols, x.cols); });
END_CALL

// x, out_codes, out_scales, symm, world
CALL(mx_quant_allgather, 5)
    const Rows x = matrix(a[0]);
    const catccos_b200_tiling_t t = tiling(x.rows, 1, x.cols, count(a[4]));  // the quantised axis is `n` for this operator
    void *st = stream(), *in = x.t.data_ptr(), *c = pointer(a[1]), *s = pointer(a[2]), *symm = address(a[3]);
    return released([&] { return mx_quant_allgather_fn(st, in, c, s, symm, &t, 0); });
END_CALL

// a_bf16, b, b_scales, c, symm, world
CALL(mx_quant_allgather_matmul, 6)
    const Rows x = matrix(a[0]);
    const catccos_b200_tiling_t t = tiling(x.rows, x.cols, product_columns(a[2]), count(a[5]));
    void *st = stream(), *in = x.t.data_ptr(), *b = pointer(a[1]), *bs = pointer(a[2]), *c = pointer(a[3]), *symm = address(a[4]);
    return released([&] { return mx_quant_allgather_matmul_fn(st, in, b, bs, c, symm, &t, 0); });
END_CALL

// a, a_scales, b, b_scales, c, symm, world
CALL(fp8_mx_allgather_matmul, 7)
    const Rows x = matrix(a[0]);
    const catccos_b200_tiling_t t = tiling(x.rows, x.cols, product_columns(a[3]), count(a[6]));
    void *st = stream(), *ac = x.t.data_ptr(), *as = pointer(a[1]), *b = pointer(a[2]), *bs = pointer(a[3]), *c = pointer(a[4]);
    void* symm = address(a[5]);
    return released([&] { return fp8_mx_allgather_matmul_fn(st, ac, b, as, bs, c, symm, &t, 0); });
END_CALL

// a_packed [m, k / 2], a_scales, b_packed, b_scales, c, symm, world
CALL(fp4_mx_allgather_matmul, 7)
    const Rows x = matrix(a[0]);
    const catccos_b200_tiling_t t = tiling(x.rows, x.cols * 2, product_columns(a[3]), count(a[6]));
    void *st = stream(), *ac = x.t.data_ptr(), *as = pointer(a[1]), *b = pointer(a[2]), *bs = pointer(a[3]), *c = pointer(a[4]);
    void* symm = address(a[5]);
    return released([&] { return fp4_mx_allgather_matmul_fn(st, ac, b, as, bs, c, symm, &t, 0); });
END_CALL

// bind(name, address): which function of the loaded library a call goes to
PyObject* bind(PyObject*, PyObject* args)
{
    const char* name = nullptr;
    unsigned long long at = 0;
    if (!PyArg_ParseTuple(args, "sK", &name, &at)) {
        return nullptr;
    }
#define BIND(fn)                                          \
    if (strcmp(name, "catccos_b200_" #fn) == 0) {         \
        fn##_fn = reinterpret_cast<decltype(fn##_fn)>(at); \
        Py_RETURN_TRUE;                                   \
    }
    BIND(mx_quant)
    BIND(mx_quant_fp4)
    BIND(mx_gemm)
    BIND(mx_gemm_quant_out)
    BIND(mx_quant_scatter_packed)
    BIND(mxfp8_matmul_reduce_scatter)
    BIND(mx_quant_matmul_static)
    BIND(mx_quant_allgather)
    BIND(mx_quant_allgather_matmul)
    BIND(fp8_mx_allgather_matmul)
    BIND(fp4_mx_allgather_matmul)
#undef BIND
    Py_RETURN_FALSE;
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    METHOD(mx_quant),
    METHOD(mx_quant_fp4),
    METHOD(mx_gemm),
    METHOD(mx_gemm_quant_out),
    METHOD(mx_quant_scatter_packed),
    METHOD(mxfp8_matmul_reduce_scatter),
    METHOD(mx_quant_matmul_static),
    METHOD(mx_quant_allgather),
    METHOD(mx_quant_allgather_matmul),
    METHOD(fp8_mx_allgather_matmul),
    METHOD(fp4_mx_allgather_matmul),
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
#undef METHOD

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_calls(void) { return PyModule_Create(&module); }
