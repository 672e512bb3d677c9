// The host side of the two library calls that small linears are made of, native: taking a dozen tensors apart, allocating the output and the scratch
// and passing twenty arguments costs an interpreter more than such a linear takes on the GPU (batch of 64 tokens, 5120 x 5120: 18 us of host work
// a call, 6 of them in the library's two launches and 12 in Python and ctypes; here 10.6).  The module decides nothing: the caller has chosen path,
// tile variant and scratch, and passes the address of the library's entry point.  A call that is not of the plain form (tensors of another
// class, strides, types) comes back as None and takes the general way.
//
//   linear(address, x, weight, scale, bias, residual, residual_scale, out, act_weight, group, act, eps, path, variant, sms, scratch bytes)
//   few(address, x, weight, scale, bias, residual, residual_scale, out, act_weight, act, eps, form, sms, scratch bytes, where in them the tile counters lie)
//
// both return the output, None, or the library's error code as an int.  Built against the PyTorch that runs it
// (BUILT_FOR names it; another one may lay tensors out otherwise), without CUDA code of its own.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

using Linear = int (*)(const void*, int64_t, const int8_t*, const float*, const void*, const void*, const void*, void*, int, int, int, int, int, int, const void*, float,
                       int, int, int, void*, void*);
using Few = int (*)(const void*, int64_t, const int8_t*, const float*, const void*, const void*, const void*, void*, int, int, int, int, int, const void*, float, int,
                    void*, void*, void*);

constexpr int kSwiglu = 2;

// What both calls have in common.
struct Operands {
    at::Tensor x, weight, out;
    const void *scale, *bias, *residual, *rscale, *act_weight;
    PyObject* given;  // the caller's output, or nullptr
    int64_t m, n, k;
    int dtype;
};

const void* pointer(PyObject* object) { return object == Py_None ? nullptr : THPVariable_Unpack(object).data_ptr(); }

// x, weight, scale, bias, residual, residual_scale, out, act_weight; false when the call takes the general way
bool take(PyObject* const* a, int act, Operands& o) {
    for (int i = 0; i < 3; ++i)
        if (!THPVariable_CheckExact(a[i])) return false;
    for (int i = 3; i < 8; ++i)
        if (a[i] != Py_None && !THPVariable_CheckExact(a[i])) return false;
    o.x = THPVariable_Unpack(a[0]);
    o.weight = THPVariable_Unpack(a[1]);
    if (!o.x.is_cuda() || o.x.dim() != 2 || o.x.stride(1) != 1 || o.weight.dim() != 2) return false;
    const auto type = o.x.scalar_type();
    if (type != at::kHalf && type != at::kBFloat16) return false;
    o.dtype = type == at::kHalf ? 0 : 1;
    o.m = o.x.size(0);
    o.n = o.weight.size(0);
    o.k = act == kSwiglu ? o.x.size(1) / 2 : o.x.size(1);
    if (o.weight.size(1) != o.k) return false;
    for (const int i : {4, 6}) {  // residual, out: contiguous rows
        if (a[i] == Py_None) continue;
        const at::Tensor& t = THPVariable_Unpack(a[i]);
        if (t.dim() != 2 || t.stride(0) != o.n) return false;
    }
    o.scale = pointer(a[2]);
    o.bias = pointer(a[3]);
    o.residual = pointer(a[4]);
    o.rscale = pointer(a[5]);
    o.act_weight = pointer(a[7]);
    o.given = a[6] == Py_None ? nullptr : a[6];
    return true;
}

void allocate_output(Operands& o) { o.out = o.given ? THPVariable_Unpack(o.given) : at::empty({o.m, o.n}, o.x.options()); }

PyObject* result(const Operands& o, int code) {
    if (code) return PyLong_FromLong(code);
    if (o.given) {
        Py_INCREF(o.given);
        return o.given;
    }
    return THPVariable_Wrap(o.out);
}

at::Tensor scratch_of(const Operands& o, int64_t bytes) { return at::empty({bytes}, o.x.options().dtype(at::kByte)); }

void* stream_of(const Operands& o) { return c10::cuda::getCurrentCUDAStream(o.x.device().index()).stream(); }

// The launches of a call, other Python threads running meanwhile (as they do under ctypes).
template <class F> int without_gil(F&& launch) {
    PyThreadState* state = PyEval_SaveThread();
    const int code = launch();
    PyEval_RestoreThread(state);
    return code;
}

int integer(PyObject* object) { return int(PyLong_AsLongLong(object)); }

PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 16) return PyErr_Format(PyExc_TypeError, "linear() takes 16 arguments, %zd given", count);
    const auto call = reinterpret_cast<Linear>(PyLong_AsVoidPtr(a[0]));
    const int group = integer(a[9]), act = integer(a[10]), path = integer(a[12]), variant = integer(a[13]), sms = integer(a[14]);
    const auto eps = float(PyFloat_AsDouble(a[11]));
    const int64_t bytes = PyLong_AsLongLong(a[15]);
    if (PyErr_Occurred()) return nullptr;
    Operands o;
    if (!take(a + 1, act, o)) Py_RETURN_NONE;
    allocate_output(o);
    const at::Tensor scratch = scratch_of(o, bytes);
    const void* x = o.x.data_ptr();
    auto w = static_cast<const int8_t*>(o.weight.data_ptr());
    void *y = o.out.data_ptr(), *memory = scratch.data_ptr(), *stream = stream_of(o);
    return result(o, without_gil([&] {
                      return call(x, o.x.stride(0), w, static_cast<const float*>(o.scale), o.bias, o.residual, o.rscale, y, int(o.m), int(o.n), int(o.k), o.dtype, group, act,
                                  o.act_weight, eps, path, variant, sms, memory, stream);
                  }));
    END_HANDLE_TH_ERRORS
}

PyObject* few(PyObject*, PyObject* const* a, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 15) return PyErr_Format(PyExc_TypeError, "few() takes 15 arguments, %zd given", count);
    const auto call = reinterpret_cast<Few>(PyLong_AsVoidPtr(a[0]));
    const int act = integer(a[9]), form = integer(a[11]), sms = integer(a[12]);
    const auto eps = float(PyFloat_AsDouble(a[10]));
    const int64_t bytes = PyLong_AsLongLong(a[13]);
    const int64_t counters = PyLong_AsLongLong(a[14]);
    if (PyErr_Occurred()) return nullptr;
    Operands o;
    if (!take(a + 1, act, o)) Py_RETURN_NONE;
    const void* x = o.x.data_ptr();
    auto w = static_cast<const int8_t*>(o.weight.data_ptr());
    const uintptr_t rows = reinterpret_cast<uintptr_t>(x) | uintptr_t(o.x.stride(0)) * 2;  // what wq8_few asks of x, w and the norm weights
    if ((reinterpret_cast<uintptr_t>(w) & 15) || (rows & (form == 1 ? 7 : 15)) || (reinterpret_cast<uintptr_t>(o.act_weight) & 15)) Py_RETURN_NONE;
    allocate_output(o);
    const at::Tensor scratch = bytes ? scratch_of(o, bytes) : at::Tensor();
    void *y = o.out.data_ptr(), *memory = bytes ? scratch.data_ptr() : nullptr, *stream = stream_of(o);
    void* tile_counters = bytes ? static_cast<char*>(memory) + counters : nullptr;  // of this call alone: other streams' calls count their own
    return result(o, without_gil([&] {
                      return call(x, o.x.stride(0), w, static_cast<const float*>(o.scale), o.bias, o.residual, o.rscale, y, int(o.m), int(o.n), int(o.k), o.dtype, act,
                                  o.act_weight, eps, sms, memory, tile_counters, stream);
                  }));
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear)), METH_FASTCALL, "A whole linear through wq8_linear."},
                         {"few", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(few)), METH_FASTCALL, "A few tokens through wq8_few."},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", "Native host side of wq8_linear and wq8_few.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

#ifndef WQ_BUILT_FOR
#error "the build passes the PyTorch and the Python that this is compiled against"
#endif

PyMODINIT_FUNC PyInit__calls() {
    PyObject* made = PyModule_Create(&module);
    if (made && PyModule_AddStringConstant(made, "BUILT_FOR", WQ_BUILT_FOR) < 0) {
        Py_DECREF(made);
        return nullptr;
    }
    return made;
}
