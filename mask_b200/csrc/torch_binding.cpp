// Python binding of the products: checks the tensors, allocates C and the scratch from torch's allocator and calls
// the C ABI, without building Python or ctypes objects on the way.  A product took 14 us of host time through
// ctypes; the smallest ones take the GPU 5.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "mask_b200.h"

namespace {

PyObject* raise(const char* what) {
    PyErr_SetString(PyExc_RuntimeError, what);
    return nullptr;
}

// NULL for None, else the tensor's address
bool pointer_of(PyObject* o, const void** out) {
    *out = nullptr;
    if (o == Py_None) return true;
    if (!THPVariable_Check(o)) return false;
    *out = THPVariable_Unpack(o).data_ptr();
    return true;
}

// The tensor must be a contiguous float32 CUDA tensor; messages as the package's own checks word them.
const at::Tensor* float_tensor(PyObject* o, const char* name) {
    const char* rule = "a CUDA tensor";
    if (THPVariable_Check(o)) {
        const at::Tensor& t = THPVariable_Unpack(o);
        rule = !t.is_cuda() ? "a CUDA tensor" : (!t.is_contiguous() ? "contiguous" : (t.scalar_type() != at::kFloat ? "float32" : nullptr));
        if (!rule) return &t;
    }
    PyErr_Format(PyExc_RuntimeError, "%s must be %s", name, rule);
    return nullptr;
}

// spmm(format, M, K, val_sidx, offsets, index, values, plan, dense, out or None, epilogue, whole_vectors) -> out, or an
// int: the status of a C-ABI call that failed.  whole_vectors: only N % 4 == 0 (else -1) and 16-byte aligned dense and
// out (else -2) are taken.
PyObject* product(PyObject* const* args, Py_ssize_t n_args) {
    if (n_args != 12) return raise("spmm takes 12 arguments");
    mask_matrix m{};
    m.format = (int32_t)PyLong_AsLong(args[0]);
    m.M = (int32_t)PyLong_AsLong(args[1]);
    m.K = (int32_t)PyLong_AsLong(args[2]);
    const void *sidx, *offsets;
    if (!pointer_of(args[3], &sidx) || !pointer_of(args[4], &offsets) || !pointer_of(args[5], &m.index) || !pointer_of(args[6], &m.values))
        return raise("the packed arrays must be tensors");
    m.val_sidx = static_cast<const int32_t*>(sidx);
    m.offsets = static_cast<const int32_t*>(offsets);
    const auto* plan = static_cast<const mask_plan*>(PyLong_AsVoidPtr(args[7]));
    const int epilogue = (int)PyLong_AsLong(args[10]);
    if (PyErr_Occurred()) return nullptr;
    const at::Tensor* dense = float_tensor(args[8], "dense");
    if (!dense) return nullptr;
    if (dense->dim() != 2) return raise("dense must be 2-D");
    const int64_t K = dense->size(0), N = dense->size(1);
    if (K != m.K) {
        PyErr_Format(PyExc_RuntimeError, "dense has %lld rows, the matrix has %d columns", (long long)K, (int)m.K);
        return nullptr;
    }
    if (N > 0x7ffffffc) return raise("dense has too many columns");
    at::Tensor out;
    if (args[9] == Py_None) {
        out = at::empty({m.M, N}, dense->options());
    } else {
        const at::Tensor* given = float_tensor(args[9], "out");
        if (!given) return nullptr;
        if (given->dim() != 2 || given->size(0) != m.M || given->size(1) != N) return raise("out has the wrong shape");
        out = *given;
    }
    if (N > 0) {
        if (args[11] == Py_True) {
            if (N % 4) return PyLong_FromLong(-1);
            if ((reinterpret_cast<uintptr_t>(dense->data_ptr()) | reinterpret_cast<uintptr_t>(out.data_ptr())) & 15) return PyLong_FromLong(-2);
        }
        const int32_t n4 = (int32_t)((N + 3) & ~(int64_t)3);
        const float* B = static_cast<const float*>(dense->data_ptr());
        // freed to torch's allocator on return: it is reused in stream order
        at::Tensor pad, scratch;
        if (n4 != N || (reinterpret_cast<uintptr_t>(B) & 15)) pad = at::empty({K * n4}, dense->options());
        const size_t need = mask_plan_scratch_bytes(plan, n4);
        if (need) scratch = at::empty({(int64_t)need}, dense->options().dtype(at::kByte));
        float* C = static_cast<float*>(out.data_ptr());
        cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = mask_spmm(plan, &m, (int32_t)N, B, N, C, N, pad.defined() ? static_cast<float*>(pad.data_ptr()) : nullptr,
                       need ? scratch.data_ptr() : nullptr, need, epilogue, stream);
        Py_END_ALLOW_THREADS
        if (rc != MASK_OK) return PyLong_FromLong(rc);
    }
    if (args[9] != Py_None) {
        Py_INCREF(args[9]);
        return args[9];
    }
    return THPVariable_Wrap(std::move(out));
}

// Tensors without storage or strides (sparse ones, those of torch.func's transforms) throw already when they are asked
// for an address or whether they are contiguous.
PyObject* spmm(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
    try {
        return product(args, n_args);
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

PyMethodDef methods[] = {
    {"spmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(spmm)), METH_FASTCALL, "out = A @ dense, or a status"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() { return PyModule_Create(&module); }
