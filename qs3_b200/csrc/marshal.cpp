// Descriptor marshalling of the Python host layer: fills the qsfi_tensorN fields of a C descriptor from torch
// tensors. Done field by field through ctypes a layer call spends ~50 us on it, which is more than its GPU work
// at decode sizes; here a call costs about a microsecond.
//
//   fill(address, layout, tensors)
//     address   of the descriptor structure
//     layout    bytes: per tensor three int32 {byte offset, rank, dtype code or -1 for the tensor's own}; rank 0 means
//               a rank-1 view of all elements of a contiguous tensor
//     tensors   tuple of the same length; None leaves the field zero (absent optional tensor)
//   returns -1, or the index of a tensor whose rank (or contiguity, rank 0) does not fit
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>

#include "../../include/qs3_moe.h"

#include <cstring>
#include <exception>

namespace {

int32_t dtype_code(at::ScalarType t)
{
    switch (t) {
    case at::kFloat: return QSFI_DTYPE_F32;
    case at::kHalf: return QSFI_DTYPE_F16;
    case at::kBFloat16: return QSFI_DTYPE_BF16;
    case at::kInt: return QSFI_DTYPE_I32;
    case at::kChar: return QSFI_DTYPE_I8;
    case at::kByte: return QSFI_DTYPE_U8;
    case at::kFloat8_e4m3fn: return QSFI_DTYPE_FP8_E4M3;
    default: return 0;
    }
}

template <typename Tensor, uint32_t RANK> void put(char* at_, const at::Tensor& t, int32_t dtype)
{
    Tensor d;
    std::memset(&d, 0, sizeof(d));
    d.data = t.data_ptr();
    d.dtype = static_cast<qsfi_dtype>(dtype);
    for (uint32_t i = 0; i < RANK; ++i) {
        d.shape[i] = t.size(i);
        d.stride[i] = t.stride(i);
    }
    std::memcpy(at_, &d, sizeof(d));
}

PyObject* fill_checked(PyObject* const* args, Py_ssize_t nargs)
{
    if (nargs != 3 || !PyBytes_Check(args[1]) || !PyTuple_Check(args[2])) {
        PyErr_SetString(PyExc_TypeError, "fill(address, layout bytes, tensor tuple)");
        return nullptr;
    }
    char* base = static_cast<char*>(PyLong_AsVoidPtr(args[0]));
    if (base == nullptr) {
        if (!PyErr_Occurred())
            PyErr_SetString(PyExc_ValueError, "null descriptor address");
        return nullptr;
    }
    const int32_t* layout = reinterpret_cast<const int32_t*>(PyBytes_AS_STRING(args[1]));
    const Py_ssize_t n = PyTuple_GET_SIZE(args[2]);
    if (PyBytes_GET_SIZE(args[1]) != n * 12) {
        PyErr_SetString(PyExc_ValueError, "layout and tensors differ in length");
        return nullptr;
    }
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* o = PyTuple_GET_ITEM(args[2], i);
        if (o == Py_None)
            continue;
        if (!THPVariable_Check(o)) {
            PyErr_Format(PyExc_TypeError, "expected a tensor or None at position %zd", i);
            return nullptr;
        }
        const at::Tensor& t = THPVariable_Unpack(o);
        char* at_ = base + layout[3 * i];
        const int32_t rank = layout[3 * i + 1];
        const int32_t dtype = layout[3 * i + 2] >= 0 ? layout[3 * i + 2] : dtype_code(t.scalar_type());
        if (rank == 0 ? !t.is_contiguous() : t.dim() != rank)
            return PyLong_FromSsize_t(i);
        if (rank == 0) {
            qsfi_tensor1 d;
            std::memset(&d, 0, sizeof(d));
            d.data = t.data_ptr();
            d.dtype = static_cast<qsfi_dtype>(dtype);
            d.shape[0] = t.numel();
            d.stride[0] = 1;
            std::memcpy(at_, &d, sizeof(d));
        } else if (rank == 1) {
            put<qsfi_tensor1, 1>(at_, t, dtype);
        } else if (rank == 2) {
            put<qsfi_tensor2, 2>(at_, t, dtype);
        } else {
            put<qsfi_tensor3, 3>(at_, t, dtype);
        }
    }
    return PyLong_FromLong(-1);
}

PyObject* fill(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    try {
        return fill_checked(args, nargs);
    } catch (const std::exception& e) { // tensors without storage and the like
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyMethodDef methods[] = {
    { "fill", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fill)), METH_FASTCALL,
      "fill(address, layout, tensors) -> -1 or the index of a tensor of the wrong rank" },
    { nullptr, nullptr, 0, nullptr },
};

PyModuleDef module = { PyModuleDef_HEAD_INIT, "_marshal", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr };

} // namespace

PyMODINIT_FUNC PyInit__marshal()
{
    PyObject* m = PyModule_Create(&module);
    if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", QS3_TORCH_VERSION) != 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
