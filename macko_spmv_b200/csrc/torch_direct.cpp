// `multiply` and the batched product of a frozen matrix without the operator dispatcher, a Python module beside the operator library.
//
// A product of a small matrix takes less time on the GPU than the way of its arguments through the operator boundary
// (Python asserts, schema matching, boxing). The module function below takes that way out for calls that only
// want the product: plain CUDA tensors, no gradient, and nobody watching operators go by (no tensor subclass, dispatch
// or function mode, transform, tracer, profiler). It answers None for everything else and the caller goes through
// the operator. The checks of the operator's CUDA implementation run here as well and raise what they raise there.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "macko_b200.h"
#include "torch_products.h"

namespace {

PyObject *g_frozen_type = nullptr;   // macko_spmv_b200.FrozenMatrix
PyObject *g_even_name = nullptr, *g_plan_name = nullptr, *g_plan_meta_name = nullptr, *g_windows_name = nullptr, *g_windows_of_name = nullptr, *g_windows_batch_name = nullptr;

bool nobody_watches()
{
    const c10::DispatchKeySet included = c10::impl::tls_local_dispatch_key_set().included_ -
                                         c10::DispatchKeySet({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView});
    return included.empty() && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() &&
           !at::getStepCallbacksUnlessEmpty(at::RecordScope::FUNCTION).has_value();
}

// The tensor of a Python object if it is a plain CUDA tensor, else null.
const at::Tensor *plain_tensor(PyObject *o)
{
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.requires_grad()) return nullptr;
    const c10::DispatchKeySet odd({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                   c10::DispatchKey::Functionalize, c10::DispatchKey::Batched, c10::DispatchKey::Conjugate,
                                   c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
    return t.key_set().has_any(odd) ? nullptr : &t;
}

bool as_int64(PyObject *o, int64_t &v)
{
    if (!PyLong_CheckExact(o)) return false;
    v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
}

// multiply(compressed, V) -> y, or None where the call has to go through the operator
PyObject *direct_multiply(PyObject *, PyObject *const *args, Py_ssize_t n_args)
{
    HANDLE_TH_ERRORS
    if (n_args != 2 || !PyTuple_Check(args[0])) Py_RETURN_NONE;
    PyObject *m = args[0];
    const bool frozen = reinterpret_cast<PyObject *>(Py_TYPE(m)) == g_frozen_type;
    if (!(frozen || PyTuple_CheckExact(m)) || PyTuple_GET_SIZE(m) < 5 || !nobody_watches()) Py_RETURN_NONE;
    const at::Tensor *values = plain_tensor(PyTuple_GET_ITEM(m, 0)), *deltas = plain_tensor(PyTuple_GET_ITEM(m, 1)),
                     *ri = plain_tensor(PyTuple_GET_ITEM(m, 2)), *V = plain_tensor(args[1]);
    int64_t rows, cols;
    if (!values || !deltas || !ri || !V || !V->is_contiguous() || !as_int64(PyTuple_GET_ITEM(m, 3), rows) || !as_int64(PyTuple_GET_ITEM(m, 4), cols))
        Py_RETURN_NONE;
    const at::Tensor *plan = nullptr;
    int64_t virtual_rows = 0, segment = 0, split_rows = 0;
    uint32_t flags = frozen ? MACKO_SPMV_MATRIX_IMMUTABLE : 0u;
    if (frozen) {
        PyObject *p = PyObject_GetAttr(m, g_plan_name);   // new references; the attributes outlive the call in the matrix
        if (!p) return nullptr;
        Py_DECREF(p);
        if (p != Py_None) {
            PyObject *meta = PyObject_GetAttr(m, g_plan_meta_name);
            if (!meta) return nullptr;
            Py_DECREF(meta);
            plan = plain_tensor(p);
            if (!plan || !PyTuple_CheckExact(meta) || PyTuple_GET_SIZE(meta) < 4 || !as_int64(PyTuple_GET_ITEM(meta, 0), virtual_rows) ||
                !as_int64(PyTuple_GET_ITEM(meta, 1), segment) || !as_int64(PyTuple_GET_ITEM(meta, 3), split_rows))
                Py_RETURN_NONE;
        } else {
            PyObject *even = PyObject_GetAttr(m, g_even_name);
            if (!even) return nullptr;
            Py_DECREF(even);
            if (even == Py_True) flags |= MACKO_SPMV_ROWS_EVEN;
        }
    }
    // own handles: another thread may drop the Python ones while the interpreter lock is released
    const at::Tensor v = *values, d = *deltas, r = *ri, x = *V, pl = plan ? *plan : at::Tensor();
    at::Tensor y;
    {
        struct NoGil { PyThreadState *s = PyEval_SaveThread(); ~NoGil() { PyEval_RestoreThread(s); } } no_gil;
        y = plan ? macko_torch::multiply_planned_cuda(v, d, r, rows, cols, pl, virtual_rows, segment, split_rows, x, true)
                 : macko_torch::multiply_flags(v, d, r, rows, cols, x, flags);
    }
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// Attribute `name` of a frozen matrix; the new reference is dropped at once, the attribute outlives the call in the matrix.
PyObject *attribute(PyObject *m, PyObject *name)
{
    PyObject *p = PyObject_GetAttr(m, name);
    Py_XDECREF(p);
    return p;
}

// Whether the matrix is as `freeze` found it: `of` = (write count of the deltas, of the row offsets, their addresses, write count and
// address of the values), or None where the caller has promised that nobody writes it.
bool as_frozen(PyObject *of, const at::Tensor &values, const at::Tensor &deltas, const at::Tensor &ri)
{
    if (of == Py_None) return true;
    if (!PyTuple_CheckExact(of) || PyTuple_GET_SIZE(of) != 6 || deltas.is_inference() || ri.is_inference() || values.is_inference()) return false;
    const int64_t now[6] = {deltas._version(), ri._version(), reinterpret_cast<int64_t>(deltas.data_ptr()), reinterpret_cast<int64_t>(ri.data_ptr()),
                            values._version(), reinterpret_cast<int64_t>(values.data_ptr())};
    for (int i = 0; i < 6; ++i) {
        int64_t was;
        if (!as_int64(PyTuple_GET_ITEM(of, i), was) || was != now[i]) return false;
    }
    return true;
}

// multiply_batched(compressed, V) -> y for 3 vectors and more of a frozen matrix with windows: over the windows up to the batch that
// `freeze` found them faster for, else a dense copy and a GEMM. None where the call has to take another route.
PyObject *direct_multiply_batched(PyObject *, PyObject *const *args, Py_ssize_t n_args)
{
    HANDLE_TH_ERRORS
    PyObject *m = n_args == 2 ? args[0] : nullptr;
    if (!m || reinterpret_cast<PyObject *>(Py_TYPE(m)) != g_frozen_type || PyTuple_GET_SIZE(m) < 5) Py_RETURN_NONE;
    const at::Tensor *V = plain_tensor(args[1]);
    if (!V || V->dim() != 2 || V->size(0) < 3 || !V->is_contiguous() || V->scalar_type() != at::kHalf || V->_fw_grad(0).defined() || !nobody_watches())
        Py_RETURN_NONE;
    const at::Tensor *values = plain_tensor(PyTuple_GET_ITEM(m, 0)), *deltas = plain_tensor(PyTuple_GET_ITEM(m, 1)),
                     *ri = plain_tensor(PyTuple_GET_ITEM(m, 2));
    int64_t rows, cols;
    if (!values || !deltas || !ri || values->_fw_grad(0).defined() || !as_int64(PyTuple_GET_ITEM(m, 3), rows) ||
        !as_int64(PyTuple_GET_ITEM(m, 4), cols))
        Py_RETURN_NONE;
    PyObject *w = attribute(m, g_windows_name);
    if (!w) return nullptr;
    const at::Tensor *windows = plain_tensor(w);
    if (!windows) Py_RETURN_NONE;
    PyObject *limit = attribute(m, g_windows_batch_name);
    if (!limit) return nullptr;
    int64_t windows_batch;
    if (!as_int64(limit, windows_batch) || V->size(1) != cols) Py_RETURN_NONE;
    const bool dense = V->size(0) > windows_batch;
    if (!dense) {
        PyObject *of = attribute(m, g_windows_of_name);
        if (!of) return nullptr;
        if (!as_frozen(of, *values, *deltas, *ri)) Py_RETURN_NONE;
    }
    // own handles: another thread may drop the Python ones while the interpreter lock is released
    const at::Tensor v = *values, d = *deltas, r = *ri, x = *V, win = *windows;
    at::Tensor y;
    {
        struct NoGil { PyThreadState *s = PyEval_SaveThread(); ~NoGil() { PyEval_RestoreThread(s); } } no_gil;
        y = dense ? at::matmul(x, macko_torch::decompress_cuda(v, d, r, rows, cols).t()) : macko_torch::multiply_windowed_cuda(v, d, r, rows, cols, win, x, true);
    }
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// set_frozen_type(FrozenMatrix): the class that `freeze` returns
PyObject *set_frozen_type(PyObject *, PyObject *type)
{
    Py_INCREF(type);
    Py_XSETREF(g_frozen_type, type);
    Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"multiply", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&direct_multiply)), METH_FASTCALL, nullptr},
    {"multiply_batched", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&direct_multiply_batched)), METH_FASTCALL, nullptr},
    {"set_frozen_type", &set_frozen_type, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_torch_direct", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_direct()
{
    g_even_name = PyUnicode_InternFromString("even_rows");
    g_plan_name = PyUnicode_InternFromString("plan");
    g_plan_meta_name = PyUnicode_InternFromString("plan_meta");
    g_windows_name = PyUnicode_InternFromString("windows");
    g_windows_of_name = PyUnicode_InternFromString("windows_of");
    g_windows_batch_name = PyUnicode_InternFromString("windows_batch");
    return g_even_name && g_plan_name && g_plan_meta_name && g_windows_name && g_windows_of_name && g_windows_batch_name ? PyModule_Create(&g_module) : nullptr;
}
