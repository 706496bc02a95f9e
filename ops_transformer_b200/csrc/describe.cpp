// Tensor descriptions for gmmB200Call (include/gmm_b200.h), written from the tensors themselves.
//
// In Python the description of a call - address, type, format, sizes, strides and storage sizes of seven to ten tensors - cost
// 7 us, more than the call's launches; here 0.6.
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <Python.h>
#include <cstdint>
#include <vector>

namespace {

// aclDataType (include/aclnn/aclnn_base.h); -1: none
int acl_dtype(at::ScalarType t)
{
    switch (t) {
        case at::kFloat: return 0;
        case at::kHalf: return 1;
        case at::kChar: return 2;
        case at::kInt: return 3;
        case at::kLong: return 9;
        case at::kBFloat16: return 27;
        default: return -1;
    }
}

bool read_ints(PyObject *seq, std::vector<int64_t> &out)
{
    PyObject *fast = PySequence_Fast(seq, "a sequence of integers is wanted");
    if (!fast) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
    for (Py_ssize_t i = 0; i < n; ++i) {
        const int64_t v = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(fast, i));
        if (v == -1 && PyErr_Occurred()) {
            Py_DECREF(fast);
            return false;
        }
        out.push_back(v);
    }
    Py_DECREF(fast);
    return true;
}

// rank of the view (-1 for None), address, type, format, view sizes, view strides, rank of the storage, storage sizes
bool put_tensor(std::vector<int64_t> &w, PyObject *obj, int64_t format, PyObject *view_dims)
{
    if (obj == Py_None) {
        w.push_back(-1);
        return true;
    }
    if (!THPVariable_Check(obj)) {
        PyErr_Format(PyExc_TypeError, "a tensor or None is wanted, not %s", Py_TYPE(obj)->tp_name);
        return false;
    }
    const at::Tensor &t = THPVariable_Unpack(obj);
    const int64_t rank = t.dim();
    if (rank > 8) {
        PyErr_SetString(PyExc_MemoryError, "a tensor of more than 8 dimensions cannot be described");
        return false;
    }
    const int dtype = acl_dtype(t.scalar_type());
    if (dtype < 0) {
        PyErr_SetObject(PyExc_KeyError, reinterpret_cast<PyObject *>(torch::getTHPDtype(t.scalar_type())));
        return false;
    }
    std::vector<int64_t> dims;
    if (view_dims != Py_None && !read_ints(view_dims, dims)) return false;
    const auto sizes = t.sizes();
    w.push_back(view_dims == Py_None ? rank : (int64_t)dims.size());
    w.push_back((int64_t)reinterpret_cast<uintptr_t>(t.data_ptr()));
    w.push_back(dtype);
    w.push_back(format);
    if (view_dims == Py_None) {
        const auto strides = t.strides();
        w.insert(w.end(), sizes.begin(), sizes.end());
        w.insert(w.end(), strides.begin(), strides.end());
    } else {
        std::vector<int64_t> strides(dims.size(), 1);
        for (size_t i = dims.size(); i-- > 1;) strides[i - 1] = strides[i] * dims[i];
        w.insert(w.end(), dims.begin(), dims.end());
        w.insert(w.end(), strides.begin(), strides.end());
    }
    w.push_back(rank);
    w.insert(w.end(), sizes.begin(), sizes.end());
    return true;
}

// One argument of a call.  What it has to be follows from its place in the operator's description, not from what is given: an
// integer may be any object with __index__ (numpy's, a tensor of one element), and only tensors and lists may be None.
//   't'  a tensor (row-major format) or None          'i'  an integer, one word as it is
//   'f'  (tensor, format, view sizes or None)         'l'  a list of integers (length, then the values) or None
bool put_item(std::vector<int64_t> &w, char kind, PyObject *a)
{
    if (kind == 't') return put_tensor(w, a, 2, Py_None);
    if (kind == 'f') {
        if (!PyTuple_Check(a) || PyTuple_GET_SIZE(a) != 3) {
            PyErr_SetString(PyExc_TypeError, "(tensor, format, view sizes) is wanted");
            return false;
        }
        const int64_t format = PyLong_AsLongLong(PyTuple_GET_ITEM(a, 1));
        if (format == -1 && PyErr_Occurred()) return false;
        return put_tensor(w, PyTuple_GET_ITEM(a, 0), format, PyTuple_GET_ITEM(a, 2));
    }
    if (kind == 'i') {
        PyObject *index = PyNumber_Index(a);
        const int64_t v = index ? PyLong_AsLongLong(index) : -1;
        Py_XDECREF(index);
        if (v == -1 && PyErr_Occurred()) return false;
        w.push_back(v);
        return true;
    }
    if (kind == 'l') {
        if (a == Py_None) {
            w.push_back(-1);
            return true;
        }
        if (!PyList_Check(a)) {
            PyErr_Format(PyExc_TypeError, "a list of integers or None is wanted, not %s", Py_TYPE(a)->tp_name);
            return false;
        }
        w.push_back((int64_t)PyList_GET_SIZE(a));
        return read_ints(a, w);
    }
    PyErr_SetString(PyExc_ValueError, "unknown kind of argument");
    return false;
}

// The kind of an item described by itself: integers are told by their type, tensors stay tensors.
char kind_of(PyObject *a)
{
    if (PyLong_Check(a)) return 'i';
    if (PyList_Check(a)) return 'l';
    if (PyTuple_Check(a) && PyTuple_GET_SIZE(a) == 3) return 'f';
    return a != Py_None && !THPVariable_Check(a) && PyIndex_Check(a) ? 'i' : 't';
}

template <typename Kind>
PyObject *packed(PyObject *const *items, Py_ssize_t n, Kind kind)
{
    try {
        std::vector<int64_t> w;
        w.reserve(192);
        for (Py_ssize_t i = 0; i < n; ++i)
            if (!put_item(w, kind(i), items[i])) return nullptr;
        return PyBytes_FromStringAndSize(reinterpret_cast<const char *>(w.data()), (Py_ssize_t)(w.size() * sizeof(int64_t)));
    } catch (const std::exception &e) {   // a tensor without storage, for instance
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// describe(item, ...) -> bytes of int64 words
PyObject *describe(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    return packed(args, nargs, [&](Py_ssize_t i) { return kind_of(args[i]); });
}

// describe_call(kinds, item, ...) -> bytes of int64 words: the arguments of one operator, a letter of `kinds` for each
PyObject *describe_call(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    Py_ssize_t n = 0;
    const char *kinds = nargs > 0 ? PyUnicode_AsUTF8AndSize(args[0], &n) : "";
    if (!kinds) return nullptr;
    if (nargs < 1 || n != nargs - 1) {
        PyErr_SetString(PyExc_TypeError, "the kinds of the arguments and as many arguments are wanted");
        return nullptr;
    }
    return packed(args + 1, n, [&](Py_ssize_t i) { return kinds[i]; });
}

PyMethodDef methods[] = {
    {"describe", (PyCFunction)(void (*)(void))describe, METH_FASTCALL, "Packed description of items by themselves."},
    {"describe_call", (PyCFunction)(void (*)(void))describe_call, METH_FASTCALL, "Packed description of an operator's arguments."},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_describe", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__describe(void)
{
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "built_for", DESCRIBE_BUILT_FOR) < 0) Py_CLEAR(m);
    return m;
}
