// The way from Python to the kernels' launchers: a Python module of five functions.  A step of few tokens is a handful of launches of a few
// microseconds each, and through ctypes making a launcher's arguments (an object each), checking its tensors and asking for its outputs took
// longer than the launches: one token through Mamba-2's convolution and recurrence 27 us of the host for 6 us of the GPU.
//
//     call(address, *arguments)           the launcher at `address`: None, tensors (their data's address), whole numbers, floats (32-bit), or
//                                         ctypes objects where another type is wanted (double, unsigned, 64-bit)
//     fits(tensor, dtype, dimensions)     whether it is a contiguous CUDA tensor of this type (None: any) and number of dimensions (None: any)
//     empty(shape, dtype=, device=)       torch.empty for these arguments
//     same(x)                             x
//     fill(array, numbers)                a list's whole numbers into a contiguous array of as many 32-bit ones; False where the list holds anything
//                                         else, or a number that does not fit: the array then holds any part of them
//
// Launchers take integers, pointers, floats and doubles and return an int.  On x86-64 (System V) integers and pointers go into six registers
// and then onto the stack, in their order, floats and doubles into eight registers of their own, so one function type with many integers
// behind each other and eight doubles calls any of them; what a launcher does not take it does not look at.
#include <Python.h>

#include <ATen/ops/empty.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>

#if !defined(__x86_64__) || defined(_WIN32)
#error "calls by the System V convention of x86-64"
#endif

#define QWB_MAX_WHOLE 56
#define QWB_MAX_REAL 8

namespace {

struct WithoutGil {
    PyThreadState* state = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

typedef int (*Launcher)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                        uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                        uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                        uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                        double, double, double, double, double, double, double, double);

double bits_of(float f) {               // a float argument is the low half of its register
    uint64_t b = 0;
    std::memcpy(&b, &f, sizeof f);
    double d;
    std::memcpy(&d, &b, sizeof d);
    return d;
}

// A ctypes object: its `value`, of the type that `_type_` names
bool from_ctypes(PyObject* o, uint64_t& whole, double& real, bool& is_real) {
    PyObject* type = PyObject_GetAttrString(o, "_type_");
    PyObject* value = type ? PyObject_GetAttrString(o, "value") : nullptr;
    bool ok = value && PyUnicode_Check(type) && PyUnicode_GetLength(type) == 1;
    if (ok) {
        const Py_UCS4 t = PyUnicode_ReadChar(type, 0);
        is_real = t == 'd' || t == 'f';
        if (is_real) {
            const double v = PyFloat_AsDouble(value);
            real = t == 'd' ? v : bits_of((float)v);
        } else if (value == Py_None) {
            whole = 0;
        } else {
            whole = PyLong_AsUnsignedLongLongMask(value);
        }
        ok = !PyErr_Occurred();
    } else if (!PyErr_Occurred()) {
        PyErr_Format(PyExc_TypeError, "call: an argument of type %s", Py_TYPE(o)->tp_name);
    }
    Py_XDECREF(type);
    Py_XDECREF(value);
    return ok;
}

PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n < 1) return PyErr_Format(PyExc_TypeError, "call: no function");
    void* address = PyLong_AsVoidPtr(args[0]);
    if (!address) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "call: no function");
    uint64_t w[QWB_MAX_WHOLE] = {};
    double r[QWB_MAX_REAL] = {};
    int whole = 0, real = 0;
    for (Py_ssize_t i = 1; i < n; ++i) {
        PyObject* o = args[i];
        uint64_t v = 0;
        double d = 0.0;
        bool is_real = false;
        if (PyLong_Check(o)) {
            v = PyLong_AsUnsignedLongLongMask(o);
            if (v == (uint64_t)-1 && PyErr_Occurred()) return nullptr;
        } else if (o == Py_None) {
            v = 0;
        } else if (PyFloat_Check(o)) {
            d = bits_of((float)PyFloat_AS_DOUBLE(o));
            is_real = true;
        } else if (THPVariable_Check(o)) {
            v = (uint64_t)THPVariable_Unpack(o).mutable_data_ptr();
        } else if (!from_ctypes(o, v, d, is_real)) {
            return nullptr;
        }
        if (is_real ? real == QWB_MAX_REAL : whole == QWB_MAX_WHOLE) return PyErr_Format(PyExc_TypeError, "call: too many arguments");
        if (is_real) r[real++] = d;
        else w[whole++] = v;
    }
    int rc;
    {
        WithoutGil gil;
        rc = reinterpret_cast<Launcher>(address)(
            w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], w[9], w[10], w[11], w[12], w[13], w[14], w[15], w[16], w[17], w[18], w[19], w[20], w[21], w[22],
            w[23], w[24], w[25], w[26], w[27], w[28], w[29], w[30], w[31], w[32], w[33], w[34], w[35], w[36], w[37], w[38], w[39], w[40], w[41], w[42], w[43], w[44],
            w[45], w[46], w[47], w[48], w[49], w[50], w[51], w[52], w[53], w[54], w[55], r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7]);
    }
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

PyObject* fits(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 3 || !THPVariable_Check(args[0])) Py_RETURN_FALSE;
    const at::Tensor& t = THPVariable_Unpack(args[0]);
    bool ok = t.is_cuda() && t.is_contiguous();
    if (ok && args[1] != Py_None) ok = THPDtype_Check(args[1]) && t.scalar_type() == reinterpret_cast<THPDtype*>(args[1])->scalar_type;
    if (ok && args[2] != Py_None) ok = t.dim() == PyLong_AsLong(args[2]);
    if (PyErr_Occurred()) return nullptr;
    return PyBool_FromLong(ok);
    END_HANDLE_TH_ERRORS
}

PyObject* torch_empty = nullptr;

PyObject* empty(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* names) {
    HANDLE_TH_ERRORS
    PyObject *dtype = nullptr, *device = nullptr;
    bool plain = n == 1 && names && PyTuple_GET_SIZE(names) == 2 && PyTuple_CheckExact(args[0]) && PyTuple_GET_SIZE(args[0]) <= 8;
    for (Py_ssize_t i = 0; plain && i < 2; ++i) {
        PyObject* name = PyTuple_GET_ITEM(names, i);
        if (PyUnicode_CompareWithASCIIString(name, "dtype") == 0) dtype = args[1 + i];
        else if (PyUnicode_CompareWithASCIIString(name, "device") == 0) device = args[1 + i];
    }
    plain = plain && dtype && device && THPDtype_Check(dtype) && THPDevice_Check(device);
    int64_t sizes[8];
    const Py_ssize_t dims = plain ? PyTuple_GET_SIZE(args[0]) : 0;
    for (Py_ssize_t i = 0; plain && i < dims; ++i) {
        PyObject* o = PyTuple_GET_ITEM(args[0], i);
        plain = PyLong_Check(o);
        if (plain) sizes[i] = PyLong_AsLongLong(o);
    }
    if (PyErr_Occurred()) return nullptr;
    if (!plain) return PyObject_Vectorcall(torch_empty, args, n, names);      // whatever else torch takes
    const auto options = at::TensorOptions().dtype(reinterpret_cast<THPDtype*>(dtype)->scalar_type).device(reinterpret_cast<THPDevice*>(device)->device);
    at::Tensor t;
    {
        WithoutGil gil;
        t = at::empty(at::IntArrayRef(sizes, (size_t)dims), options);
    }
    return THPVariable_Wrap(std::move(t));
    END_HANDLE_TH_ERRORS
}

PyObject* same(PyObject*, PyObject* x) {
    Py_INCREF(x);
    return x;
}

PyObject* fill(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 2 || !PyList_CheckExact(args[1])) Py_RETURN_FALSE;
    Py_buffer to;
    if (PyObject_GetBuffer(args[0], &to, PyBUF_WRITABLE | PyBUF_FORMAT | PyBUF_C_CONTIGUOUS)) return nullptr;
    const Py_ssize_t count = PyList_GET_SIZE(args[1]);
    bool ok = to.itemsize == 4 && to.len == 4 * count && to.format && std::strcmp(to.format, "i") == 0;
    int32_t* out = static_cast<int32_t*>(to.buf);
    for (Py_ssize_t i = 0; ok && i < count; ++i) {
        PyObject* o = PyList_GET_ITEM(args[1], i);
        int overflow = 0;
        const long v = PyLong_CheckExact(o) ? PyLong_AsLongAndOverflow(o, &overflow) : INT64_MAX;
        ok = !overflow && v >= INT32_MIN && v <= INT32_MAX;
        if (ok) out[i] = (int32_t)v;
    }
    PyBuffer_Release(&to);
    return PyBool_FromLong(ok);
}

PyMethodDef methods[] = {{"call", (PyCFunction)(void*)call, METH_FASTCALL, nullptr},
                         {"fits", (PyCFunction)(void*)fits, METH_FASTCALL, nullptr},
                         {"empty", (PyCFunction)(void*)empty, METH_FASTCALL | METH_KEYWORDS, nullptr},
                         {"same", same, METH_O, nullptr},
                         {"fill", (PyCFunction)(void*)fill, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "qwb_host_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_qwb_host_call() {
    PyObject* torch = PyImport_ImportModule("torch");
    if (!torch) return nullptr;
    torch_empty = PyObject_GetAttrString(torch, "empty");
    Py_DECREF(torch);
    return torch_empty ? PyModule_Create(&module_def) : nullptr;
}
