// Calls from Python into the kernels' C entry points, and the checks that go before them, without the cost of ctypes (a call of 20
// arguments 4 us, a checked pointer 0.35): a step of a small layer is bound by its host's calls, some ten of them with ten pointers each.
//
//   Function(address, signature, name)(...)   calls `int name(...)`; a letter an argument: p pointer (int or None), i int, l long long,
//                                             u unsigned long long, f float.  The GIL is released during the call.
//   pointer(tensor or None)                   the data pointer; a tensor that is not on a CUDA device is an error
//   need(tensor, dtype, name)                 dtype and contiguity;  need_columns(..): dtype and columns side by side
//   tiled_operands(x, w)                      whether a tensor-core product takes the two matrices
//   set_error(class)                          what the checks raise
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

static PyObject* error_class;

// The integer arguments of a call beyond those in registers lie on the stack in order, eight bytes each, and the float arguments in
// registers of their own (x86-64 System V and AArch64 Linux alike), so one prototype calls every entry point: what a function does not
// take it does not read.
#if defined(__x86_64__) && defined(__linux__)
enum { INTS = 6 };
#define CALL(a, f) ((int (*)(I6, F8, I40))address)(REG6(a), f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], STACK(a, 6))
#elif defined(__aarch64__) && defined(__linux__)
enum { INTS = 8 };
#define CALL(a, f) ((int (*)(I6, long long, long long, F8, I40))address)(REG6(a), a[6], a[7], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], STACK(a, 8))
#else
#error "no calling convention known for this machine"
#endif
#define I6 long long, long long, long long, long long, long long, long long
#define I8 I6, long long, long long
#define I40 I8, I8, I8, I8, I8
#define F8 float, float, float, float, float, float, float, float
#define REG6(a) a[0], a[1], a[2], a[3], a[4], a[5]
#define AT8(a, k) a[k], a[(k) + 1], a[(k) + 2], a[(k) + 3], a[(k) + 4], a[(k) + 5], a[(k) + 6], a[(k) + 7]
#define STACK(a, k) AT8(a, k), AT8(a, (k) + 8), AT8(a, (k) + 16), AT8(a, (k) + 24), AT8(a, (k) + 32)
enum { MAX_INTS = INTS + 40, MAX_FLOATS = 8 };

typedef struct {
    PyObject_HEAD
    vectorcallfunc call;
    void* address;
    PyObject *signature, *name;
    const char* letters;
    Py_ssize_t count;
} Function;

static PyObject* function_call(PyObject* self, PyObject* const* args, size_t flags, PyObject* names) {
    Function* fn = (Function*)self;
    const Py_ssize_t n = PyVectorcall_NARGS(flags);
    if (n != fn->count || (names && PyTuple_GET_SIZE(names))) {
        PyErr_Format(PyExc_TypeError, "%U takes %zd arguments (%zd given)", fn->name, fn->count, n);
        return NULL;
    }
    long long ints[MAX_INTS] = {0};
    float floats[MAX_FLOATS] = {0};
    int i = 0, f = 0;
    for (Py_ssize_t k = 0; k < n; ++k) {
        PyObject* arg = args[k];
        if (fn->letters[k] == 'f') {
            const double v = PyFloat_AsDouble(arg);
            if (v == -1.0 && PyErr_Occurred()) return NULL;
            floats[f++] = (float)v;
        } else if (fn->letters[k] == 'p' && arg == Py_None) {
            ints[i++] = 0;
        } else if (PyLong_Check(arg)) {
            const unsigned long long v = PyLong_AsUnsignedLongLongMask(arg);
            if (v == (unsigned long long)-1 && PyErr_Occurred()) return NULL;
            ints[i++] = fn->letters[k] == 'i' ? (long long)(int)v : (long long)v;
        } else {
            PyErr_Format(PyExc_TypeError, "%U: argument %zd must be an int, not %s", fn->name, k + 1, Py_TYPE(arg)->tp_name);
            return NULL;
        }
    }
    void* address = fn->address;
    int code;
    Py_BEGIN_ALLOW_THREADS
    code = CALL(ints, floats);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(code);
}

static PyObject* function_new(PyTypeObject* type, PyObject* args, PyObject* kwargs) {
    unsigned long long address;
    PyObject *signature, *name;
    if (!PyArg_ParseTuple(args, "KUU", &address, &signature, &name)) return NULL;
    Py_ssize_t count;
    const char* letters = PyUnicode_AsUTF8AndSize(signature, &count);
    if (!letters) return NULL;
    int ints = 0, floats = 0;
    for (Py_ssize_t k = 0; k < count; ++k) {
        if (letters[k] == 'f') ++floats;
        else if (letters[k] == 'p' || letters[k] == 'i' || letters[k] == 'l' || letters[k] == 'u') ++ints;
        else return PyErr_Format(PyExc_ValueError, "%U: no argument type %c", name, letters[k]);
    }
    if (!address || ints > MAX_INTS || floats > MAX_FLOATS) return PyErr_Format(PyExc_ValueError, "%U: no address, or too many arguments", name);
    Function* fn = (Function*)type->tp_alloc(type, 0);
    if (!fn) return NULL;
    fn->call = function_call;
    fn->address = (void*)(uintptr_t)address;
    Py_INCREF(signature);
    Py_INCREF(name);
    fn->signature = signature;
    fn->name = name;
    fn->letters = letters;
    fn->count = count;
    return (PyObject*)fn;
}

static void function_free(PyObject* self) {
    Py_XDECREF(((Function*)self)->signature);
    Py_XDECREF(((Function*)self)->name);
    Py_TYPE(self)->tp_free(self);
}

static PyTypeObject function_type = {PyVarObject_HEAD_INIT(NULL, 0)};

// torch's checks may throw (tensors without storage, layouts without strides)
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
static PyObject* guarded(PyObject* module, PyObject* const* args, Py_ssize_t n) {
    try {
        return F(module, args, n);
    } catch (const std::exception& error) {
        PyErr_SetString(PyExc_RuntimeError, error.what());
        return NULL;
    }
}

// the tensor behind an object, or null with an error
static const at::Tensor* tensor_of(PyObject* object) {
    if (THPVariable_Check(object)) return &THPVariable_Unpack(object);
    PyErr_Format(PyExc_TypeError, "expected a tensor, not %s", Py_TYPE(object)->tp_name);
    return NULL;
}

static PyObject* host_pointer(PyObject* module, PyObject* const* args, Py_ssize_t n) {
    if (n != 1) return PyErr_Format(PyExc_TypeError, "pointer takes a tensor or None");
    PyObject* object = args[0];
    if (object == Py_None) return PyLong_FromLong(0);
    const at::Tensor* tensor = tensor_of(object);
    if (!tensor) return NULL;
    if (tensor->is_cuda()) return PyLong_FromUnsignedLongLong((unsigned long long)(uintptr_t)tensor->mutable_data_ptr());
    return PyErr_Format(error_class, "thintensor_b200 kernels run on CUDA tensors only; got a tensor on %s", tensor->device().str().c_str());
}

// the tensor where it has the dtype, null with an error otherwise
static const at::Tensor* with_dtype(PyObject* object, PyObject* dtype, PyObject* name) {
    const at::Tensor* tensor = tensor_of(object);
    if (!tensor) return NULL;
    if (!THPDtype_Check(dtype)) {
        PyErr_Format(PyExc_TypeError, "expected a dtype, not %s", Py_TYPE(dtype)->tp_name);
        return NULL;
    }
    if (tensor->scalar_type() == ((THPDtype*)dtype)->scalar_type) return tensor;
    PyObject* own = PyObject_GetAttrString(object, "dtype");
    if (own) PyErr_Format(error_class, "%U must be %S, got %S", name, dtype, own);
    Py_XDECREF(own);
    return NULL;
}

static PyObject* host_need(PyObject* module, PyObject* const* args, Py_ssize_t n) {
    if (n != 3) return PyErr_Format(PyExc_TypeError, "need takes a tensor, a dtype and a name");
    const at::Tensor* tensor = with_dtype(args[0], args[1], args[2]);
    if (!tensor) return NULL;
    if (!tensor->is_contiguous()) return PyErr_Format(error_class, "%U must be contiguous", args[2]);
    Py_RETURN_NONE;
}

static PyObject* host_need_columns(PyObject* module, PyObject* const* args, Py_ssize_t n) {
    if (n != 3) return PyErr_Format(PyExc_TypeError, "need_columns takes a tensor, a dtype and a name");
    const at::Tensor* tensor = with_dtype(args[0], args[1], args[2]);
    if (!tensor) return NULL;
    if (tensor->dim() < 1 || tensor->strides().back() != 1) return PyErr_Format(error_class, "%U must have its columns side by side", args[2]);
    Py_RETURN_NONE;
}

// rows of bfloat16 numbers that a tiled copy can address: 16-byte aligned base and row stride, whole 16-byte rows, columns side by side
static bool tiled_rows(const at::Tensor& tensor) {
    return tensor.scalar_type() == at::kBFloat16 && tensor.dim() == 2 && tensor.stride(0) % 8 == 0 && tensor.stride(1) == 1
        && reinterpret_cast<uintptr_t>(tensor.mutable_data_ptr()) % 16 == 0;
}

static PyObject* host_tiled_operands(PyObject* module, PyObject* const* args, Py_ssize_t n) {
    if (n != 2) return PyErr_Format(PyExc_TypeError, "tiled_operands takes two tensors");
    const at::Tensor *x = tensor_of(args[0]), *w = x ? tensor_of(args[1]) : NULL;
    if (!w) return NULL;
    return PyBool_FromLong(tiled_rows(*x) && tiled_rows(*w) && x->size(1) % 8 == 0);
}

static PyObject* host_set_error(PyObject* module, PyObject* error) {
    Py_INCREF(error);
    Py_XSETREF(error_class, error);
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"pointer", (PyCFunction)(void (*)(void))guarded<host_pointer>, METH_FASTCALL, "The data pointer of a CUDA tensor; 0 for None."},
    {"need", (PyCFunction)(void (*)(void))guarded<host_need>, METH_FASTCALL, "Check a tensor's dtype and contiguity."},
    {"need_columns", (PyCFunction)(void (*)(void))guarded<host_need_columns>, METH_FASTCALL, "Check a tensor's dtype and that its columns lie side by side."},
    {"tiled_operands", (PyCFunction)(void (*)(void))guarded<host_tiled_operands>, METH_FASTCALL, "Whether two matrices can be the operands of a tiled bfloat16 product."},
    {"set_error", host_set_error, METH_O, "The exception class for refused tensors."},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef definition = {PyModuleDef_HEAD_INIT, "host_calls", "Calls into the kernels' C entry points.", -1, methods};

PyMODINIT_FUNC PyInit_host_calls(void) {
    function_type.tp_name = "host_calls.Function";
    function_type.tp_basicsize = sizeof(Function);
    function_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
    function_type.tp_vectorcall_offset = offsetof(Function, call);
    function_type.tp_call = PyVectorcall_Call;
    function_type.tp_new = function_new;
    function_type.tp_dealloc = function_free;
    if (PyType_Ready(&function_type) < 0) return NULL;
    error_class = PyExc_RuntimeError;
    Py_INCREF(error_class);
    PyObject* module = PyModule_Create(&definition);
    if (!module) return NULL;
    Py_INCREF(&function_type);
    if (PyModule_AddObject(module, "Function", (PyObject*)&function_type) < 0) return NULL;
    return module;
}
