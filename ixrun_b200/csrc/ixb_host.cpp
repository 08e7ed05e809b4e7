// The host side of a packed linear's call, as a Python extension: checks, output, stream and launch in one call from Python.
// Through ctypes and torch's Python functions the same takes 7 us, more than the kernel of a 2048 x 2048 layer; here 4, of which
// the launch is 3.  Anything out of the ordinary (another type, a subclass, a transform, a layout, a device) is left to the
// Python path: the call returns None.
#include <Python.h>
#include <structmember.h>

#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/SmallVector.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

using gemv_fn = int (*)(const void *, const void *, int64_t, const void *, void *, int, void *, size_t, void *);
using rows_fn = int (*)(const void *, const void *, int64_t, const void *, void *, int, void *);
gemv_fn g_gemv = nullptr;
rows_fn g_rows = nullptr;
PyObject *g_check = nullptr;                             // raises the library's error for a status

// The interpreter's lock, given up while torch allocates (which may wait for the device) and while a launch is made (which waits
// where the queue is full): another thread may be the one that would end the wait.
struct Unlocked {
    PyThreadState *state = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked &) = delete;
    ~Unlocked() { PyEval_RestoreThread(state); }
};

struct P6Call {
    PyObject_HEAD
    vectorcallfunc call;
    const void *tensor;                                  // the ixb_p6 structure (of the object that holds this one)
    int64_t out_f, in_f;
    int index;
    void *scratch;                                       // of ixb_p6_gemv
    size_t scratch_bytes;
    PyObject *keep;                                      // the scratch's tensor
};

// (x, bias or None, many): y = x W^T for 1..8 rows, and with `many` 9..64 rows of a layer whose in_f is a multiple of 64
PyObject *p6_call(PyObject *self_, PyObject *const *args, size_t nargsf, PyObject *kw)
{
    const P6Call *self = (const P6Call *)self_;
    if (PyVectorcall_NARGS(nargsf) != 3 || kw) {
        PyErr_SetString(PyExc_TypeError, "expected (x, bias, many)");
        return nullptr;
    }
    try {
        if (!THPVariable_Check(args[0])) Py_RETURN_NONE;
        const at::Tensor x = THPVariable_Unpack(args[0]);            // (held: other threads run below)
        if (x.scalar_type() != at::kBFloat16 || x.layout() != at::kStrided || !x.is_cuda() || x.get_device() != self->index ||
            at::isTensorSubclassLike(x) || x.is_neg() || x.dim() < 1 || x.size(-1) != self->in_f || !x.is_contiguous())
            Py_RETURN_NONE;
        const int64_t m = x.numel() / self->in_f;
        if (m < 1 || m > 64 || (m > 8 && (self->in_f % 64 || args[2] != Py_True))) Py_RETURN_NONE;
        const void *bias = nullptr;
        at::Tensor b;
        if (args[1] != Py_None) {
            if (!THPVariable_Check(args[1])) Py_RETURN_NONE;
            b = THPVariable_Unpack(args[1]);
            if (b.scalar_type() != at::kBFloat16 || b.numel() != self->out_f || !b.is_cuda() || b.get_device() != self->index || !b.is_contiguous())
                Py_RETURN_NONE;
            bias = b.data_ptr();
        }
        at::DimVector shape(x.sizes().begin(), x.sizes().end());
        shape.back() = self->out_f;
        at::Tensor y;
        int rc = 0;
        bool plain;
        {
            const Unlocked unlocked;
            c10::cuda::OptionalCUDAGuard guard;
            if (c10::cuda::current_device() != self->index) guard.set_index((c10::DeviceIndex)self->index);
            y = at::empty(shape, at::TensorOptions().dtype(at::kBFloat16).device(at::Device(at::kCUDA, (c10::DeviceIndex)self->index)));
            plain = !at::isTensorSubclassLike(y);
            if (plain) {
                void *stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->index).stream();
                rc = m <= 8 ? g_gemv(self->tensor, x.data_ptr(), m, bias, y.data_ptr(), 0, self->scratch, self->scratch_bytes, stream)
                            : g_rows(self->tensor, x.data_ptr(), m, bias, y.data_ptr(), 0, stream);
            }
        }
        if (!plain) Py_RETURN_NONE;
        if (rc) {
            PyObject *r = PyObject_CallFunction(g_check, "i", rc);
            Py_XDECREF(r);
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "packed linear failed");
            return nullptr;
        }
        return THPVariable_Wrap(std::move(y));
    } catch (...) {                                      // as torch's functions raise it: out of memory, an error of Python code
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

void p6_dealloc(PyObject *self_)
{
    Py_XDECREF(((P6Call *)self_)->keep);
    Py_TYPE(self_)->tp_free(self_);
}

PyMemberDef p6_members[] = {{"__vectorcalloffset__", T_PYSSIZET, offsetof(P6Call, call), READONLY, nullptr}, {nullptr, 0, 0, 0, nullptr}};
PyTypeObject P6CallType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// p6(structure address, out_f, in_f, device index, scratch tensor)
PyObject *new_p6(PyObject *, PyObject *args)
{
    unsigned long long tensor;
    long long out_f, in_f;
    int index;
    PyObject *scratch;
    if (!PyArg_ParseTuple(args, "KLLiO", &tensor, &out_f, &in_f, &index, &scratch)) return nullptr;
    if (!g_gemv || !THPVariable_Check(scratch) || out_f <= 0 || in_f <= 0) {
        PyErr_SetString(PyExc_ValueError, "p6: not bound, or bad arguments");
        return nullptr;
    }
    P6Call *c = PyObject_New(P6Call, &P6CallType);
    if (!c) return nullptr;
    c->call = p6_call;
    c->tensor = (const void *)(uintptr_t)tensor;
    c->out_f = out_f;
    c->in_f = in_f;
    c->index = index;
    const at::Tensor &s = THPVariable_Unpack(scratch);
    c->scratch = s.data_ptr();
    c->scratch_bytes = (size_t)s.numel() * s.element_size();
    c->keep = scratch;
    Py_INCREF(scratch);
    return (PyObject *)c;
}

// bind(address of ixb_p6_gemv, of ixb_p6_rows, check)
PyObject *bind(PyObject *, PyObject *args)
{
    unsigned long long gemv, rows;
    PyObject *check;
    if (!PyArg_ParseTuple(args, "KKO", &gemv, &rows, &check)) return nullptr;
    g_gemv = (gemv_fn)(uintptr_t)gemv;
    g_rows = (rows_fn)(uintptr_t)rows;
    Py_XDECREF(g_check);
    g_check = check;
    Py_INCREF(check);
    Py_RETURN_NONE;
}

// empty(device index, (n, type), (n, type), ...): uninitialised one-dimensional tensors (n < 0: of no dimension);
// type 'B' uint8, 'b' int8, 'i' int32, 'h' bfloat16
PyObject *empty(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    if (nargs < 1) {
        PyErr_SetString(PyExc_TypeError, "empty(index, (n, type), ...)");
        return nullptr;
    }
    const long index = PyLong_AsLong(args[0]);
    if (index < 0) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "expected a CUDA device");
        return nullptr;
    }
    struct Spec {
        long long n;
        int type;
    };
    try {
        c10::SmallVector<Spec, 8> specs((size_t)(nargs - 1));
        c10::SmallVector<at::Tensor, 8> tensors;
        for (Py_ssize_t i = 1; i < nargs; ++i)
            if (!PyArg_ParseTuple(args[i], "LC", &specs[i - 1].n, &specs[i - 1].type)) return nullptr;
        {
            const Unlocked unlocked;
            for (const Spec &s : specs) {
                const auto dt = s.type == 'B' ? at::kByte : s.type == 'b' ? at::kChar : s.type == 'i' ? at::kInt : at::kBFloat16;
                const int64_t size[1] = {s.n};
                tensors.push_back(at::empty(at::IntArrayRef(size, s.n < 0 ? 0 : 1), at::TensorOptions().dtype(dt).device(at::Device(at::kCUDA, (c10::DeviceIndex)index))));
            }
        }
        PyObject *out = PyTuple_New(nargs - 1);
        for (Py_ssize_t i = 0; out && i < nargs - 1; ++i) {
            PyObject *o = THPVariable_Wrap(std::move(tensors[i]));
            if (!o) {
                Py_DECREF(out);
                return nullptr;
            }
            PyTuple_SET_ITEM(out, i, o);
        }
        return out;
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

PyMethodDef methods[] = {{"p6", new_p6, METH_VARARGS, nullptr},
                         {"bind", bind, METH_VARARGS, nullptr},
                         {"empty", (PyCFunction)(void (*)(void))empty, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ixbhost", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ixbhost()
{
    P6CallType.tp_name = "ixrun_b200._ixbhost.P6Call";
    P6CallType.tp_basicsize = sizeof(P6Call);
    P6CallType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
    P6CallType.tp_vectorcall_offset = offsetof(P6Call, call);
    P6CallType.tp_call = PyVectorcall_Call;
    P6CallType.tp_dealloc = p6_dealloc;
    P6CallType.tp_members = p6_members;
    P6CallType.tp_free = PyObject_Free;
    if (PyType_Ready(&P6CallType) < 0) return nullptr;
    return PyModule_Create(&module);
}
