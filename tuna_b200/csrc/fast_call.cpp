// The argument checks and the launch of `ops.matmul` in one native call.  In Python they take 8 us of host time, more than the
// kernel of a small layer (4096x4096 at 1 token 6.8 us), so a decode step's small GEMMs waited for the host.
//
// matmul(x, q, s, c, o, m, n, k) answers True when the GEMM was launched and False when anything is not as the
// common case has it - a wrong type, device, layout or size, no workspace yet, one too small.  Nothing has been launched
// then, and ops.py takes the call through its own checks, which raise what is wrong.  Any other status of the
// library is the answer itself: a call of several launches may have made some of them, and is not made again.
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/cuda/CUDAFunctions.h>
#include "../../include/tuna_b200.h"

namespace {

using MatmulFn = int (*)(const void *q, const void *x, const void *code, const void *absmax, void *o, int m, int n, int k, void *workspace,
                         size_t workspace_bytes, void *stream);

MatmulFn g_matmul = nullptr;
PyObject *g_workspaces = nullptr;  // the dict (device, stream) -> tensor that ops.py fills: there is no other record of them

// The workspace of a device and stream, with a reference of the caller's own: another thread may put a larger one in its
// place while this one is in use.  Null where there is none.
struct Workspace {
    PyObject *tensor = nullptr;
    Workspace(int device, void *stream)
    {
        PyObject *key = Py_BuildValue("(iK)", device, (unsigned long long)stream);
        PyObject *found = key ? PyDict_GetItemWithError(g_workspaces, key) : nullptr;
        Py_XDECREF(key);
        if (found && THPVariable_Check(found)) tensor = Py_NewRef(found);
        PyErr_Clear();
    }
    ~Workspace() { Py_XDECREF(tensor); }
    Workspace(const Workspace &) = delete;
    Workspace &operator=(const Workspace &) = delete;
    void *ptr() const { return THPVariable_Unpack(tensor).mutable_data_ptr(); }
    size_t bytes() const { return THPVariable_Unpack(tensor).nbytes(); }
};

// The interpreter lock is released for this object's life: a launch waits where the stream's queue is full, and other
// threads - one of which may be what the stream waits for - have to run meanwhile.
struct Unlocked {
    PyThreadState *state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
};

// The tensor of `o` if it is a plain contiguous CUDA tensor of `numel` elements of `type` on `device` (-1: any), else null.
const at::Tensor *plain(PyObject *o, at::ScalarType type, int64_t numel, int device)
{
    if (!THPVariable_CheckExact(o)) return nullptr;  // subclasses take the Python way
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.scalar_type() != type || t.layout() != at::kStrided || t.numel() != numel || !t.is_contiguous()) return nullptr;
    if (device >= 0 && t.get_device() != device) return nullptr;
    return &t;
}

constexpr int kPythonWay = 1;  // no status of the library: those are negative or TUNA_OK

int launch(PyObject *const *args)
{
    long long dim[3];
    for (int i = 0; i < 3; ++i) {
        if (!PyLong_CheckExact(args[5 + i])) return kPythonWay;
        int overflow = 0;
        dim[i] = PyLong_AsLongLongAndOverflow(args[5 + i], &overflow);
        if (overflow || dim[i] <= 0 || dim[i] > 0x7fffffff) return kPythonWay;
    }
    const long long m = dim[0], n = dim[1], k = dim[2];
    const at::Tensor *x = plain(args[0], at::kHalf, n * k, -1);
    if (!x) return kPythonWay;
    const int device = x->get_device();
    const at::Tensor *q = plain(args[1], at::kByte, m * k / 2, device), *s = plain(args[2], at::kFloat, m, device),
                     *c = plain(args[3], at::kFloat, 16, device), *o = plain(args[4], at::kHalf, n * m, device);
    if (!q || !s || !c || !o || device != c10::cuda::current_device()) return kPythonWay;
    void *stream = c10::cuda::getCurrentCUDAStream(device).stream();
    const Workspace ws(device, stream);
    if (!ws.tensor) return kPythonWay;
    const void *qp = q->const_data_ptr(), *xp = x->const_data_ptr(), *cp = c->const_data_ptr(), *sp = s->const_data_ptr();
    void *op = o->mutable_data_ptr(), *wp = ws.ptr();
    const size_t bytes = ws.bytes();
    const MatmulFn matmul = g_matmul;
    const Unlocked unlocked;  // the caller's arguments and `ws` keep the tensors
    const int st = matmul(qp, xp, cp, sp, op, (int)m, (int)n, (int)k, wp, bytes, stream);
    return st == TUNA_ERR_WORKSPACE ? kPythonWay : st;
}

PyObject *fast_matmul(PyObject *, PyObject *const *args, Py_ssize_t nargs)
{
    int st = kPythonWay;
    try {
        if (nargs == 8 && g_matmul) st = launch(args);
    } catch (...) {  // a tensor without storage of its own (vmap, a trace): the Python way says what is wrong
    }
    return st == TUNA_OK || st == kPythonWay ? PyBool_FromLong(st == TUNA_OK) : PyLong_FromLong(st);
}

// workspace(device, stream) -> (address, bytes) of the one that a launch there uses, or None
PyObject *workspace(PyObject *, PyObject *args)
{
    int device;
    unsigned long long stream;
    if (!PyArg_ParseTuple(args, "iK", &device, &stream)) return nullptr;
    if (!g_workspaces) Py_RETURN_NONE;
    const Workspace ws(device, (void *)stream);
    if (!ws.tensor) Py_RETURN_NONE;
    return Py_BuildValue("(KK)", (unsigned long long)ws.ptr(), (unsigned long long)ws.bytes());
}

// bind(address of tuna_matmul, dict of the workspaces)
PyObject *bind(PyObject *, PyObject *args)
{
    unsigned long long fn;
    PyObject *workspaces;
    if (!PyArg_ParseTuple(args, "KO!", &fn, &PyDict_Type, &workspaces)) return nullptr;
    g_matmul = (MatmulFn)fn;
    Py_XSETREF(g_workspaces, Py_NewRef(workspaces));
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"matmul", (PyCFunction)(void (*)(void))fast_matmul, METH_FASTCALL, nullptr},
    {"workspace", workspace, METH_VARARGS, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// torch's layouts are compiled in: _lib.py uses the module, and build.py keeps it, only where this names the torch and Python at hand.
#ifndef FAST_CALL_STAMP
#error "build.py says what this is built for"
#endif
PyMODINIT_FUNC PyInit__fast_call()
{
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "stamp", FAST_CALL_STAMP) < 0) Py_CLEAR(m);
    return m;
}
