// _host -- the calls of the Python layer whose inputs are plain, from the tensors to the launches: checks,
// output tensors and liba2a.so's entry points without an interpreter in between.  What it finds unusual (another
// type, shape, layout, place or device, a recorded error, a closed context) it leaves alone and answers None:
// the Python code then looks again and converts, raises or runs it, so what is accepted and how errors read is
// decided there and nowhere else.
//
// One call of one rank costs the host 4.4 us where the interpreter took 9.9, a
// histogram 2.6 / 5.9, the three launches for eight ranks 18 / 53 (of which the launches 7.5, the outputs 6), four
// phases of four ranks 14.6 / 39.
#include <Python.h>
#include <structmember.h>

#include <ATen/ops/empty.h>
#include <ATen/ops/empty_cuda_dispatch.h>
#include <ATen/record_function.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "a2a.h"

namespace {

// A context as this layer sees it: the library's handle (nullptr once closed) and what its tensors look like.
struct Rank {
    PyObject_HEAD
    a2a_ctx* ctx;
    int device, topk, hidden;
    int tokens;  // of the current call
    at::ScalarType dtype;
};

PyTypeObject* rank_type = nullptr;
PyObject *s_native, *s_x, *s_indices, *s_weights, *s_keep, *s_y;  // interned attribute names

// A plain tensor (no subclass, no wrapper without memory) of `dtype` in `device`'s memory, contiguous.
const at::Tensor* plain(PyObject* o, at::ScalarType dtype, int device) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || t.layout() != at::kStrided || !t.is_cuda() || !t.unsafeGetTensorImpl()->has_storage()) return nullptr;
    if (t.scalar_type() != dtype || t.get_device() != device || !t.is_contiguous()) return nullptr;
    return &t;
}

const at::Tensor* matrix(PyObject* o, at::ScalarType dtype, int device, int64_t rows, int64_t cols) {
    const at::Tensor* t = plain(o, dtype, device);
    return t != nullptr && t->dim() == 2 && t->size(1) == cols && (rows < 0 || t->size(0) == rows) ? t : nullptr;
}

// The tensors of a rank's call; false where one is not plain.
bool call_of(const Rank* r, PyObject* x, PyObject* idx, PyObject* w, a2a_call& c) {
    const at::Tensor* tx = matrix(x, r->dtype, r->device, -1, r->hidden);
    if (tx == nullptr || tx->size(0) > INT32_MAX) return false;
    const int64_t n = tx->size(0);
    const at::Tensor* ti = matrix(idx, at::kInt, r->device, n, r->topk);
    const at::Tensor* tw = matrix(w, at::kFloat, r->device, n, r->topk);
    if (ti == nullptr || tw == nullptr) return false;
    c.x = tx->const_data_ptr();
    c.topk_idx = static_cast<const int32_t*>(ti->const_data_ptr());
    c.topk_weights = static_cast<const float*>(tw->const_data_ptr());
    c.num_tokens = (int32_t)n;
    return true;
}

at::Tensor output_of(const Rank* r, a2a_call& c) {
    const at::TensorOptions options = at::TensorOptions().dtype(r->dtype).device(at::kCUDA, (c10::DeviceIndex)r->device);
    // the allocation itself, unless a mode or an observer (a profiler) wants to hear of operators
    const bool heard = c10::impl::dispatch_mode_enabled() || at::hasCallbacks();
    at::Tensor y = heard ? at::empty({c.num_tokens, r->hidden}, options) : at::cuda::empty({c.num_tokens, r->hidden}, options);
    c.y = y.mutable_data_ptr();
    return y;
}

// forward(x, indices, weights, look): the output, a status code (int) or None.  look: None too where a kernel of the
// context has recorded an error.
PyObject* rank_forward(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
    Rank* r = reinterpret_cast<Rank*>(self);
    if (nargs != 4) {
        PyErr_SetString(PyExc_TypeError, "forward takes x, indices, weights and a truth value");
        return nullptr;
    }
    if (r->ctx == nullptr || (args[3] == Py_True && a2a_status_peek(r->ctx) != 0)) Py_RETURN_NONE;
    HANDLE_TH_ERRORS
    if (c10::cuda::current_device() != r->device) Py_RETURN_NONE;
    a2a_call c;
    if (!call_of(r, args[0], args[1], args[2], c)) Py_RETURN_NONE;
    at::Tensor y = output_of(r, c);
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = a2a_forward(r->ctx, c.x, c.topk_idx, c.topk_weights, c.y, c.num_tokens, stream);
    Py_END_ALLOW_THREADS
    r->tokens = c.num_tokens;
    if (rc != A2A_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

PyObject* rank_close(PyObject* self, PyObject*) {
    reinterpret_cast<Rank*>(self)->ctx = nullptr;
    Py_RETURN_NONE;
}

// Rank(handle, device, topk, hidden, dtype)
PyObject* rank_new(PyTypeObject* type, PyObject* args, PyObject*) {
    unsigned long long handle;
    int device, topk, hidden;
    PyObject* dtype;
    if (!PyArg_ParseTuple(args, "KiiiO", &handle, &device, &topk, &hidden, &dtype)) return nullptr;
    if (!THPDtype_Check(dtype)) {
        PyErr_SetString(PyExc_TypeError, "not a torch.dtype");
        return nullptr;
    }
    Rank* r = reinterpret_cast<Rank*>(type->tp_alloc(type, 0));
    if (r == nullptr) return nullptr;
    r->ctx = reinterpret_cast<a2a_ctx*>(handle);
    r->device = device;
    r->topk = topk;
    r->hidden = hidden;
    r->dtype = reinterpret_cast<THPDtype*>(dtype)->scalar_type;
    return reinterpret_cast<PyObject*>(r);
}

struct Ref {  // a reference given back at the end of its scope
    PyObject* o = nullptr;
    ~Ref() { Py_XDECREF(o); }
};

// group_forward(contexts, rank data, phases, pipelined): those phases of a call on a whole group; the outputs, a status
// code (int) or None.  `pipelined`: role 2 rank by rank may answer with the outputs, which the contexts therefore keep.
PyObject* group_forward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 4 || !PyList_Check(args[0]) || !PyTuple_Check(args[2])) {
        PyErr_SetString(PyExc_TypeError, "group_forward takes a list of contexts, their data, a tuple of phases and a truth value");
        return nullptr;
    }
    const Py_ssize_t n = PyList_GET_SIZE(args[0]);
    const bool pipelined = args[3] == Py_True;
    if (n < 1 || n > A2A_MAX_WORLD || !(PyList_Check(args[1]) || PyTuple_Check(args[1])) || PySequence_Fast_GET_SIZE(args[1]) < n)
        Py_RETURN_NONE;
    int32_t phases[4];
    const Py_ssize_t num_phases = PyTuple_GET_SIZE(args[2]);
    if (num_phases > 4) Py_RETURN_NONE;
    for (Py_ssize_t i = 0; i < num_phases; ++i) {
        phases[i] = (int)PyLong_AsLong(PyTuple_GET_ITEM(args[2], i));
        if (PyErr_Occurred()) return nullptr;
    }
    HANDLE_TH_ERRORS
    Ref native[A2A_MAX_WORLD], x[A2A_MAX_WORLD], idx[A2A_MAX_WORLD], w[A2A_MAX_WORLD];
    a2a_ctx* group[A2A_MAX_WORLD];
    a2a_call calls[A2A_MAX_WORLD];
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* data = PySequence_Fast_GET_ITEM(args[1], i);
        if ((native[i].o = PyObject_GetAttr(PyList_GET_ITEM(args[0], i), s_native)) == nullptr ||
            (x[i].o = PyObject_GetAttr(data, s_x)) == nullptr || (idx[i].o = PyObject_GetAttr(data, s_indices)) == nullptr ||
            (w[i].o = PyObject_GetAttr(data, s_weights)) == nullptr) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        if (!PyObject_TypeCheck(native[i].o, rank_type)) Py_RETURN_NONE;
        const Rank* r = reinterpret_cast<Rank*>(native[i].o);
        if (r->ctx == nullptr || c10::cuda::current_device() != r->device || !call_of(r, x[i].o, idx[i].o, w[i].o, calls[i]))
            Py_RETURN_NONE;
        group[i] = r->ctx;
    }
    at::Tensor ys[A2A_MAX_WORLD];
    for (Py_ssize_t i = 0; i < n; ++i) ys[i] = output_of(reinterpret_cast<Rank*>(native[i].o), calls[i]);
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    int32_t through = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = a2a_group_steps(group, phases, (int)num_phases, calls, stream, &through);
    Py_END_ALLOW_THREADS
    if (through == 0) return PyLong_FromLong(rc);  // nothing begun
    Ref out;
    if ((out.o = PyList_New(n)) == nullptr) return nullptr;
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* y = THPVariable_Wrap(std::move(ys[i]));
        if (y == nullptr) return nullptr;
        PyList_SET_ITEM(out.o, i, y);
        reinterpret_cast<Rank*>(native[i].o)->tokens = calls[i].num_tokens;
        PyObject* ctx = PyList_GET_ITEM(args[0], i);
        Ref keep;
        keep.o = pipelined ? Py_BuildValue("[OOOO]", x[i].o, idx[i].o, w[i].o, y) : Py_BuildValue("[OOO]", idx[i].o, x[i].o, w[i].o);
        if (keep.o == nullptr || PyObject_SetAttr(ctx, s_keep, keep.o) < 0) return nullptr;
        if (pipelined && PyObject_SetAttr(ctx, s_y, y) < 0) return nullptr;
    }
    if (rc != A2A_OK) return PyLong_FromLong(rc);
    PyObject* got = out.o;
    out.o = nullptr;
    return got;
    END_HANDLE_TH_ERRORS
}

// histogram(data, output): output, a status code (int) or None.
PyObject* histogram(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 2) {
        PyErr_SetString(PyExc_TypeError, "histogram takes data and output");
        return nullptr;
    }
    HANDLE_TH_ERRORS
    if (!THPVariable_CheckExact(args[0]) || !THPVariable_Unpack(args[0]).is_cuda()) Py_RETURN_NONE;
    const int device = c10::cuda::current_device();
    const at::Tensor* data = plain(args[0], at::kByte, device);
    const at::Tensor* out = plain(args[1], at::kLong, device);
    if (data == nullptr || out == nullptr || data->dim() != 1 || out->numel() != 256) Py_RETURN_NONE;
    const uint8_t* from = static_cast<const uint8_t*>(data->const_data_ptr());
    const size_t n = (size_t)data->numel();
    int64_t* to = static_cast<int64_t*>(out->mutable_data_ptr());
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = a2a_histogram256(from, n, to, stream);
    Py_END_ALLOW_THREADS
    if (rc != A2A_OK) return PyLong_FromLong(rc);
    Py_INCREF(args[1]);
    return args[1];
    END_HANDLE_TH_ERRORS
}

PyMethodDef rank_methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(rank_forward)), METH_FASTCALL, nullptr},
    {"close", rank_close, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyMemberDef rank_members[] = {{"tokens", T_INT, offsetof(Rank, tokens), 0, nullptr}, {nullptr, 0, 0, 0, nullptr}};

PyType_Slot rank_slots[] = {{Py_tp_new, reinterpret_cast<void*>(rank_new)},
                            {Py_tp_methods, rank_methods},
                            {Py_tp_members, rank_members},
                            {0, nullptr}};

PyType_Spec rank_spec = {"_host.Rank", sizeof(Rank), 0, Py_TPFLAGS_DEFAULT, rank_slots};

PyMethodDef module_methods[] = {
    {"group_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(group_forward)), METH_FASTCALL, nullptr},
    {"histogram", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(histogram)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    s_native = PyUnicode_InternFromString("_native");
    s_x = PyUnicode_InternFromString("x");
    s_indices = PyUnicode_InternFromString("indices");
    s_weights = PyUnicode_InternFromString("weights");
    s_keep = PyUnicode_InternFromString("_keep");
    s_y = PyUnicode_InternFromString("_y");
    rank_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&rank_spec));
    PyObject* m = PyModule_Create(&module_def);
    if (rank_type == nullptr || m == nullptr) return nullptr;
    if (PyModule_AddObjectRef(m, "Rank", reinterpret_cast<PyObject*>(rank_type)) < 0) return nullptr;
    return m;
}
