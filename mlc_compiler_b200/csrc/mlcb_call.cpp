// The steady-state call of a one-kernel schedule, in native code: check the inputs, take
// their addresses, enqueue the kernel on the caller's stream, return the output object.
// Done in Python these checks take longer than a small kernel runs: a call of LayerNorm
// [128, 768] took 5.6 us on the host, of which the driver's launch is about 2.
//
// Built against the torch it is loaded with (build.py); without it the Python form in
// executor.py does the same.

#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <vector>

namespace {

typedef int (*LaunchFn)(void*, uint32_t, uint32_t, uint32_t, const uint64_t*, int, uint64_t, uint32_t);

struct Input {
    std::vector<int64_t> shape;
    int dtype;
    uint64_t bytes;
    std::vector<int> slots;
};

struct Call {
    PyObject_HEAD
    LaunchFn launch;
    void* kernel;
    uint32_t grid, block, smem, flags;
    int device;
    std::vector<uint64_t>* ptrs;
    std::vector<Input>* inputs;
    std::vector<std::pair<uint64_t, uint64_t>>* written;
    PyObject* out;    // what a call returns
    PyObject* fail;   // called with a launch's error code, with 0 when `fault` is set
    PyObject* last;   // inputs of the last call, or None
    volatile uint32_t* fault;   // set when a wait inside the kernel has run out; null: it has none
};

void call_free(PyObject* self) {
    Call* c = (Call*)self;
    delete c->ptrs;
    delete c->inputs;
    delete c->written;
    Py_XDECREF(c->out);
    Py_XDECREF(c->fail);
    Py_XDECREF(c->last);
    PyTypeObject* t = Py_TYPE(self);
    t->tp_free(self);
    Py_DECREF(t);
}

// Call(launch, kernel, grid, block, smem, flags, device, ptrs, inputs, written, out, fail, fault)
// inputs: [(shape, exemplar tensor, bytes, slots)], written: [(begin, end)]
PyObject* call_new(PyTypeObject* type, PyObject* args, PyObject*) {
    HANDLE_TH_ERRORS
    unsigned long long launch, kernel, fault;
    unsigned grid, block, smem, flags;
    int device;
    PyObject *ptrs, *inputs, *written, *out, *fail;
    if (!PyArg_ParseTuple(args, "KKIIIIiO!O!O!OOK", &launch, &kernel, &grid, &block, &smem, &flags, &device,
                          &PyList_Type, &ptrs, &PyList_Type, &inputs, &PyList_Type, &written, &out, &fail, &fault))
        return nullptr;
    Call* c = (Call*)type->tp_alloc(type, 0);
    if (!c) return nullptr;
    c->launch = (LaunchFn)(uintptr_t)launch;
    c->kernel = (void*)(uintptr_t)kernel;
    c->grid = grid; c->block = block; c->smem = smem; c->flags = flags;
    c->device = device;
    c->fault = (volatile uint32_t*)(uintptr_t)fault;
    c->ptrs = new std::vector<uint64_t>();
    c->inputs = new std::vector<Input>();
    c->written = new std::vector<std::pair<uint64_t, uint64_t>>();
    Py_INCREF(out); c->out = out;
    Py_INCREF(fail); c->fail = fail;
    Py_INCREF(Py_None); c->last = Py_None;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(ptrs); ++i)
        c->ptrs->push_back(PyLong_AsUnsignedLongLong(PyList_GET_ITEM(ptrs, i)));
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(inputs); ++i) {
        PyObject *shape, *exemplar, *slots;
        unsigned long long bytes;
        if (!PyArg_ParseTuple(PyList_GET_ITEM(inputs, i), "O!OKO!", &PyTuple_Type, &shape, &exemplar, &bytes,
                              &PyTuple_Type, &slots)) { Py_DECREF(c); return nullptr; }
        if (!THPVariable_Check(exemplar)) {
            PyErr_SetString(PyExc_TypeError, "expected a tensor that names the input's type");
            Py_DECREF(c);
            return nullptr;
        }
        Input in;
        for (Py_ssize_t j = 0; j < PyTuple_GET_SIZE(shape); ++j)
            in.shape.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(shape, j)));
        in.dtype = (int)THPVariable_Unpack(exemplar).scalar_type();
        in.bytes = bytes;
        for (Py_ssize_t j = 0; j < PyTuple_GET_SIZE(slots); ++j) {
            const long slot = PyLong_AsLong(PyTuple_GET_ITEM(slots, j));
            if (!PyErr_Occurred() && (slot < 0 || (size_t)slot >= c->ptrs->size()))
                PyErr_SetString(PyExc_ValueError, "an input's slot is none of the pointers");
            if (PyErr_Occurred()) { Py_DECREF(c); return nullptr; }
            in.slots.push_back((int)slot);
        }
        c->inputs->push_back(std::move(in));
    }
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(written); ++i) {
        unsigned long long lo, hi;
        if (!PyArg_ParseTuple(PyList_GET_ITEM(written, i), "KK", &lo, &hi)) { Py_DECREF(c); return nullptr; }
        c->written->emplace_back(lo, hi);
    }
    if (PyErr_Occurred() || c->ptrs->size() > 64) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "more than 64 pointers");
        Py_DECREF(c);
        return nullptr;
    }
    return (PyObject*)c;
    END_HANDLE_TH_ERRORS
}

PyObject* refuse(Call* c) {
    Py_INCREF(Py_None);
    Py_SETREF(c->last, Py_None);
    Py_RETURN_NONE;
}

// Whether input `in` can be read where `t` has it, and where that is.  Asking a tensor that
// stands for another one (a wrapper, a nested or batched tensor) throws: it cannot.
bool in_place(const Call* c, const Input& in, const at::Tensor& t, uint64_t& p) {
    try {
        if (!t.is_cuda() || t.layout() != at::kStrided || (int)t.scalar_type() != in.dtype || t.is_neg() ||
            t.sizes() != at::IntArrayRef(in.shape) || !t.is_contiguous() || t.get_device() != c->device)
            return false;
        p = (uint64_t)(uintptr_t)t.data_ptr();
    } catch (const std::exception&) {
        return false;
    }
    if (!p || (p & 31)) return false;                  // (null: a tensor without memory of its own)
    for (const auto& w : *c->written)
        if (p < w.second && w.first < p + in.bytes) return false;
    return true;
}

// call(inputs tuple) -> output, or None when these inputs cannot be read in place
PyObject* call_call(PyObject* self, PyObject* args, PyObject*) {
    HANDLE_TH_ERRORS
    Call* c = (Call*)self;
    PyObject* tuple;
    if (PyTuple_GET_SIZE(args) != 1 || !PyTuple_Check(tuple = PyTuple_GET_ITEM(args, 0))) {
        PyErr_SetString(PyExc_TypeError, "expected one tuple of tensors");
        return nullptr;
    }
    if (c->fault && *c->fault) return PyObject_CallFunction(c->fail, "i", 0);
    const size_t n = c->inputs->size();
    if ((size_t)PyTuple_GET_SIZE(tuple) != n) return refuse(c);
    uint64_t ptrs[64];
    for (size_t i = 0; i < c->ptrs->size(); ++i) ptrs[i] = (*c->ptrs)[i];
    for (size_t i = 0; i < n; ++i) {
        const Input& in = (*c->inputs)[i];
        PyObject* o = PyTuple_GET_ITEM(tuple, (Py_ssize_t)i);
        if (!THPVariable_Check(o)) return refuse(c);
        uint64_t p = 0;
        if (!in_place(c, in, THPVariable_Unpack(o), p)) return refuse(c);
        for (int s : in.slots) ptrs[s] = p;
    }
    const uint64_t stream = (uint64_t)(uintptr_t)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)c->device).stream();
    const int code = c->launch(c->kernel, c->grid, c->block, c->smem, ptrs, (int)c->ptrs->size(), stream, c->flags);
    if (code != 0) return PyObject_CallFunction(c->fail, "i", code);
    Py_INCREF(tuple);
    Py_SETREF(c->last, tuple);
    Py_INCREF(c->out);
    return c->out;
    END_HANDLE_TH_ERRORS
}

PyObject* call_last(PyObject* self, void*) {
    Call* c = (Call*)self;
    Py_INCREF(c->last);
    return c->last;
}

PyGetSetDef call_get[] = {{"last", call_last, nullptr, "inputs of the last call", nullptr}, {}};
PyType_Slot slots[] = {{Py_tp_new, (void*)call_new}, {Py_tp_dealloc, (void*)call_free},
                       {Py_tp_call, (void*)call_call}, {Py_tp_getset, (void*)call_get}, {0, nullptr}};
PyType_Spec spec = {"_mlcb_call.Call", sizeof(Call), 0, Py_TPFLAGS_DEFAULT, slots};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_mlcb_call", nullptr, -1, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__mlcb_call(void) {
    PyObject* m = PyModule_Create(&module);
    if (!m) return nullptr;
    PyObject* type = PyType_FromSpec(&spec);
    if (!type || PyModule_AddObject(m, "Call", type) < 0) {
        Py_XDECREF(type);
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
