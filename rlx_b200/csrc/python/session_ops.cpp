// CompiledGraph.run of rlx_b200/api.py as one native call: host arrays through the buffer protocol, then rlxq_compiled_run.
// A run of a small graph lasts 20-30 us, and building the argument arrays in Python over ctypes took 4 us of it.
#include <Python.h>

#include <vector>

#include "rlxq.h"
#include "rlxq_session.h"

namespace {

PyObject* g_error = nullptr;       // rlx_b200.RlxqError
PyObject* g_as_f32 = nullptr;      // array -> contiguous f32 array

struct Buffers {
    std::vector<Py_buffer> views;
    std::vector<PyObject*> pairs;  // the names are theirs
    ~Buffers() {
        for (Py_buffer& v : views) PyBuffer_Release(&v);
        for (PyObject* p : pairs) Py_DECREF(p);
    }
    bool add(PyObject* o, int flags) {
        Py_buffer v;
        if (PyObject_GetBuffer(o, &v, flags)) return false;
        views.push_back(v);
        return true;
    }
};

bool is_f32(const Py_buffer& v) { return v.itemsize == 4 && v.format && v.format[0] == 'f' && !v.format[1]; }

bool add_input(Buffers& b, PyObject* a) {
    if (PyObject_CheckBuffer(a)) {
        if (b.add(a, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT)) {
            if (is_f32(b.views.back())) return true;
            PyBuffer_Release(&b.views.back());
            b.views.pop_back();
        }
        PyErr_Clear();
    }
    PyObject* c = PyObject_CallOneArg(g_as_f32, a);          // the view keeps it alive
    const bool ok = c && b.add(c, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT);
    Py_XDECREF(c);
    return ok;
}

// run(handle or None, sequence of (name, array), out)
PyObject* op_run(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (na != 3) { PyErr_SetString(PyExc_TypeError, "run takes 3 arguments"); return nullptr; }
    rlxq_compiled* h = nullptr;
    if (a[0] != Py_None) {
        h = static_cast<rlxq_compiled*>(PyLong_AsVoidPtr(a[0]));
        if (PyErr_Occurred()) return nullptr;
    }
    PyObject* seq = PySequence_Fast(a[1], "inputs must be a sequence of (name, array)");
    if (!seq) return nullptr;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    Buffers bufs;
    bufs.views.reserve(n + 1);
    bufs.pairs.reserve(n);
    std::vector<const char*> names(n);
    std::vector<const float*> data(n);
    std::vector<uint64_t> elems(n);
    bool ok = true;
    for (Py_ssize_t i = 0; ok && i < n; ++i) {
        PyObject* pair = PySequence_Tuple(PySequence_Fast_GET_ITEM(seq, i));       // any two things in a row; owns both
        ok = pair != nullptr;
        if (!ok) break;
        bufs.pairs.push_back(pair);
        if (PyTuple_GET_SIZE(pair) != 2) {
            PyErr_Format(PyExc_ValueError, "inputs must be (name, array) pairs, got %zd values", PyTuple_GET_SIZE(pair));
            ok = false;
            break;
        }
        names[i] = PyUnicode_AsUTF8(PyTuple_GET_ITEM(pair, 0));
        ok = names[i] && add_input(bufs, PyTuple_GET_ITEM(pair, 1));
        if (ok) {
            data[i] = static_cast<const float*>(bufs.views.back().buf);
            elems[i] = (uint64_t)bufs.views.back().len / 4;
        }
    }
    ok = ok && bufs.add(a[2], PyBUF_C_CONTIGUOUS | PyBUF_WRITABLE);
    int rc = 0;
    if (ok) {
        float* out = static_cast<float*>(bufs.views.back().buf);
        const uint64_t out_elems = (uint64_t)bufs.views.back().len / 4;
        Py_BEGIN_ALLOW_THREADS
        rc = rlxq_compiled_run(h, (uint32_t)n, names.data(), data.data(), elems.data(), out, out_elems);
        Py_END_ALLOW_THREADS
    }
    Py_DECREF(seq);
    if (!ok) return nullptr;
    if (rc < 0) {
        PyObject* arg = PyLong_FromLong(rc);
        PyObject* e = arg ? PyObject_CallOneArg(g_error, arg) : nullptr;
        Py_XDECREF(arg);
        if (e) { PyErr_SetObject(g_error, e); Py_DECREF(e); }
        return nullptr;
    }
    Py_RETURN_NONE;
}

// setup(RlxqError, array -> contiguous f32 array)
PyObject* op_setup(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (na != 2) { PyErr_SetString(PyExc_TypeError, "setup takes 2 arguments"); return nullptr; }
    Py_INCREF(a[0]);
    Py_INCREF(a[1]);
    Py_XDECREF(g_error);
    Py_XDECREF(g_as_f32);
    g_error = a[0];
    g_as_f32 = a[1];
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {{"run", (PyCFunction)(void (*)(void))op_run, METH_FASTCALL, nullptr},
                          {"setup", (PyCFunction)(void (*)(void))op_setup, METH_FASTCALL, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_session_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__session_ops(void) { return PyModule_Create(&kModule); }
