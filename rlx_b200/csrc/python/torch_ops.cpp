// The device-pointer calls of rlx_b200/api.py on torch CUDA tensors, as one native call each: argument checks,
// output and scratch allocation, the current stream and the C-ABI call (include/rlxq.h and its siblings).
//
// A decode-sized call lasts 6-15 us on the GPU, and the same steps written in Python over ctypes took 15 us of host
// time per call (25-30 us for the chain, expert-stack and LM-head calls), so an eager decode loop was bound by its
// host.  Here they take 4-6 us, most of it the kernel launches themselves.
//
// Errors keep their Python types: AssertionError for a tensor of the wrong kind, TypeError for a dtype the library
// does not take, RlxqError for a status the library returns.
#include <Python.h>

#include <ATen/Functions.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "rlxq.h"
#include "rlxq_lm.h"
#include "rlxq_moe.h"

namespace {

PyObject* g_error = nullptr;       // rlx_b200.RlxqError, handed over by api.py

struct Failed {};                  // a Python exception is set

void raise_status(int rc) {
    PyObject* arg = PyLong_FromLong(rc);
    PyObject* e = (arg && g_error) ? PyObject_CallOneArg(g_error, arg) : nullptr;
    Py_XDECREF(arg);
    if (e) { PyErr_SetObject(g_error, e); Py_DECREF(e); }
    else if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "rlxq status %d", rc);
    throw Failed{};
}
inline void check(int rc) { if (rc < 0) raise_status(rc); }

void require(bool ok, const char* what) {
    if (!ok) { PyErr_SetString(PyExc_AssertionError, what); throw Failed{}; }
}

const at::Tensor& tensor(PyObject* o, const char* what) {
    if (!THPVariable_Check(o)) { PyErr_Format(PyExc_TypeError, "%s must be a torch tensor", what); throw Failed{}; }
    return THPVariable_Unpack(o);
}

uint32_t dtype_of(const at::Tensor& t) {
    const auto st = t.scalar_type();
    if (st == at::kFloat) return RLXQ_F32;
    if (st == at::kBFloat16) return RLXQ_BF16;
    PyErr_Format(PyExc_TypeError, "activations must be float32 or bfloat16, got %s", c10::toString(st));
    throw Failed{};
}

uint32_t u32(PyObject* o) {
    if (PyLong_Check(o)) {
        const unsigned long v = PyLong_AsUnsignedLong(o);
        if (!PyErr_Occurred() && v <= 0xFFFFFFFFul) return (uint32_t)v;
    } else if (PyObject* i = PyNumber_Index(o)) {
        const unsigned long v = PyLong_AsUnsignedLong(i);
        Py_DECREF(i);
        if (!PyErr_Occurred() && v <= 0xFFFFFFFFul) return (uint32_t)v;
    }
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_OverflowError, "value does not fit 32 bits");
    throw Failed{};
}

const at::Tensor& activations(PyObject* o) {
    const at::Tensor& x = tensor(o, "x");
    require(x.is_cuda() && x.dim() == 2 && x.is_contiguous(), "x must be a contiguous two-dimensional CUDA tensor");
    return x;
}
const at::Tensor& weights(PyObject* o) {
    const at::Tensor& w = tensor(o, "w_blocks");
    require(w.is_cuda() && w.scalar_type() == at::kByte && w.is_contiguous(), "w_blocks must be a contiguous CUDA uint8 tensor");
    return w;
}

at::Tensor new_tensor(at::IntArrayRef size, at::ScalarType st, const at::Tensor& like) {
    return at::empty(size, at::TensorOptions().dtype(st).device(like.device()));
}

// The caller's output, or a new one of out_dtype (f32 when that is None).
struct Output {
    at::Tensor owned;
    PyObject* given = nullptr;
    const at::Tensor* t = nullptr;
    Output(PyObject* out, PyObject* out_dtype, int64_t m, int64_t n, const at::Tensor& like) {
        if (out != Py_None) {
            given = out;
            t = &tensor(out, "out");
            return;
        }
        at::ScalarType st = at::kFloat;
        if (out_dtype != Py_None) {
            if (!THPDtype_Check(out_dtype)) { PyErr_SetString(PyExc_TypeError, "out_dtype must be a torch dtype"); throw Failed{}; }
            st = reinterpret_cast<THPDtype*>(out_dtype)->scalar_type;
        }
        owned = new_tensor({m, n}, st, like);
        t = &owned;
    }
    PyObject* result() {
        if (given) { Py_INCREF(given); return given; }
        return THPVariable_Wrap(std::move(owned));
    }
};

// The caller's workspace when it holds `need` bytes, else `need` (at least `least`) bytes for this call, stream-ordered
// like any torch tensor.
struct Scratch {
    c10::DataPtr owned;
    void* ptr = nullptr;
    size_t bytes = 0;
    Scratch(PyObject* ws, size_t need, size_t least) {
        if (ws != Py_None) {
            const at::Tensor& t = tensor(ws, "workspace");
            if ((size_t)t.numel() >= need) { ptr = t.data_ptr(); bytes = (size_t)t.numel(); return; }
        }
        bytes = need > least ? need : least;
        if (bytes) { owned = c10::cuda::CUDACachingAllocator::get()->allocate(bytes); ptr = owned.get(); }
    }
};

// The library call itself runs without the interpreter lock, like any ctypes call.
template <typename F> int unlocked(F&& f) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return rc;
}

rlxq_stream_t stream_of(const at::Tensor& t) {
    return (rlxq_stream_t)c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

bool nargs_are(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    return false;
}

template <typename F> PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const Failed&) {
        return nullptr;
    } catch (const std::exception&) {      // torch's own errors (out of memory and the like) keep their Python types
        HANDLE_TH_ERRORS
        throw;
        END_HANDLE_TH_ERRORS
    }
}
}  // namespace

// matmul(x, w_blocks, scheme, n, out, out_dtype, workspace)
static PyObject* op_matmul(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!nargs_are(na, 7)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &x = activations(a[0]), &w = weights(a[1]);
        const uint32_t scheme = u32(a[2]), n = u32(a[3]), m = (uint32_t)x.size(0), k = (uint32_t)x.size(1);
        const c10::cuda::CUDAGuard dev(x.device());
        Output y(a[4], a[5], m, n, x);
        const uint32_t xd = dtype_of(x), yd = dtype_of(*y.t);
        size_t need = 0;
        check(rlxq_workspace_bytes(scheme, m, k, n, xd, yd, &need));
        Scratch ws(a[6], need, 0);
        const rlxq_stream_t s = stream_of(x);
        const void *xp = x.data_ptr(), *wp = w.data_ptr();
        void* yp = y.t->data_ptr();
        check(unlocked([&] { return rlxq_matmul(s, scheme, xp, xd, wp, yp, yd, m, k, n, need ? ws.ptr : nullptr, need); }));
        return y.result();
    });
}

// matmul_chain(x, layers, scheme, out, out_dtype, workspace); a layer is (w_blocks, n) or (w_blocks, n, swiglu)
static PyObject* op_matmul_chain(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!nargs_are(na, 6)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor& x = activations(a[0]);
        const uint32_t m = (uint32_t)x.size(0), scheme = u32(a[2]);
        constexpr Py_ssize_t kMost = 16;              // the library takes eight and says so
        rlxq_chain_layer layers[kMost];
        PyObject* seq = PySequence_Fast(a[1], "layers must be a sequence");
        if (!seq) throw Failed{};
        struct Drop { PyObject* o; ~Drop() { Py_DECREF(o); } } drop{seq};
        const Py_ssize_t nl = PySequence_Fast_GET_SIZE(seq);
        if (nl > kMost) raise_status(RLXQ_E_LIMIT);
        uint32_t width = (uint32_t)x.size(1);
        for (Py_ssize_t i = 0; i < nl; ++i) {
            PyObject* ly = PySequence_Fast(PySequence_Fast_GET_ITEM(seq, i), "a layer is (w_blocks, n) or (w_blocks, n, swiglu)");
            if (!ly) throw Failed{};
            Drop dl{ly};
            const Py_ssize_t len = PySequence_Fast_GET_SIZE(ly);
            if (len < 2) { PyErr_SetString(PyExc_IndexError, "a layer is (w_blocks, n) or (w_blocks, n, swiglu)"); throw Failed{}; }
            const at::Tensor& w = weights(PySequence_Fast_GET_ITEM(ly, 0));
            const uint32_t n = u32(PySequence_Fast_GET_ITEM(ly, 1));
            const int sw = len > 2 ? PyObject_IsTrue(PySequence_Fast_GET_ITEM(ly, 2)) : 0;
            if (sw < 0) throw Failed{};
            layers[i] = rlxq_chain_layer{w.data_ptr(), sw ? width / 2 : width, n, (uint32_t)sw};
            width = n;
        }
        const c10::cuda::CUDAGuard dev(x.device());
        Output y(a[3], a[4], m, width, x);
        const uint32_t xd = dtype_of(x);
        size_t need = 0;
        check(rlxq_chain_workspace_bytes(scheme, layers, (uint32_t)nl, m, xd, &need));
        Scratch ws(a[5], need, 256);
        const uint32_t yd = dtype_of(*y.t);
        const rlxq_stream_t s = stream_of(x);
        const void* xp = x.data_ptr();
        void* yp = y.t->data_ptr();
        check(unlocked([&] { return rlxq_matmul_chain(s, scheme, layers, (uint32_t)nl, xp, xd, yp, yd, m, ws.ptr, ws.bytes); }));
        return y.result();
    });
}

// grouped_matmul(x, w_blocks, expert_idx, scheme, n, num_experts, out, out_dtype, workspace)
static PyObject* op_grouped(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!nargs_are(na, 9)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &x = activations(a[0]), &w = weights(a[1]), &idx = tensor(a[2], "expert_idx");
        require(idx.is_cuda() && idx.scalar_type() == at::kFloat && idx.is_contiguous(), "expert_idx must be a contiguous CUDA float32 tensor");
        const uint32_t scheme = u32(a[3]), n = u32(a[4]), experts = u32(a[5]), m = (uint32_t)x.size(0), k = (uint32_t)x.size(1);
        require(idx.numel() == (int64_t)m, "expert_idx has one entry per row of x");
        const c10::cuda::CUDAGuard dev(x.device());
        Output y(a[6], a[7], m, n, x);
        size_t need = 0;
        check(rlxq_grouped_workspace_bytes(scheme, m, k, n, experts, &need));
        Scratch ws(a[8], need, 16);
        const uint32_t xd = dtype_of(x), yd = dtype_of(*y.t);
        const rlxq_stream_t s = stream_of(x);
        const void *xp = x.data_ptr(), *wp = w.data_ptr();
        const float* ip = idx.data_ptr<float>();
        void* yp = y.t->data_ptr();
        check(unlocked([&] { return rlxq_grouped_matmul(s, scheme, xp, xd, wp, ip, yp, yd, m, k, n, experts, ws.ptr, need); }));
        return y.result();
    });
}

// lm_head(hidden, w_bytes, n_embd, n_vocab, scheme, cap, exact, workspace); cap 0: the argmax call
static PyObject* op_lm_head(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!nargs_are(na, 8)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor &h = tensor(a[0], "hidden"), &w = weights(a[1]);
        const uint32_t k = u32(a[2]), n = u32(a[3]), scheme = u32(a[4]), cap = u32(a[5]);
        require(h.is_cuda() && h.is_contiguous() && h.numel() == (int64_t)k, "hidden must be a contiguous CUDA tensor of n_embd values");
        const int exact = PyObject_IsTrue(a[6]);
        if (exact < 0) throw Failed{};
        const c10::cuda::CUDAGuard dev(h.device());
        const uint32_t hd = dtype_of(h), rows = cap ? cap : 1u, flags = exact ? RLXQ_LM_EXACT : 0u;
        size_t need = 0;
        check(rlxq_lm_head_workspace_bytes(scheme, k, n, hd, rows, &need));
        Scratch ws(a[7], need, 0);
        at::Tensor idx = new_tensor({(int64_t)rows}, at::kInt, h), val = new_tensor({(int64_t)rows}, at::kFloat, h);
        const rlxq_stream_t s = stream_of(h);
        const void *hp = h.data_ptr(), *wp = w.data_ptr();
        uint32_t* ip = reinterpret_cast<uint32_t*>(idx.data_ptr<int32_t>());
        float* vp = val.data_ptr<float>();
        check(unlocked([&] {
            return cap ? rlxq_lm_head_topk(s, scheme, hp, hd, wp, k, n, cap, flags, ws.ptr, need, ip, vp)
                       : rlxq_lm_head_argmax(s, scheme, hp, hd, wp, k, n, flags, ws.ptr, need, ip, vp);
        }));
        PyObject* pi = THPVariable_Wrap(std::move(idx));
        PyObject* pv = THPVariable_Wrap(std::move(val));
        PyObject* r = pi && pv ? PyTuple_Pack(2, pi, pv) : nullptr;
        Py_XDECREF(pi);
        Py_XDECREF(pv);
        return r;
    });
}

// dequant_f32(w_blocks, scheme, n_elems, out)
static PyObject* op_dequant(PyObject*, PyObject* const* a, Py_ssize_t na) {
    if (!nargs_are(na, 4)) return nullptr;
    return guarded([&]() -> PyObject* {
        const at::Tensor& w = weights(a[0]);
        const uint32_t scheme = u32(a[1]);
        const unsigned long long count = PyLong_AsUnsignedLongLong(a[2]);
        if (PyErr_Occurred()) throw Failed{};
        const c10::cuda::CUDAGuard dev(w.device());
        at::Tensor owned;
        if (a[3] == Py_None) owned = new_tensor({(int64_t)count}, at::kFloat, w);
        const at::Tensor& out = a[3] == Py_None ? owned : tensor(a[3], "out");
        const rlxq_stream_t s = stream_of(w);
        const void* wp = w.data_ptr();
        float* op = static_cast<float*>(out.data_ptr());
        check(unlocked([&] { return rlxq_dequant_f32(s, scheme, wp, count, op); }));
        if (a[3] != Py_None) { Py_INCREF(a[3]); return a[3]; }
        return THPVariable_Wrap(std::move(owned));
    });
}

static PyObject* op_set_error(PyObject*, PyObject* cls) {
    Py_INCREF(cls);
    Py_XDECREF(g_error);
    g_error = cls;
    Py_RETURN_NONE;
}

static PyMethodDef kMethods[] = {
    {"matmul", (PyCFunction)(void (*)(void))op_matmul, METH_FASTCALL, nullptr},
    {"matmul_chain", (PyCFunction)(void (*)(void))op_matmul_chain, METH_FASTCALL, nullptr},
    {"grouped_matmul", (PyCFunction)(void (*)(void))op_grouped, METH_FASTCALL, nullptr},
    {"lm_head", (PyCFunction)(void (*)(void))op_lm_head, METH_FASTCALL, nullptr},
    {"dequant_f32", (PyCFunction)(void (*)(void))op_dequant, METH_FASTCALL, nullptr},
    {"set_error", op_set_error, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

static PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

PyMODINIT_FUNC PyInit__torch_ops(void) { return PyModule_Create(&kModule); }
