// hk_torch.cpp -- attention_forward / attention_backward over torch tensors, from native code: reads the tensors,
// allocates the outputs that were not given, fills the argument block and calls the library.
//
// The two calls on a small problem are host-bound: filling the ctypes blocks, allocating through torch's Python API and
// asking for the current stream took longer than the kernels run.  This module does the same work without Python
// objects in between.  The library is the one attention.py loads (dlsym on its handle), so an instrumented build given
// by HK_ATTENTION_LIB is used here too.
#include <ATen/ATen.h>
#include <Python.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/hk_attention.h"

namespace {

typedef int (*FwdFn)(const hk_attn_fwd_params*, void*);
typedef int (*BwdFn)(const hk_attn_bwd_params*, void*);
typedef int (*ZeroFn)(const hk_attn_bwd_params*, void*);
typedef size_t (*FwdSizeFn)(const hk_attn_fwd_params*);
typedef size_t (*BwdSizeFn)(const hk_attn_bwd_params*);
struct Library {
    FwdFn forward;
    BwdFn backward;
    ZeroFn zero_dq;
    FwdSizeFn fwd_bytes;
    BwdSizeFn bwd_bytes;
} g_lib = {};

// A tensor argument; None, where it may be left out, gives nullptr.  Anything else is refused: a mask or an output buffer
// of another kind must not pass for one that was not given.  False with TypeError set.
struct TensorArg {
    PyObject* object;
    const char* name;
    bool optional;
    const at::Tensor** tensor;
};
bool tensors(std::initializer_list<TensorArg> args) {
    for (const TensorArg& x : args) {
        *x.tensor = nullptr;
        if (THPVariable_Check(x.object)) {
            *x.tensor = &THPVariable_Unpack(x.object);
        } else if (!x.optional || x.object != Py_None) {
            PyErr_Format(PyExc_TypeError, "%s: expected a tensor%s, not %s", x.name, x.optional ? " or None" : "",
                         Py_TYPE(x.object)->tp_name);
            return false;
        }
    }
    return true;
}

// strides of a [B, H, T, 64] view into the block's (B, M, H) triple; false with AssertionError set
bool strides(const at::Tensor& t, int64_t* sB, int64_t* sM, int64_t* sH) {
    if (t.dim() != 4 || t.size(3) != 64 || t.stride(3) != 1) {
        PyErr_SetString(PyExc_AssertionError, "expected [B,H,T,64] with unit last stride");
        return false;
    }
    *sB = t.stride(0);
    *sM = t.stride(2);
    *sH = t.stride(1);
    return true;
}

void* stream_of(PyObject* o) {
    if (o == Py_None) return c10::cuda::getCurrentCUDAStream().stream();
    return reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(o));
}

// Runs an entry point's body.  A C++ exception thrown anywhere in it (no device, no memory, a tensor without strides or
// data) becomes the Python exception torch raises for it; left to itself it would end the process.
template <class F>
PyObject* guarded(F&& body) {
    try {
        return body();
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

// The interpreter is free for other threads while this lives; it is taken back on every way out.
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

float* data(const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); }

// workspace: 256-byte aligned start inside a tensor a caller brought; false with AssertionError set if `need` does not fit
bool given_workspace(const at::Tensor* t, size_t need, void** ptr, size_t* bytes) {
    if (!t) return true;
    uint8_t* base = static_cast<uint8_t*>(t->data_ptr());
    const size_t off = (256 - (reinterpret_cast<uintptr_t>(base) & 255u)) & 255u;
    const size_t have = (size_t)t->numel();
    if (need > 0 && have < off + need) {
        PyErr_SetString(PyExc_AssertionError, "workspace too small");
        return false;
    }
    *ptr = base + off;
    *bytes = have > off ? have - off : 0;
    return true;
}

}  // namespace

// forward(Q, K, V, scale, causal, dropout_p, dropout_mask, seed, offset, q_pos0, k_pos0, bh_pos0, flags, workspace, out,
//         lse, stream) -> (O, LSE), or the negative status of the call
static PyObject* forward_body(PyObject* const* a, Py_ssize_t n) {
    if (n != 17) {
        PyErr_SetString(PyExc_TypeError, "forward: 17 arguments");
        return nullptr;
    }
    const at::Tensor *Q, *K, *V, *mask, *ws, *out, *lse;
    if (!tensors({{a[0], "Q", false, &Q}, {a[1], "K", false, &K}, {a[2], "V", false, &V}, {a[6], "dropout_mask", true, &mask},
                  {a[13], "workspace", true, &ws}, {a[14], "out", true, &out}, {a[15], "lse", true, &lse}}))
        return nullptr;
    hk_attn_fwd_params p = {};
    if (!strides(*Q, &p.q_strideB, &p.q_strideM, &p.q_strideH) || !strides(*K, &p.k_strideB, &p.k_strideM, &p.k_strideH) ||
        !strides(*V, &p.v_strideB, &p.v_strideM, &p.v_strideH))
        return nullptr;
    const int64_t B = Q->size(0), H = Q->size(1), Tq = Q->size(2), Tk = K->size(2);
    const auto opt = Q->options().dtype(at::kFloat);
    at::Tensor O = out ? *out : at::empty({B, H, Tq, 64}, opt);
    at::Tensor L = lse ? *lse : at::empty({B, H, Tq}, opt);
    if (!strides(O, &p.o_strideB, &p.o_strideM, &p.o_strideH)) return nullptr;
    p.lse_strideB = L.stride(0);
    p.lse_strideH = L.stride(1);
    p.Q = data(*Q); p.K = data(*K); p.V = data(*V); p.O = data(O); p.LSE = data(L);
    p.B = (int)B; p.nh = (int)H; p.T = Tq;
    p.scale = (float)PyFloat_AsDouble(a[3]);
    p.is_causal = PyObject_IsTrue(a[4]) != 0;
    p.dropout_p = (float)PyFloat_AsDouble(a[5]);
    p.dropout_mask = mask ? data(*mask) : nullptr;
    p.kv_len = Tk != Tq ? Tk : 0;
    if (a[7] != Py_None) {  // the offset counts only beside a seed
        p.dropout_seed = PyLong_AsUnsignedLongLongMask(a[7]);
        p.dropout_offset = PyLong_AsUnsignedLongLongMask(a[8]);
    }
    p.q_pos0 = PyLong_AsLongLong(a[9]);
    p.k_pos0 = PyLong_AsLongLong(a[10]);
    p.bh_pos0 = (uint32_t)PyLong_AsUnsignedLongLongMask(a[11]);
    p.flags = (uint32_t)PyLong_AsUnsignedLongLongMask(a[12]);
    void* stream = stream_of(a[16]);
    if (PyErr_Occurred()) return nullptr;
    if (ws && !given_workspace(ws, g_lib.fwd_bytes(&p), &p.workspace, &p.workspace_bytes)) return nullptr;
    int rc;
    {
        NoGil nogil;
        rc = g_lib.forward(&p, stream);
    }
    if (rc != 0) return PyLong_FromLong(rc);
    PyObject* res = PyTuple_New(2);
    if (!res) return nullptr;
    PyTuple_SET_ITEM(res, 0, THPVariable_Wrap(std::move(O)));
    PyTuple_SET_ITEM(res, 1, THPVariable_Wrap(std::move(L)));
    return res;
}

// backward(Q, K, V, O, dO, LSE, scale, causal, dropout_p, dropout_mask, seed, offset, q_pos0, k_pos0, bh_pos0, flags,
//          workspace, D, dQ, dK, dV, stream) -> (dQ, dK, dV, D), or the negative status of the call
static PyObject* backward_body(PyObject* const* a, Py_ssize_t n) {
    if (n != 22) {
        PyErr_SetString(PyExc_TypeError, "backward: 22 arguments");
        return nullptr;
    }
    const at::Tensor *Q, *K, *V, *O, *dO, *LSE, *mask, *ws, *given[4];  // given: dQ, dK, dV, D
    if (!tensors({{a[0], "Q", false, &Q}, {a[1], "K", false, &K}, {a[2], "V", false, &V}, {a[3], "O", true, &O}, {a[4], "dO", false, &dO},
                  {a[5], "LSE", false, &LSE}, {a[9], "dropout_mask", true, &mask}, {a[16], "workspace", true, &ws},
                  {a[17], "D", true, &given[3]}, {a[18], "dQ", true, &given[0]}, {a[19], "dK", true, &given[1]}, {a[20], "dV", true, &given[2]}}))
        return nullptr;
    hk_attn_bwd_params p = {};
    if (!strides(*Q, &p.q_strideB, &p.q_strideM, &p.q_strideH) || !strides(*K, &p.k_strideB, &p.k_strideM, &p.k_strideH) ||
        !strides(*V, &p.v_strideB, &p.v_strideM, &p.v_strideH) || !strides(*dO, &p.do_strideB, &p.do_strideM, &p.do_strideH) ||
        (O && !strides(*O, &p.o_strideB, &p.o_strideM, &p.o_strideH)))
        return nullptr;
    const int64_t B = Q->size(0), H = Q->size(1), Tq = Q->size(2), Tk = K->size(2);
    p.flags = (uint32_t)PyLong_AsUnsignedLongLongMask(a[15]);
    p.B = (int)B; p.nh = (int)H; p.T = (int)Tq;
    p.kv_len = Tk != Tq ? Tk : 0;
    void* stream = stream_of(a[21]);
    if (PyErr_Occurred()) return nullptr;
    at::Tensor r[4], slabs;  // dQ, dK, dV, D
    const auto opt = Q->options().dtype(at::kFloat);
    for (int i = 0; i < 4; ++i)
        r[i] = given[i] ? *given[i] : i == 3 ? at::empty({B, H, Tq}, opt) : at::empty({B, H, i == 0 ? Tq : Tk, 64}, opt);
    if (!strides(r[0], &p.dq_strideB, &p.dq_strideM, &p.dq_strideH) || !strides(r[1], &p.dk_strideB, &p.dk_strideM, &p.dk_strideH) ||
        !strides(r[2], &p.dv_strideB, &p.dv_strideM, &p.dv_strideH))
        return nullptr;
    p.d_strideB = r[3].stride(0);
    p.d_strideH = r[3].stride(1);
    p.lse_strideB = LSE->stride(0);
    p.lse_strideH = LSE->stride(1);
    if (ws) {
        if (!given_workspace(ws, g_lib.bwd_bytes(&p), &p.workspace, &p.workspace_bytes)) return nullptr;
    } else if (p.flags & HK_FLAG_DETERMINISTIC_DQ) {  // the slabs of partial dQ are the only scratch there is
        hk_attn_bwd_params q = p;
        q.flags |= HK_FLAG_OPERANDS_PREROUNDED;
        const size_t bytes = g_lib.bwd_bytes(&q);
        // They are given back when this call returns, long before the kernels are done with them: they have to come from
        // the pool of the stream the kernels run on, where the next user of the memory is behind these.
        c10::cuda::OptionalCUDAStreamGuard guard;
        if (a[21] != Py_None && Q->is_cuda()) {
            const cudaStream_t s = static_cast<cudaStream_t>(stream);
            const auto device = Q->device().index();
            // 0 and cudaStreamLegacy are the default stream, which torch does not know by a handle
            guard.reset_stream(s == nullptr || s == cudaStreamLegacy ? c10::cuda::getDefaultCUDAStream(device)
                                                                     : c10::cuda::getStreamFromExternal(s, device));
        }
        slabs = at::empty({(int64_t)bytes + 256}, Q->options().dtype(at::kByte));
        if (!given_workspace(&slabs, bytes, &p.workspace, &p.workspace_bytes)) return nullptr;
    }
    p.Q = data(*Q); p.K = data(*K); p.V = data(*V); p.O = O ? data(*O) : nullptr; p.dO = data(*dO); p.LSE = data(*LSE);
    p.dQ = data(r[0]); p.dK = data(r[1]); p.dV = data(r[2]); p.D = data(r[3]);
    p.scale = (float)PyFloat_AsDouble(a[6]);
    p.is_causal = PyObject_IsTrue(a[7]) != 0;
    p.dropout_p = (float)PyFloat_AsDouble(a[8]);
    p.dropout_mask = mask ? data(*mask) : nullptr;
    if (a[10] != Py_None) {  // the offset counts only beside a seed
        p.dropout_seed = PyLong_AsUnsignedLongLongMask(a[10]);
        p.dropout_offset = PyLong_AsUnsignedLongLongMask(a[11]);
    }
    p.q_pos0 = PyLong_AsLongLong(a[12]);
    p.k_pos0 = PyLong_AsLongLong(a[13]);
    p.bh_pos0 = (uint32_t)PyLong_AsUnsignedLongLongMask(a[14]);
    if (PyErr_Occurred()) return nullptr;
    int rc;
    {
        NoGil nogil;
        rc = g_lib.backward(&p, stream);
    }
    if (rc != 0) return PyLong_FromLong(rc);
    PyObject* res = PyTuple_New(4);
    if (!res) return nullptr;
    for (int i = 0; i < 4; ++i) PyTuple_SET_ITEM(res, i, THPVariable_Wrap(std::move(r[i])));
    return res;
}

// zero(x, stream) -> status: zeroes a [B, H, T, 64] view
static PyObject* zero_body(PyObject* const* a, Py_ssize_t n) {
    if (n != 2) {
        PyErr_SetString(PyExc_TypeError, "zero: 2 arguments");
        return nullptr;
    }
    const at::Tensor* x;
    if (!tensors({{a[0], "dQ", false, &x}})) return nullptr;
    hk_attn_bwd_params p = {};
    if (!strides(*x, &p.dq_strideB, &p.dq_strideM, &p.dq_strideH)) return nullptr;
    p.B = (int)x->size(0); p.nh = (int)x->size(1); p.T = (int)x->size(2);
    p.dQ = data(*x);
    void* stream = stream_of(a[1]);
    if (PyErr_Occurred()) return nullptr;
    return PyLong_FromLong(g_lib.zero_dq(&p, stream));
}

static PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) { return guarded([&] { return forward_body(a, n); }); }
static PyObject* backward(PyObject*, PyObject* const* a, Py_ssize_t n) { return guarded([&] { return backward_body(a, n); }); }
static PyObject* zero(PyObject*, PyObject* const* a, Py_ssize_t n) { return guarded([&] { return zero_body(a, n); }); }

// bind(handle): the dlopen handle of libhk_attention.so
static PyObject* bind(PyObject*, PyObject* h) {
    void* so = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(h));
    if (PyErr_Occurred()) return nullptr;
    g_lib.forward = reinterpret_cast<FwdFn>(dlsym(so, "hk_attn_forward_noscratch"));
    g_lib.backward = reinterpret_cast<BwdFn>(dlsym(so, "hk_attn_backward_noscratch"));
    g_lib.zero_dq = reinterpret_cast<ZeroFn>(dlsym(so, "hk_attn_zero_dq"));
    g_lib.fwd_bytes = reinterpret_cast<FwdSizeFn>(dlsym(so, "hk_attn_fwd_workspace_bytes"));
    g_lib.bwd_bytes = reinterpret_cast<BwdSizeFn>(dlsym(so, "hk_attn_bwd_workspace_bytes"));
    if (!g_lib.forward || !g_lib.backward || !g_lib.zero_dq || !g_lib.fwd_bytes || !g_lib.bwd_bytes) {
        PyErr_SetString(PyExc_ImportError, "libhk_attention.so lacks an entry point");
        return nullptr;
    }
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL, nullptr},
    {"backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(backward)), METH_FASTCALL, nullptr},
    {"zero", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(zero)), METH_FASTCALL, nullptr},
    {"bind", bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
static PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hk_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

PyMODINIT_FUNC PyInit__hk_torch() { return PyModule_Create(&module); }
