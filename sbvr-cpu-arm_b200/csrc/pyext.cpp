// Python entry points of the package: everything between `sbvr.linear(x, w)` and the C ABI of libsbvr_b200.so.
//
// What bounds a call on few rows is the host: the kernel of a 1024 x 4096 linear on one row takes 5 us, and the same
// checks, look-ups and the ctypes call written in Python took 22 us (measured, calls back to back).  Here the weight's
// tensors are read straight from the module's dictionaries, the output is allocated through ATen and the library is called
// directly.  Nothing is remembered between calls but the workspace of a (device, stream) pair, which the Python side owns
// (`_lib.workspace`) and reports here; tensors are looked up again on every call, so a weight that was moved or replaced is
// seen as it is now.  The GIL is released around the library call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/core/InferenceMode.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <mutex>
#include <string>
#include <utility>

#include "../../include/sbvr_b200.h"

namespace {

struct Raised {};                                  // a Python exception is set

[[noreturn]] void fail(PyObject* type, const std::string& msg) {
    PyErr_SetString(type, msg.c_str());
    throw Raised();
}
// the message format of `_lib.check`
void check(int rc, const char* what) {
    if (rc == SBVR_OK) return;
    std::string m = std::string(what) + ": " + sbvr_strerror(rc);
    if (rc == SBVR_ERR_CUDA) m += " (cudaError " + std::to_string(sbvr_last_cuda_error()) + ")";
    fail(PyExc_RuntimeError, m);
}

// ---- workspaces -----------------------------------------------------------------------------------------------------
struct Ws {
    sbvr_workspace_t* handle;
    size_t bytes;
};
std::mutex g_ws_mu;
std::map<std::pair<int, uintptr_t>, Ws> g_ws;
PyObject* g_ws_callback = nullptr;                 // _lib.workspace(device, stream, nbytes): creates or enlarges, then reports here

// `few`: a call on few rows, which some kernel serves in any workspace: under capture it takes what is there, since an allocation
// would end the capture.
sbvr_workspace_t* workspace(int dev, uintptr_t stream, size_t need, bool few = false) {
    const auto key = std::make_pair(dev, stream);
    for (int attempt = 0; attempt < 2; ++attempt) {
        {
            std::lock_guard<std::mutex> lock(g_ws_mu);
            auto it = g_ws.find(key);
            if (it != g_ws.end() &&
                (it->second.bytes >= need || (few && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)))
                return it->second.handle;
        }
        if (attempt) break;
        PyObject* r = PyObject_CallFunction(g_ws_callback, "iKK", dev, (unsigned long long)stream, (unsigned long long)need);
        if (!r) throw Raised();
        Py_DECREF(r);
    }
    fail(PyExc_RuntimeError, "sbvr: workspace was not created");
}

// ---- the container's fields -------------------------------------------------------------------------------------------
PyObject *s_dict, *s_params, *s_bvr, *s_idx, *s_cache, *s_shape, *s_glen;

struct Weight {
    at::Tensor bvr, idx, coeff;                    // idx undefined: direct coefficients
    int KW, N, S, G, C, idx_bytes, dev;
    int64_t K;                                     // original inner length
};

struct Ref {                                       // an owned reference (or none)
    PyObject* o;
    explicit Ref(PyObject* p) : o(p) {}
    ~Ref() { Py_XDECREF(o); }
    Ref(const Ref&) = delete;
};
// An attribute of the container: from the module's dictionaries, which costs little; what is not there (a buffer, a property, an
// object that is no module) the way Python looks it up.
PyObject* field(PyObject* w, PyObject* d, PyObject* params, PyObject* name) {
    PyObject* v = params ? PyDict_GetItemWithError(params, name) : nullptr;
    if (!v && d) v = PyDict_GetItemWithError(d, name);
    if (v) {
        Py_INCREF(v);
        return v;
    }
    if (PyErr_Occurred()) throw Raised();
    v = PyObject_GetAttr(w, name);
    if (!v) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw Raised();
        PyErr_Clear();
    }
    return v;
}
at::Tensor tensor_field(const Ref& r, const char* name) {
    if (!r.o || !THPVariable_Check(r.o)) fail(PyExc_ValueError, std::string("not an sbvr weight: ") + name + " is missing");
    return THPVariable_Unpack(r.o);
}

int cuda_index(const at::Device& d) {
    if (!d.is_cuda())
        fail(PyExc_RuntimeError, "SBVR kernels run on CUDA tensors only (there is no CPU path); got device " + d.str());
    return d.has_index() ? d.index() : c10::cuda::current_device();
}

void read_weight(PyObject* w, Weight* o) {
    Ref dict(PyObject_GetAttr(w, s_dict));
    if (!dict.o) PyErr_Clear();
    PyObject* d = dict.o && PyDict_Check(dict.o) ? dict.o : nullptr;
    PyObject* params = d ? PyDict_GetItemWithError(d, s_params) : nullptr;
    if (params && !PyDict_Check(params)) params = nullptr;
    o->bvr = tensor_field(Ref(field(w, d, params, s_bvr)), "bvr");
    o->coeff = tensor_field(Ref(field(w, d, params, s_cache)), "coeff_cache");
    Ref ix(field(w, d, params, s_idx));
    if (o->bvr.dim() != 3) fail(PyExc_ValueError, "bvr must have three dimensions");
    o->KW = (int)o->bvr.size(0), o->N = (int)o->bvr.size(1), o->S = (int)o->bvr.size(2);
    o->dev = cuda_index(o->bvr.device());
    if (ix.o && ix.o != Py_None) {
        o->idx = tensor_field(ix, "coeff_idx");
        o->idx_bytes = (int)o->idx.element_size();
        o->C = (int)o->coeff.size(0);
        // the reference picks the index width from the codebook size (sbvr/kernels/sbvr_kernel.cu:887)
        if (o->idx_bytes != (o->C <= 256 ? 1 : 2)) fail(PyExc_AssertionError, "coeff_idx dtype disagrees with codebook size");
    } else {
        o->idx_bytes = 0, o->C = 0;
    }
    Ref gl(field(w, d, nullptr, s_glen)), sh(field(w, d, nullptr, s_shape));
    if (!gl.o || !sh.o) fail(PyExc_ValueError, "not an sbvr weight");
    o->G = (int)PyLong_AsLong(gl.o);
    const Py_ssize_t nd = PySequence_Size(sh.o);
    if (nd == 0) fail(PyExc_ValueError, "not an sbvr weight");
    Ref last(nd > 0 ? PySequence_GetItem(sh.o, nd - 1) : nullptr);
    if (!last.o) throw Raised();
    o->K = PyLong_AsLongLong(last.o);
    if (PyErr_Occurred()) throw Raised();
}
size_t workspace_need(const Weight& w, const void* x, int64_t M);
const uint32_t* bvr_ptr(const Weight& w) { return reinterpret_cast<const uint32_t*>(w.bvr.data_ptr()); }
const void* idx_ptr(const Weight& w) { return w.idx.defined() ? w.idx.data_ptr() : nullptr; }

at::Tensor opt_tensor(PyObject* o, const char* name) {
    if (!o || o == Py_None) return at::Tensor();
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, std::string(name) + " must be a tensor or None");
    return THPVariable_Unpack(o);
}
// "no bias" is None or an empty tensor (the reference's convention, sbvr/core.py:353-358)
at::Tensor bias_tensor(PyObject* o, int64_t N) {
    at::Tensor b = opt_tensor(o, "bias");
    if (!b.defined() || b.numel() == 0) return at::Tensor();
    if (b.numel() != N || b.scalar_type() != at::kHalf) fail(PyExc_ValueError, "bias must be float16 of length N");
    return b.contiguous();
}
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// Which kernel a call runs on must not depend on the calls before it: the workspace is asked to hold what the automatic choice
// would use, for few rows as for many.  One row, and two to four on weights that the decode GEMV takes, fit any workspace.
size_t workspace_need(const Weight& w, const void* x, int64_t M) {
    const int Kp = w.KW * 32;
    size_t need = 0;
    if (M > 4 || w.K != Kp || (M > 1 && (reinterpret_cast<uintptr_t>(x) & 15)))
        check(sbvr_workspace_bytes(w.dev, (int)M, w.N, Kp, &need), "sbvr_workspace_bytes");
    else if (M > 1)
        check(sbvr_linear_workspace_bytes(w.dev, bvr_ptr(w), idx_ptr(w), w.idx_bytes, w.coeff.data_ptr(), w.C, (int)M, w.N, Kp, w.S,
                                          w.G, &need), "sbvr_linear_workspace_bytes");
    return need;
}

struct ReleaseGil {
    PyThreadState* st;
    ReleaseGil() : st(PyEval_SaveThread()) {}
    ~ReleaseGil() { PyEval_RestoreThread(st); }
};

template <typename F>
PyObject* guarded(F f) {
    try {
        return f();
    } catch (const Raised&) {
    } catch (...) {                                // torch's own errors (out of memory among them) as torch raises them
        torch::translate_exception_to_python(std::current_exception());
    }
    return nullptr;
}

at::Tensor empty_half(at::IntArrayRef shape, const at::Device& dev) {
    return at::empty(shape, at::TensorOptions().dtype(at::kHalf).device(dev));
}

// ---- entry points -----------------------------------------------------------------------------------------------------
// linear(x, w, bias, algo, out)
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 5) fail(PyExc_TypeError, "linear takes 5 arguments");
        c10::InferenceMode im;
        if (!THPVariable_Check(a[0])) fail(PyExc_TypeError, "x must be a tensor");
        const at::Tensor x = THPVariable_Unpack(a[0]);
        if (x.scalar_type() != at::kHalf) fail(PyExc_ValueError, "activations must be float16");
        Weight w;
        read_weight(a[1], &w);
        if (x.device() != w.bvr.device())
            fail(PyExc_ValueError, "activation on " + x.device().str() + ", weight on " + w.bvr.device().str());
        const int64_t Kp = (int64_t)w.KW * 32;
        if (x.dim() < 1 || x.size(-1) != w.K)
            fail(PyExc_ValueError, "\033[91minner dimension mismatch: activation " +
                                       std::to_string(x.dim() ? x.size(-1) : 0) + ", weight " + std::to_string(w.K) + "\033[0m");
        const long algo = PyLong_AsLong(a[3]);
        if (algo == -1 && PyErr_Occurred()) throw Raised();
        const at::Tensor x2 = x.is_contiguous() ? x : x.contiguous();
        const int64_t M = w.K ? x.numel() / w.K : 0;
        const at::Tensor bias = bias_tensor(a[2], w.N);
        at::Tensor y = opt_tensor(a[4], "out");
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != w.dev) guard.set_index(w.dev);
        c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
        shape.back() = w.N;
        const bool given = y.defined();
        if (!given) y = empty_half(shape, x.device());
        if (M > 0) {
            const uintptr_t st = (uintptr_t)c10::cuda::getCurrentCUDAStream(w.dev).stream();
            sbvr_workspace_t* ws = workspace(w.dev, st, workspace_need(w, x2.data_ptr(), M), M <= 4 && w.K == Kp);
            int rc;
            {
                ReleaseGil nogil;
                rc = sbvr_linear_padded_f16(x2.data_ptr(), (int)w.K, bvr_ptr(w), idx_ptr(w), w.idx_bytes, w.coeff.data_ptr(), w.C,
                                            ptr(bias), y.data_ptr(), (int)M, w.N, (int)Kp, w.S, w.G, (int)algo, ws,
                                            reinterpret_cast<sbvr_stream_t>(st));
            }
            check(rc, "sbvr_linear_f16");
        }
        return THPVariable_Wrap(given ? y.view(shape) : y);
    });
}

// linear_fused(op, x, w, out, delta, norm_weight, h_out, eps, bias) -> bool
PyObject* py_linear_fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 9) fail(PyExc_TypeError, "linear_fused takes 9 arguments");
        c10::InferenceMode im;
        const long op = PyLong_AsLong(a[0]);
        const at::Tensor x = opt_tensor(a[1], "x"), out = opt_tensor(a[3], "out"), delta = opt_tensor(a[4], "delta");
        const at::Tensor nw = opt_tensor(a[5], "norm_weight"), ho = opt_tensor(a[6], "h_out"), bias = opt_tensor(a[8], "bias");
        const double eps = PyFloat_AsDouble(a[7]);
        if (PyErr_Occurred()) throw Raised();
        if (!x.defined() || !out.defined()) fail(PyExc_TypeError, "x and out must be tensors");
        Weight w;
        read_weight(a[2], &w);
        const int64_t Kp = (int64_t)w.KW * 32, M = x.size(0);
        if (M > 16 || w.K != Kp || !x.is_contiguous()) Py_RETURN_FALSE;
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != w.dev) guard.set_index(w.dev);
        const uintptr_t st = (uintptr_t)c10::cuda::getCurrentCUDAStream(w.dev).stream();
        sbvr_workspace_t* ws = workspace(w.dev, st, workspace_need(w, x.data_ptr(), M), M <= 4);
        int rc;
        {
            ReleaseGil nogil;
            rc = sbvr_linear_fused_f16((int)op, x.data_ptr(), ptr(delta), ptr(nw), ptr(ho), (float)eps, bvr_ptr(w), idx_ptr(w),
                                       w.idx_bytes, w.coeff.data_ptr(), w.C, ptr(bias), out.data_ptr(), (int)M, w.N, (int)Kp, w.S,
                                       w.G, ws, reinterpret_cast<sbvr_stream_t>(st));
        }
        if (rc == SBVR_ERR_UNSUPPORTED) Py_RETURN_FALSE;
        check(rc, "sbvr_linear_fused_f16");
        Py_RETURN_TRUE;
    });
}

// decode(w) -> [N, K] fp16
PyObject* py_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 1) fail(PyExc_TypeError, "decode takes 1 argument");
        c10::InferenceMode im;
        Weight w;
        read_weight(a[0], &w);
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != w.dev) guard.set_index(w.dev);
        at::Tensor out = empty_half({w.N, w.K}, w.bvr.device());
        const uintptr_t st = (uintptr_t)c10::cuda::getCurrentCUDAStream(w.dev).stream();
        int rc;
        {
            ReleaseGil nogil;
            rc = sbvr_decode_f16(bvr_ptr(w), idx_ptr(w), w.idx_bytes, w.coeff.data_ptr(), w.C, out.data_ptr(), (int)w.K, w.N,
                                 w.KW * 32, (int)w.K, w.S, w.G, reinterpret_cast<sbvr_stream_t>(st));
        }
        check(rc, "sbvr_decode_f16");
        return THPVariable_Wrap(out);
    });
}

// mm_T(lhs, rhs, bias) -> [M, N] fp16, or None where the popcount kernel does not cover the pair
PyObject* py_mm_T(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 3) fail(PyExc_TypeError, "mm_T takes 3 arguments");
        c10::InferenceMode im;
        Weight l, r;
        read_weight(a[0], &l);
        read_weight(a[1], &r);
        const bool ok = l.G == 256 && r.G == 256 && l.idx_bytes && r.idx_bytes && l.S >= 2 && l.S <= 4 && r.S >= 2 && r.S <= 4 &&
                        l.KW == r.KW && l.bvr.device() == r.bvr.device();
        if (!ok) Py_RETURN_NONE;
        const at::Tensor bias = bias_tensor(a[2], r.N);
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != r.dev) guard.set_index(r.dev);
        at::Tensor y = empty_half({l.N, r.N}, r.bvr.device());
        const uintptr_t st = (uintptr_t)c10::cuda::getCurrentCUDAStream(r.dev).stream();
        int rc;
        {
            ReleaseGil nogil;
            rc = sbvr_popc_mm_f16(bvr_ptr(l), idx_ptr(l), l.idx_bytes, l.coeff.data_ptr(), l.C, l.S, bvr_ptr(r), idx_ptr(r),
                                  r.idx_bytes, r.coeff.data_ptr(), r.C, r.S, ptr(bias), y.data_ptr(), l.N, r.N, r.KW * 32,
                                  reinterpret_cast<sbvr_stream_t>(st));
        }
        check(rc, "sbvr_popc_mm_f16");
        return THPVariable_Wrap(y);
    });
}

// row_deq(x, bvr_t, coeff_idx, coeff_cache, bias) -> [M, N] fp16; "no bias" is None or a tensor whose length is not N
// (the binding's convention, sbvr/kernels/sbvr_ops.cpp:102-104)
PyObject* py_row_deq(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 5) fail(PyExc_TypeError, "row_deq takes 5 arguments");
        c10::InferenceMode im;
        at::Tensor x = opt_tensor(a[0], "l_w"), bvr = opt_tensor(a[1], "r_bvr"), idx = opt_tensor(a[2], "r_coeff_idx");
        at::Tensor cache = opt_tensor(a[3], "r_coeff_cache"), bias = opt_tensor(a[4], "bias");
        if (!x.defined() || !bvr.defined() || !idx.defined() || !cache.defined()) fail(PyExc_TypeError, "tensors expected");
        if (x.scalar_type() != at::kHalf || cache.scalar_type() != at::kHalf)
            fail(PyExc_ValueError, "activations and coefficients must be float16");
        if ((bvr.scalar_type() != at::kUInt32 && bvr.scalar_type() != at::kInt) || bvr.dim() != 3)
            fail(PyExc_ValueError, "r_bvr must be uint32 [N/32, K, S]");
        if (!x.is_cuda()) fail(PyExc_ValueError, "tensors must live on a CUDA device");
        const int dev = x.device().has_index() ? x.device().index() : c10::cuda::current_device();
        const int64_t M = x.size(0), K = bvr.size(1), N = bvr.size(0) * 32;
        const int S = (int)bvr.size(2), C = (int)cache.size(0);
        if (x.dim() != 2 || x.size(1) != K)
            fail(PyExc_ValueError, "inner dimension mismatch: activation " + std::to_string(x.size(-1)) + ", weight " + std::to_string(K));
        const int G = (int)(N / std::max<int64_t>(1, idx.size(0)));
        // the reference picks the index width from the codebook size (sbvr/kernels/sbvr_kernel.cu:887, :931-932)
        const int ib = C <= 256 ? 1 : 2;
        if ((int)idx.element_size() != ib)
            fail(PyExc_ValueError, std::string("coefficient index must be ") + (ib == 1 ? "uint8" : "uint16") + " for " +
                                       std::to_string(C) + " cache lines");
        x = x.contiguous(), bvr = bvr.contiguous(), idx = idx.contiguous(), cache = cache.contiguous();
        if (bias.defined()) bias = bias.numel() == N ? bias.contiguous() : at::Tensor();
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != dev) guard.set_index(dev);
        at::Tensor out = empty_half({M, N}, x.device());
        if (M > 0) {
            const uintptr_t st = (uintptr_t)c10::cuda::getCurrentCUDAStream(dev).stream();
            sbvr_workspace_t* ws = workspace(dev, st, 0);
            int rc;
            {
                ReleaseGil nogil;
                rc = sbvr_linear_t_f16(x.data_ptr(), reinterpret_cast<const uint32_t*>(bvr.data_ptr()), idx.data_ptr(), ib,
                                       cache.data_ptr(), C, ptr(bias), out.data_ptr(), (int)M, (int)N, (int)K, S, G, ws,
                                       reinterpret_cast<sbvr_stream_t>(st));
            }
            check(rc, "sbvr_linear_t_f16");
        }
        return THPVariable_Wrap(out);
    });
}

// set_workspace(device, stream, handle, nbytes): what `_lib.workspace` now holds for this pair
PyObject* py_set_workspace(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 4) fail(PyExc_TypeError, "set_workspace takes 4 arguments");
        const int dev = (int)PyLong_AsLong(a[0]);
        const uintptr_t st = (uintptr_t)PyLong_AsUnsignedLongLong(a[1]);
        Ws v{reinterpret_cast<sbvr_workspace_t*>((uintptr_t)PyLong_AsUnsignedLongLong(a[2])),
             (size_t)PyLong_AsUnsignedLongLong(a[3])};
        if (PyErr_Occurred()) throw Raised();
        std::lock_guard<std::mutex> lock(g_ws_mu);
        if (v.handle) g_ws[std::make_pair(dev, st)] = v;
        else g_ws.erase(std::make_pair(dev, st));
        Py_RETURN_NONE;
    });
}
PyObject* py_set_callback(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 1) {
        PyErr_SetString(PyExc_TypeError, "set_workspace_callback takes 1 argument");
        return nullptr;
    }
    Py_XDECREF(g_ws_callback);
    g_ws_callback = a[0];
    Py_INCREF(g_ws_callback);
    Py_RETURN_NONE;
}

#define SBVR_FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL
PyMethodDef g_methods[] = {
    {"linear", SBVR_FAST(py_linear), "linear(x, w, bias, algo, out) -> y"},
    {"linear_fused", SBVR_FAST(py_linear_fused), "linear_fused(op, x, w, out, delta, norm_weight, h_out, eps, bias) -> bool"},
    {"decode", SBVR_FAST(py_decode), "decode(w) -> [N, K]"},
    {"mm_T", SBVR_FAST(py_mm_T), "mm_T(lhs, rhs, bias) -> [M, N] or None"},
    {"row_deq", SBVR_FAST(py_row_deq), "row_deq(x, bvr_t, idx, cache, bias) -> [M, N]"},
    {"set_workspace", SBVR_FAST(py_set_workspace), "set_workspace(device, stream, handle, nbytes)"},
    {"set_workspace_callback", SBVR_FAST(py_set_callback), "set_workspace_callback(f(device, stream, nbytes))"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_sbvr_native", "Host path of the SBVR package.", -1, g_methods};

}  // namespace

PyMODINIT_FUNC PyInit__sbvr_native(void) {
    s_dict = PyUnicode_InternFromString("__dict__");
    s_params = PyUnicode_InternFromString("_parameters");
    s_bvr = PyUnicode_InternFromString("bvr");
    s_idx = PyUnicode_InternFromString("coeff_idx");
    s_cache = PyUnicode_InternFromString("coeff_cache");
    s_shape = PyUnicode_InternFromString("original_data_shape");
    s_glen = PyUnicode_InternFromString("bvr_len");
    return PyModule_Create(&g_module);
}
